"""The host's rules that choose a kernel variant, run on the CPU: a small program calls them
from csrc/bes_launch.cu, compiled with a system definition of the test's choice."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "bubbleensemble_implicitextension_b200" / "csrc"

SMS = 148


def run_rules(tmp_path, body, model="", lib=None, decl=""):
    """Output of `body`, C++ statements over namespace bes; `model`: lines that change the system definition.
    Linked with the library `lib` where the body asks what fits on an SM, else the kernels' entry points stay
    unresolved: the rules alone call none."""
    (tmp_path / "model.cuh").write_text('#include "km_model.cuh"\n' + model)
    (tmp_path / "main.cu").write_text(
        '#include <cstdio>\n#include "bes_launch.h"\n' + decl + 'int main() {\n    using namespace bes;\n' + body + "\n}\n")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "rules"
    link = ["-Xlinker", "--unresolved-symbols=ignore-all"]
    if lib:
        link = [str(lib), "-Xlinker", f"-rpath={lib.parent}"]
    res = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", str(tmp_path),
                          "-I", str(CSRC), '-DBES_SYSTEM_DEFINITION="model.cuh"', str(CSRC / "bes_launch.cu"),
                          str(tmp_path / "main.cu"), *link, "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
    return out.stdout.split()


TEAM_OF_EIGHT = f"""
    for (int sym = 0; sym < 2; sym++) {{
        const Variant v = class_variant(0, false, sym, 0, sym, 0, 0, team_pays(8, sym, 0, {SMS}));
        std::printf("%d/%d ", v.rhs, v.G);
    }}"""


@pytest.mark.parametrize("scope", ["NSP", "NSA", "NISA", "NGP", "NIGP"])
def test_no_teams_for_models_with_shared_values(scope, tmp_path):
    """The warps of a team must come to the same bits: not where the callbacks share values between units."""
    assert run_rules(tmp_path, TEAM_OF_EIGHT, f"#undef BES_MODEL_{scope}\n#define BES_MODEL_{scope} 1\n") == ["1/1", "5/1"]


def test_no_teams_for_models_too_large_for_four_copies(tmp_path):
    assert run_rules(tmp_path, TEAM_OF_EIGHT, "#undef BES_MODEL_NUP\n#define BES_MODEL_NUP 200\n") == ["1/1", "5/1"]


def test_teams_for_models_with_unit_values_only(tmp_path):
    assert run_rules(tmp_path, TEAM_OF_EIGHT) == ["11/4", "15/4"]


def test_how_many_systems_run_on_teams(tmp_path):
    """A system to an SM always; two with the shared symmetric matrix and the single-reduction recurrence."""
    body = f"""
    for (int rec = 0; rec < 2; rec++)
        for (int sym = 0; sym < 2; sym++)
            for (int total : {{{SMS}, {SMS + 1}, {2 * SMS}, {2 * SMS + 1}}})
                std::printf("%d ", team_pays(total, sym, rec, {SMS}));"""
    assert run_rules(tmp_path, body) == ["1", "0", "0", "0"] * 3 + ["1", "1", "1", "0"]


# most banded systems of 33-64 and of 65-128 units to a CTA of eight warps, by band width: what the band, the
# operator, the vectors and the 21 unit parameters leave room for
BAND_FITS = {2: {3: 4, 4: 4, 16: 4, 19: 4, 20: 3, 28: 3, 29: 2}, 4: {3: 2, 4: 2, 17: 2, 20: 2, 21: 1, 45: 1, 48: 1}}


@pytest.mark.parametrize("rec", [0, 1])
def test_bands_that_fit(rec, tmp_path, bes_lib):
    widths = [(g, bw) for g, fits in BAND_FITS.items() for bw in fits]
    body = "".join(f"""
    std::printf("%d ", max_warps_per_block(class_variant({g // 2}, false, false, 0, false, {rec}, {bw})) / {g});"""
                   for g, bw in widths)
    from bubbleensemble_implicitextension_b200 import _build
    got = [int(x) for x in run_rules(tmp_path, body, lib=_build.LIB)]
    assert dict(zip(widths, got)) == {(g, bw): BAND_FITS[g][bw] for g, bw in widths}


@pytest.mark.parametrize("parameters,variants", [(21, ["24/4", "27/4"]), (80, ["4/4", "7/4"])])
def test_sixteen_warps_only_where_they_fit(parameters, variants, tmp_path):
    """With 80 unit parameters shared memory holds two systems of 128 units an SM at most: eight warps.  The
    layouts' sizes are those of the kernels' own macros."""
    decl = """#include "bes_kernel_inst.cuh"
namespace bes {
template <> size_t cta_smem_t<1, 4, 4, 0>(int warps, int band) { return BES_SMEM_SHARED(1, 4, true); }
template <> size_t cta_smem_t<1, 24, 4, 0>(int warps, int band) { return BES_SMEM_SHARED(1, 4, true); }
template <> size_t cta_smem_t<1, 7, 4, 0>(int warps, int band) { return BES_SMEM_BAND(4, false); }
template <> size_t cta_smem_t<1, 27, 4, 0>(int warps, int band) { return BES_SMEM_BAND(4, false); }
}
"""
    body = f"""
    const bool dense = dense_pays(2, 512, {SMS});
    const Variant v[2] = {{class_variant(2, false, true, 0, true, 0, 0, false, dense),
                          class_variant(2, false, false, 0, false, 0, 1, false, dense)}};
    for (const Variant& x : v) std::printf("%d/%d ", x.rhs, x.G);"""
    model = f"#undef BES_MODEL_NUP\n#define BES_MODEL_NUP {parameters}\n"
    assert run_rules(tmp_path, body, model, decl=decl) == variants


@pytest.mark.parametrize("components,parameters", [(2, 87), (6, 80), (12, 85)])
def test_models_up_to_the_limit_of_shared_memory(components, parameters, tmp_path):
    """128 units with a full matrix, their vectors and exchange buffers leave room for 87 unit parameters: whatever
    else a kernel keeps in shared memory has to give way."""
    body = """
    std::printf("%d %d %d", WarpSmem<1, 4>::BYTES <= SMEM_MAX,
                SharedCSmem<1, 4, false>::C_BYTES + SharedCSmem<1, 4, false>::WARP_BYTES <= SMEM_MAX,
                BandSmem<4, true>::doubles(16) * 8 <= SMEM_MAX);"""
    model = (f"#undef BES_MODEL_NUP\n#define BES_MODEL_NUP {parameters}\n"
             f"#undef BES_MODEL_UD\n#define BES_MODEL_UD {components}\n")
    decl = '#include "bes_kernel.cuh"\n'
    assert run_rules(tmp_path, body, model, decl=decl) == ["1", "1", "1"]


def test_which_variants_read_each_systems_own_matrix(tmp_path):
    """Only the shared-matrix kernels apply unit coupling factors: every other variant, the banded ones of one, two
    and four warps among them, counts as reading the system's own matrix, and factors are refused there."""
    body = """
    for (int cls = 0; cls < 3; cls++)
        for (int band : {0, 1, 9})
            for (int shared = 0; shared < 3; shared++)      /* 2: symmetric too */
                for (int wps = 0; wps < 2; wps++)
                    for (int rule = 0; rule < 4; rule++) {  /* none, team, dense, sparse */
                        const Variant v = class_variant(cls, rule == 0, shared > 0, wps, shared == 2, 0, band,
                                                        rule == 1, rule == 2, rule == 3);
                        const bool applied = shared > 0 && (cls > 0 || shared == 2);
                        if (own_matrix(v) == applied) std::printf("%d/%d/%d ", v.U, v.rhs, v.G);
                    }
    std::printf("done");"""
    decl = "namespace bes {\n" + "".join(
        f"template <> size_t cta_smem_t<1, {rhs}, {g}, 0>(int w, int) {{ return 1024 * w; }}\n"
        for rhs in (4, 7, 24, 27) for g in (2, 4)) + "}\n"
    assert run_rules(tmp_path, body, decl=decl) == ["done"]
