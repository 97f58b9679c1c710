"""The host's rules that choose a kernel variant, run on the CPU: a small program calls them
from csrc/bes_launch.cu, compiled with a system definition of the test's choice."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "bubbleensemble_implicitextension_b200" / "csrc"

SMS = 148


def run_rules(tmp_path, body, model=""):
    """Output lines of `body`, C++ statements over namespace bes; `model`: lines that change the system definition.
    The rules call no kernel, so the kernels' entry points stay unresolved."""
    (tmp_path / "model.cuh").write_text('#include "km_model.cuh"\n' + model)
    (tmp_path / "main.cu").write_text(
        '#include <cstdio>\n#include "bes_launch.h"\nint main() {\n    using namespace bes;\n' + body + "\n}\n")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "rules"
    res = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", str(tmp_path),
                          "-I", str(CSRC), '-DBES_SYSTEM_DEFINITION="model.cuh"', str(CSRC / "bes_launch.cu"),
                          str(tmp_path / "main.cu"), "-Xlinker", "--unresolved-symbols=ignore-all", "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
    return out.stdout.split()


TEAM_OF_EIGHT = f"""
    for (int sym = 0; sym < 2; sym++) {{
        const Variant v = class_variant(0, false, sym, 0, sym, 0, 0, team_pays(8, sym, {SMS}));
        std::printf("%d/%d ", v.rhs, v.G);
    }}"""


@pytest.mark.parametrize("scope", ["NSP", "NSA", "NISA", "NGP", "NIGP"])
def test_no_teams_for_models_with_shared_values(scope, tmp_path):
    """The warps of a team must come to the same bits: not where the callbacks share values between units."""
    assert run_rules(tmp_path, TEAM_OF_EIGHT, f"#undef BES_MODEL_{scope}\n#define BES_MODEL_{scope} 1\n") == ["1/1", "5/1"]


def test_teams_for_models_with_unit_values_only(tmp_path):
    assert run_rules(tmp_path, TEAM_OF_EIGHT) == ["11/4", "15/4"]
