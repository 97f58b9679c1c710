/* bes_launch.cu -- dispatch from a run-time variant to the kernel instantiations. */
#include <algorithm>

#include "bes_kernel.cuh"
#include "bes_launch.h"

namespace bes {

namespace {

template <int U_, int RHS_, int G_, int REC_>
struct Tag {
    static constexpr int U = U_, RHS = RHS_, G = G_, REC = REC_;
};

template <int REC, class F>
bool dispatch_rec(Variant v, F&& f) {
    const int key = v.U * 1000 + v.rhs * 10 + v.G;
    switch (key) {
        case 1011: f(Tag<1, 1, 1, REC>{}); return true;
        case 1021: f(Tag<1, 2, 1, REC>{}); return true;
        case 1081: f(Tag<1, 8, 1, REC>{}); return true;
        case 1091: f(Tag<1, 9, 1, REC>{}); return true;
        case 1051: f(Tag<1, 5, 1, REC>{}); return true;
        case 1061: f(Tag<1, 6, 1, REC>{}); return true;
        case 2001: f(Tag<2, 0, 1, REC>{}); return true;
        case 2031: f(Tag<2, 3, 1, REC>{}); return true;
        case 4001: f(Tag<4, 0, 1, REC>{}); return true;
        case 4031: f(Tag<4, 3, 1, REC>{}); return true;
        case 2041: f(Tag<2, 4, 1, REC>{}); return true;
        case 4041: f(Tag<4, 4, 1, REC>{}); return true;
        case 1042: f(Tag<1, 4, 2, REC>{}); return true;
        case 1044: f(Tag<1, 4, 4, REC>{}); return true;
        case 1002: f(Tag<1, 0, 2, REC>{}); return true;
        case 1032: f(Tag<1, 3, 2, REC>{}); return true;
        case 1004: f(Tag<1, 0, 4, REC>{}); return true;
        case 1034: f(Tag<1, 3, 4, REC>{}); return true;
        case 1071: f(Tag<1, 7, 1, REC>{}); return true;
        case 1072: f(Tag<1, 7, 2, REC>{}); return true;
        case 1074: f(Tag<1, 7, 4, REC>{}); return true;
        case 1101: f(Tag<1, 10, 1, REC>{}); return true;
        case 1102: f(Tag<1, 10, 2, REC>{}); return true;
        case 1104: f(Tag<1, 10, 4, REC>{}); return true;
        /* teams: four warps a system */
        case 1114: f(Tag<1, 11, 1, REC>{}); return true;
        case 1124: f(Tag<1, 12, 1, REC>{}); return true;
        case 1154: f(Tag<1, 15, 1, REC>{}); return true;
        case 1164: f(Tag<1, 16, 1, REC>{}); return true;
        /* sixteen warps an SM */
        case 1242: f(Tag<1, 24, 2, REC>{}); return true;
        case 1244: f(Tag<1, 24, 4, REC>{}); return true;
        case 1272: f(Tag<1, 27, 2, REC>{}); return true;
        case 1274: f(Tag<1, 27, 4, REC>{}); return true;
        default: return false;
    }
}

/* calls f(Tag<U, RHS, G, REC>{}) for the built variant v; false if v is not built */
template <class F>
bool dispatch(Variant v, F&& f) {
    if (v.rec == 0) return dispatch_rec<0>(v, f);
    if (v.rec == 1) return dispatch_rec<1>(v, f);
    return false;
}

}  // namespace

bool variant_exists(Variant v) {
    return dispatch(v, [](auto) {});
}

size_t cta_smem_bytes(Variant v, int warps) {
    size_t r = 0;
    dispatch(v, [&](auto t) { using T = decltype(t); r = cta_smem_t<T::U, T::RHS, T::G, T::REC>(warps, v.band); });
    return r;
}

int max_warps_per_block(Variant v) {
    /* the kernels' launch bounds: 512 threads for RHS > 20, 256 with a shared or banded matrix or G > 1, else 128 */
    const int cap = v.rhs > 20 ? 16 : (v.rhs == 3 || v.rhs == 4 || v.rhs == 7 || v.rhs == 10 || v.G > 1) ? 8 : 4;
    int w = 0;
    while (w + v.G <= cap && cta_smem_bytes(v, w + v.G) <= (size_t)SMEM_MAX) w += v.G;
    return w;
}

cudaError_t occupancy(Variant v, int warps, int* ctas_per_sm) {
    cudaError_t e = cudaErrorInvalidValue;
    dispatch(v, [&](auto t) { using T = decltype(t); e = occupancy_t<T::U, T::RHS, T::G, T::REC>(warps, v.band, ctas_per_sm); });
    return e;
}

cudaError_t launch(Variant v, const DeviceProblem& P, int grid, int warps, cudaStream_t stream) {
    cudaError_t e = cudaErrorInvalidValue;
    dispatch(v, [&](auto t) { using T = decltype(t); e = launch_t<T::U, T::RHS, T::G, T::REC>(P, grid, warps, stream); });
    return e;
}

/* kernel variant of a units class: N <= 32 keeps half of the operator in
 * registers (rhs 2: every system has exactly 32 units); larger N runs one unit
 * per lane on 2 or 4 warps with W in tensor memory (or 2 or 4 units per lane on
 * one warp with W in shared memory), or one staged copy of a matrix shared by the
 * whole class when the caller asked for shared coupling matrices
 * (SharedCouplingMatrices).  team, dense and sparse are what team_pays, dense_pays
 * and sparse_pays say of the launch.  With banded coupling storage (band > 0) every class whose matrix is not staged
 * as a shared symmetric (N <= 32) or shared (N > 32) matrix runs the banded
 * operator, one unit per lane on 1, 2 or 4 warps. */
Variant class_variant(int cls, bool all32, bool shared, int warps_per_system, bool symmetric, int rec, int band,
                      bool team, bool dense, bool sparse) {
    const bool wide = 2 * band + 1 > BAND_REGS;   /* more diagonals than the registers take */
    if (cls == 0) {
        const bool sym = shared && symmetric;   /* a share of G in registers */
        if (!sym && band > 0) return Variant{1, wide ? 10 : 7, 1, rec, band};
        const int rhs = sym ? (all32 ? 6 : 5) : (all32 ? 2 : 1);
        if (team && warps_per_system != 1) return Variant{1, rhs + 10, TEAM, rec};
        return Variant{1, !sym && sparse ? rhs + 7 : rhs, 1, rec};
    }
    const int width = cls == 1 ? 2 : 4;
    /* sixteen warps an SM only where shared memory holds more than the eight of the other kernel */
    auto denser = [&](Variant v) {
        const Variant d{v.U, v.rhs + 20, v.G, v.rec, v.band};
        return dense && max_warps_per_block(d) > max_warps_per_block(v) ? d : v;
    };
    if (!shared && band > 0) {   /* banded storage: one unit per lane */
        const Variant v{1, wide ? 10 : 7, width, rec, band};
        return wide ? v : denser(v);
    }
    const int rhs = shared ? (symmetric ? 4 : 3) : 0;
    if (warps_per_system == 1) return Variant{width, rhs, 1, rec};
    const Variant v{1, rhs, width, rec};
    return rhs == 4 ? denser(v) : v;
}

/* Can every warp of a team run the model's callbacks and come to the same bits?  Only while the callbacks
 * write nothing but their own unit's values: a global parameter would be written four times, and each warp
 * has its own copy of the system-scope values, on which the units of a system may race (plain stores, atomic
 * sums).  Nothing orders those alike in two warps, so the copies could differ, the warps decide differently,
 * and one wait at a team barrier for an exchange that the others never make.  The four warps' copies have to
 * fit in shared memory, too. */
constexpr bool TEAM_MODEL = BES_MODEL_NGP == 0 && BES_MODEL_NIGP == 0 && BES_MODEL_NSP == 0 && BES_MODEL_NSA == 0 &&
                            BES_MODEL_NISA == 0 && TEAM * WarpSmem<1, 1, TEAM>::BYTES <= SMEM_MAX;

/* Does a launch of `total` systems run those of up to 32 units on teams of four warps (where TEAM_MODEL
 * allows them)?  Eight warps of 255 registers are what an SM holds, and a team's warps repeat everything but
 * the products, so a system to an SM always gains (148 systems of 32 units, 250 steps: 5.5 -> 5.1 ms, with
 * REC 1 5.65 -> 4.7).  Two gain only with the shared symmetric matrix and REC 1, whose iteration is the more
 * product (256 x 32 to the end of a period, three draws: 353, 325, 321 -> 324, 293, 289 ms; with REC 0 350,
 * 321, 318 -> 357, 322, 330; own matrix 322 -> 326), and beside multi-warp systems none (384 uneven clouds:
 * 92 -> 112 ms). */
bool team_pays(int total, bool symmetric, int rec, int sm_count) {
    return TEAM_MODEL && total <= (symmetric && rec == 1 ? 2 : 1) * sm_count;
}

/* Does a launch of `total` systems, all of up to 32 units, keep the column share of W in tensor
 * memory?  While no sub-partition holds two of its warps (see coupled_rhs_regw for both sides);
 * beside multi-warp systems, whose matrices stream from there, it slowed both (384 uneven clouds
 * 92 -> 110 ms). */
bool sparse_pays(int count, int total, int sm_count) { return count == total && total <= 4 * sm_count; }

/* Do `count` systems of class cls (1: two warps each, 2: four) run the kernels compiled for sixteen
 * warps an SM?  As soon as there are more than the eight warps of 255 registers hold at once: the
 * 128-register kernels spill a little, but run twice the systems side by side (512 shared-geometry
 * systems of 128 bubbles 331 -> 291 ms, 512 rings of 128 307 -> 252 ms per pass).  Where shared memory
 * holds no more of them, they only spill: class_variant leaves them out there, and for bands beyond the
 * registers (512 systems of 128 units at CBW 8: 28.9 -> 18.2 ms without). */
bool dense_pays(int cls, int count, int sm_count) { return count > (cls == 1 ? 4 : 2) * sm_count; }

/* CTA shape of a launch of `count` systems: spread small ensembles over every
 * SM, fill SMs otherwise; `requested` > 0 asks for that many warps per CTA */
int class_warps_per_block(Variant v, int count, int sm_count, int requested) {
    const int cap = max_warps_per_block(v);
    int wpb = requested;
    if (wpb <= 0) {
        const int systems = count <= sm_count ? 1 : (count <= 2 * sm_count ? 2 : cap / v.G);
        wpb = systems * v.G;
    }
    wpb = std::max(v.G, std::min(wpb, cap)) / v.G * v.G;
    return wpb;
}

}  // namespace bes
