/*
 * bes_kernel.cuh -- the persistent ensemble integrator for sm_100a.
 *
 * A group of G warps integrates one system; lane l of warp w owns units
 * 32 (G m + w) + l for m < U, so the system holds up to 32 U G units (single
 * warps with U = 1, 2, 4, or U = 1 with G = 2, 4 warps for N <= 64, 128).
 * Groups pull systems from a global work counter until the ensemble is done,
 * and each system runs `n_periods` consecutive reference Solve() calls inside
 * the one launch.
 *
 * Reference behaviour restated here (file:line in the reference):
 *   step loop, callbacks, write-back  SourceCodes/CoupledSystmes_PerBlock_Solver.cuh:82-648
 *   RKCK45 stages, y5, error          SourceCodes/CoupledSystems_PerBlock_ExplicitRungeKutta_Steppers.cuh:94-425
 *   BiCG for the coupled accelerations ...ExplicitRungeKutta_Steppers.cuh:432-562, helpers :565-805
 *   step-size controller              SourceCodes/CoupledSystems_PerBlock_ExplicitRungeKutta_ErrorControllers.cuh:454-542
 *   RK4 fixed-step controller         ...ExplicitRungeKutta_ErrorControllers.cuh:424-450
 *   event step cut                    SourceCodes/CoupledSystems_PerBlock_EventHandling.cuh:216-268
 *   dense output                      SourceCodes/CoupledSystems_PerBlock_DenseOutput.cuh:312-395
 *
 * B200 design: the reference's shared-memory tree reductions and CAS
 * atomics become warp butterflies (the butterfly computes the reference's
 * halving-tree sum exactly, because IEEE addition is commutative); the
 * transposed product A^T p~, which the reference forms with N block-wide
 * reductions per BiCG iteration, becomes column trees over the operator
 * W_ij = (rD_i C_ij) X0_j^2 that is formed once per right-hand side: in
 * registers and shared memory for one warp, in tensor memory for a group.  When
 * the launch shares one matrix, it is staged once per CTA
 * instead; when that matrix is symmetric (a geometry 1/d with the radii as
 * unit factors), both products become row sums of the same entries -- read
 * once from tensor memory, or for N <= 32 held in registers for a right-hand
 * side.  Every scalar of the step control is uniform over the group
 * and held in registers; a single-warp system needs no block barrier at all,
 * a multi-warp system one named barrier per reduction.
 *
 * Arithmetic order (identical in the CPU oracle): sums over units are the
 * halving tree over units padded with zeros to 32UG; the row products use
 * four interleaved fma chains over the columns (j mod 4) combined as
 * (s0 + s1) + (s2 + s3); every fused multiply-add is explicit (the file is
 * compiled with --fmad=false).
 */
#ifndef BES_KERNEL_CUH
#define BES_KERNEL_CUH

#include "bes_device.h"
#include "bes_math.cuh"
#include "bes_status.h"
#include "bes_tmem.cuh"

#ifndef BES_SYSTEM_DEFINITION
#include "km_model.cuh"
#else
#include BES_SYSTEM_DEFINITION
#endif

namespace bes {

constexpr int UD = BES_MODEL_UD;
constexpr int NUP = BES_MODEL_NUP;
constexpr int NUA = BES_MODEL_NUA;
constexpr int NIUA = BES_MODEL_NIUA;
constexpr int NE = BES_MODEL_NE;
constexpr int NSP = BES_MODEL_NSP;
constexpr int NSA = BES_MODEL_NSA;
constexpr int NISA = BES_MODEL_NISA;
constexpr int IC = BES_MODEL_IMPLICIT_COMPONENT;
constexpr int NUPa = NUP > 0 ? NUP : 1;
constexpr int NUAa = NUA > 0 ? NUA : 1;
constexpr int NIUAa = NIUA > 0 ? NIUA : 1;
constexpr int NEa = NE > 0 ? NE : 1;
constexpr int NSPa = NSP > 0 ? NSP : 1;
constexpr int NSAa = NSA > 0 ? NSA : 1;
constexpr int NISAa = NISA > 0 ? NISA : 1;
constexpr unsigned FULL = 0xffffffffu;
/* one group-exchange buffer: two values per unit of the largest group
 * (128 units) and one flag word per warp, padded to 16-byte multiples */
constexpr int XCH_BUF = 2 * 128 + 8;
/* one buffer of warp_sum32, or one vector split by parity: the 16 even and the 16
 * odd units' values, each run padded by one double2 so that the two that a load
 * reads at once start in different banks */
constexpr int RED_RUN = 18, RED_BUF = 2 * RED_RUN;
/* shared memory a CTA can have */
constexpr int SMEM_MAX = 227 * 1024;
/* stage derivatives of a system of NMAX units (one unit per lane) that go to shared memory beside
 * `others` doubles, `systems` times in a CTA, if that fits: a model of many parameters or components
 * may leave no room, and then they are in local memory */
__host__ __device__ constexpr int stage_doubles(int nmax, long others, int systems = 1) {
    return 8L * systems * ((others + 6 * UD * nmax + 31) / 32 * 32) <= SMEM_MAX ? 6 * UD * nmax : 0;
}
/* warps of a team: one system of up to 32 units on TEAM warps (RHS > 10: the variant RHS - 10) */
constexpr int TEAM = 4;
/* Shared-memory doubles per system (G warps, U units per lane, NMAX = 32 U G
 * units): one matrix region (more than one unit per lane: the operator W, leading
 * dimension NMAX+1; one: the system's coupling matrix C, for one warp with the
 * part of W that A^T v reads), six broadcast vectors, the group's exchange buffers
 * (G > 1) or the warp's reduction buffers, the system-scope arrays, and the unit
 * parameters when each lane owns one unit (U = 1: in registers they crowd out
 * the BiCG state).  T: the warps of a team, each with such a region; 0: one warp,
 * its part of W in tensor memory. */
template <int U, int G = 1, int T = 1>
struct WarpSmem {
    static constexpr int NMAX = 32 * U * G;
    static constexpr bool ONE = U == 1 && G == 1;   /* one warp, one unit per lane */
    static constexpr int LDW = NMAX + 1;
    static constexpr int W_DOUBLES = U == 1 && G > 1 ? NMAX * NMAX : NMAX * LDW;
    static constexpr int VEC_DOUBLES = 6 * NMAX;
    static constexpr int XCH_DOUBLES = G > 1 ? 2 * XCH_BUF + 8 : 0; /* two buffers of two values per unit, vote words */
    static constexpr int SYS_DOUBLES = NSPa + NSAa + NISAa;  /* ints stored in double slots */
    static constexpr int RED_DOUBLES = ONE ? 4 * RED_BUF : 0;   /* warp_sum32's buffers, two vectors by parity */
    static constexpr int UP_DOUBLES = U == 1 ? NMAX * NUPa : 0; /* unit parameters (one unit per lane) */
    static constexpr int WT_DOUBLES = ONE && T == 1 ? NMAX * NMAX : 0;  /* each lane's column share of W */
    static constexpr int XT_DOUBLES = T > 1 ? 2 * T * 32 : 0;   /* a team's two exchange buffers (its first warp's are used) */
    static constexpr int OTHERS = W_DOUBLES + WT_DOUBLES + VEC_DOUBLES + XCH_DOUBLES + RED_DOUBLES + SYS_DOUBLES +
                                  UP_DOUBLES + XT_DOUBLES;
    static constexpr int K_DOUBLES = U == 1 ? stage_doubles(NMAX, OTHERS, T > 1 ? T : 1) : 0;   /* stage derivatives */
    /* per-system stride rounded up to 256 bytes: every system's vectors stay
     * 16-byte aligned for the double2 broadcast loads */
    static constexpr int DOUBLES = (OTHERS + K_DOUBLES + 31) / 32 * 32;
    static constexpr int BYTES = DOUBLES * 8;
    static_assert(DOUBLES % 2 == 0 && W_DOUBLES % 2 == 0 && NMAX % 2 == 0,
                  "broadcast vectors must start on 16-byte boundaries");
};

/* Shared-memory layout of the shared-matrix variants: with RHS = 3, or more than
 * one unit per lane, one padded copy of the launch's coupling matrix per CTA
 * (one unit per lane: leading dimension NMAX+1 for the quads; more: NMAX+2, rows
 * are read lane-consecutive, each lane's column is 16-byte aligned and its
 * double2 reads are conflict-free); the symmetric matrix of one-unit-per-lane
 * systems (RHS = 4) is in tensor memory.  Then per system five broadcast
 * vectors, the group's exchange buffers, the system-scope arrays, the unit
 * parameters and the stage derivatives. */
template <int U, int G, bool SYM>
struct SharedCSmem {
    static constexpr int NMAX = 32 * U * G;
    static constexpr bool TMEM = SYM && U == 1;
    static constexpr int LDC = U == 1 ? NMAX + 1 : NMAX + 2;   /* odd for the quads' 64-bit reads */
    static constexpr int C_DOUBLES = TMEM ? 0 : NMAX * LDC;
    static constexpr int XCH_DOUBLES = G > 1 ? 2 * XCH_BUF + 8 : 0;
    static constexpr int UP_DOUBLES = U == 1 ? NMAX * NUPa : 0; /* unit parameters (one unit per lane) */
    static constexpr int OTHERS = 5 * NMAX + XCH_DOUBLES + NSPa + NSAa + NISAa + UP_DOUBLES;
    static constexpr int K_DOUBLES = U == 1 ? stage_doubles(NMAX, C_DOUBLES + OTHERS) : 0;   /* stage derivatives */
    static constexpr int WARP_DOUBLES = (OTHERS + K_DOUBLES + 31) / 32 * 32;
    static constexpr int C_BYTES = C_DOUBLES * 8;
    static constexpr int WARP_BYTES = WARP_DOUBLES * 8;
    static_assert(C_DOUBLES % 2 == 0 && WARP_DOUBLES % 2 == 0, "16-byte alignment");
};

/* TMEM columns of a CTA of `warps` warps: RHS 4 keeps each lane's share of the
 * shared matrix once for all systems of the CTA (NMAX doubles a lane); RHS 0
 * keeps each system's row and column shares of W (2 NMAX doubles a lane), four
 * warps side by side in the four quarters; RHS 8 and 9 (at most four warps) each
 * warp's column share (32 doubles a lane).  0: the variant uses none. */
template <int U, int RHS, int G>
__host__ __device__ constexpr int tmem_columns(int warps) {
    return U == 1 && G == 1 && (RHS == 8 || RHS == 9) ? 64 : U != 1 || G == 1 ? 0 : RHS == 4 ? 2 * 32 * G : RHS == 0 ? 4 * 32 * G * ((warps + 3) / 4) : 0;
}

/* diagonals of the banded operator in registers; RHS 7 has no others */
constexpr int BAND_REGS = 8;

/* Shared-memory layout of the banded variants (RHS = 7 and 10, one unit per lane, G
 * warps, NMAX = 32 G units): per system the staged band of its coupling
 * matrix Cb[d][i] = C[i][(i + d - bw) mod N] and the operator by diagonal
 * Wb[d][i], ND = min(2 bw + 1, NMAX) diagonals each, then the six broadcast
 * vectors, the group's exchange buffers, the system-scope arrays and the unit
 * parameters.  The band width is a run-time value, so is the layout.  Narrow
 * bands add the stage derivatives; wide ones (RHS = 10) need the room: with the
 * derivatives' 12 KB a system of 128 units does not fit beyond bw = 45 (48
 * without), and two share an SM up to bw = 17 (20 without). */
template <int G, bool WIDE>
struct BandSmem {
    static constexpr int NMAX = 32 * G;
    static constexpr int XCH_DOUBLES = G > 1 ? 2 * XCH_BUF + 8 : 0;
    static constexpr int RED_DOUBLES = G == 1 ? 2 * RED_BUF : 0;   /* warp_sum32's buffers */
    static constexpr int OTHERS = 6 * NMAX + XCH_DOUBLES + RED_DOUBLES + NSPa + NSAa + NISAa + NMAX * NUPa;
    static constexpr int K_DOUBLES = WIDE ? 0 : stage_doubles(NMAX, 2 * (BAND_REGS - 1) * NMAX + OTHERS);   /* stage derivatives */
    __host__ __device__ static constexpr int diagonals(int bw) { return 2 * bw + 1 < NMAX ? 2 * bw + 1 : NMAX; }
    __host__ __device__ static constexpr int doubles(int bw) {
        return (2 * diagonals(bw) * NMAX + OTHERS + K_DOUBLES + 31) / 32 * 32;
    }
};

/* a compile-time constant as a function argument */
template <int V>
struct Const {
    static constexpr int value = V;
};

/* halving-tree sum S(L, i) = S(2L, i) + S(2L, i + L), S(P, i) = leaf(i) */
template <int L, int P>
struct TreeSum {
    template <class Leaf>
    __device__ __forceinline__ static double run(int i, const Leaf& leaf) {
        return TreeSum<2 * L, P>::run(i, leaf) + TreeSum<2 * L, P>::run(i + L, leaf);
    }
};
template <int P>
struct TreeSum<P, P> {
    template <class Leaf>
    __device__ __forceinline__ static double run(int i, const Leaf& leaf) { return leaf(i); }
};

/* Sum over all 32U units of the warp in halving-tree order; every lane gets it. */
template <int U>
__device__ __forceinline__ double warp_tree_sum(const double (&v)[U]) {
    double a[U];
#pragma unroll
    for (int m = 0; m < U; m++) a[m] = v[m];
#pragma unroll
    for (int h = U / 2; h >= 1; h /= 2)
#pragma unroll
        for (int m = 0; m < h; m++) a[m] = a[m] + a[m + h];
    double s = a[0];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s = s + __shfl_xor_sync(FULL, s, o);
    return s;
}

/* Minimum over the warp, NaN ignored unless every value is NaN (as a tree of fmin): the bits
 * as unsigned integers in the doubles' order, the high words' minimum first, then the low words'
 * among the lanes that hold it -- two integer reductions (22 cycles each on a B200) for five
 * levels of shuffles and fmin (56 each). */
__device__ __forceinline__ double warp_min(double s) {
    const unsigned hi = (unsigned)__double2hiint(s), lo = (unsigned)__double2loint(s);
    const unsigned flip = (unsigned)((int)hi >> 31);
    const bool nan = s != s;
    const unsigned kh = nan ? 0xffffffffu : hi ^ (flip | 0x80000000u), kl = nan ? 0xffffffffu : lo ^ flip;
    const unsigned mh = __reduce_min_sync(FULL, kh);
    const unsigned ml = __reduce_min_sync(FULL, kh == mh ? kl : 0xffffffffu);
    const unsigned back = mh & 0x80000000u ? 0u : 0xffffffffu;
    return __hiloint2double((int)(mh ^ (back | 0x80000000u)), (int)(ml ^ back));
}

/* one warp's view of its system: the system runs on G warps (wis = this
 * warp's index among them); slot m of lane l is unit 32 (G m + wis) + l */
template <int U, int G = 1>
struct Sys {
    int lane, sid, N, wis;
    unsigned bar;      /* named barrier of the system's G warps (G > 1) */
    int64_t off, tot;
    const double* C;   /* the system's coupling matrix in HBM */
    double* W;         /* matrix region in shared memory: W, or a padded copy of C */
    double *vp, *vpt, *vcpt, *vx1, *vxu, *vrd;
    double* upsh;      /* unit parameters of the register-operator variant: unit i at upsh[i * NUP] */
    double* xch;       /* the group's exchange buffers (G > 1), or warp_sum32's (U = G = 1) */
    double *tpar, *rdpar;   /* vectors split by parity (register-operator variants): entry i at par_slot(i) */
    int tw;            /* this warp's place in its team (T > 1), else 0 */
    bool lead;         /* the warp that writes the system's results: a team's first, else every warp */
    double* xt;        /* the team's exchange buffers */
    mutable int tsel;  /* which of them is next */
    uint32_t tm;       /* this warp's lanes of the system's (RHS 0) or the CTA's (RHS 4) columns in tensor memory */
    double* flag;      /* the group's exit-vote words, one per warp (G > 1) */
    mutable int xsel;  /* which of the two exchange (or warp_sum32) buffers is next */
    double* ks;        /* stage derivatives (U = 1): entry j, component c of unit i at ks[(j * UD + c) * 32 U G + i] */
    double* sPAR;
    double* sACC;
    int* isACC;
    double* gPAR;
    int* igPAR;
    __device__ __forceinline__ int unit(int m) const { return 32 * (G * m + wis) + lane; }
};

/* ---------------------------------------------------------------------------
 * Group primitives: with G = 1 they are the warp's own shuffles and votes;
 * with G > 1 each call writes this warp's values into one of two exchange
 * buffers, crosses one named barrier and reads every warp's values back (the
 * two buffers alternate, so a buffer is rewritten only after a later barrier
 * that every reader of its previous contents has passed).  All G warps of a
 * system make the same sequence of calls: their control flow is identical
 * because every decision comes out of these reductions. */
template <int U, int G>
__device__ __forceinline__ void grp_sync(const Sys<U, G>& S) {
    if constexpr (G == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(S.bar), "r"(32 * G) : "memory");
}

template <int U, int G>
__device__ __forceinline__ double* grp_buffer(const Sys<U, G>& S) {
    static_assert(2 * 32 * U * G + G <= XCH_BUF, "exchange buffer too small");
    double* b = S.xch + (S.xsel & 1) * XCH_BUF;
    S.xsel++;
    return b;
}

/* slot of unit i in a vector split by parity: 16 even entries, then 16 odd ones */
__device__ __forceinline__ int par_slot(int i) { return (i & 1) * RED_RUN + (i >> 1); }

/* Sum over the 32 units of a one-warp system in halving-tree order, every lane
 * gets it.  The tree splits into its even and its odd lanes' subtrees until its
 * last addition, so lane l reads the 16 values of its own parity from shared
 * memory (8 double2 loads, two addresses a load), adds them in tree order and
 * meets the other parity in one shuffle: 144 cycles against the five-level
 * butterfly's 176 on a B200 (a 64-bit shuffle and its addition take 35).  The
 * two buffers alternate: one is rewritten only after a later call's barrier,
 * which every reader of its previous contents has reached. */
__device__ __forceinline__ double warp_sum32(const Sys<1, 1>& S, double v) {
    double* buf = S.xch + (S.xsel & 1) * RED_BUF;
    S.xsel++;
    buf[par_slot(S.lane)] = v;
    __syncwarp();
    const double2* mine = reinterpret_cast<const double2*>(buf + (S.lane & 1) * RED_RUN);
    double a[16];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const double2 t = mine[k];
        a[2 * k] = t.x;
        a[2 * k + 1] = t.y;
    }
    auto leaf = [&](int k) -> double { return a[k]; };
    const double s = TreeSum<1, 16>::run(0, leaf);
    return s + __shfl_xor_sync(FULL, s, 1);
}

/* a[k][b]: value k of this lane's unit in block b = G m + wis, for all U G blocks */
template <int U, int G, int K>
__device__ __forceinline__ void grp_gather(const Sys<U, G>& S, const double (&v)[K][U], double (&a)[K][U * G]) {
    if constexpr (G == 1) {
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
            for (int m = 0; m < U; m++) a[k][m] = v[k][m];
    } else {
        double* buf = grp_buffer(S);
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
            for (int m = 0; m < U; m++) buf[k * 32 * U * G + (G * m + S.wis) * 32 + S.lane] = v[k][m];
        grp_sync(S);
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
            for (int b = 0; b < U * G; b++) a[k][b] = buf[k * 32 * U * G + b * 32 + S.lane];
    }
}

/* Sum over all units of the system in halving-tree order (blocks of 32 first,
 * then the lanes); every lane of every warp of the system gets it. */
template <int U, int G>
__device__ __forceinline__ double grp_tree_sum(const Sys<U, G>& S, const double (&v)[U]) {
    if constexpr (U == 1 && G == 1) {
        return warp_sum32(S, v[0]);
    } else {
        double in[1][U], a[1][U * G];
#pragma unroll
        for (int m = 0; m < U; m++) in[0][m] = v[m];
        grp_gather<U, G, 1>(S, in, a);
        return warp_tree_sum<U * G>(a[0]);
    }
}

/* BiCG exit test and next rho in one exchange: returns whether the fmax-tree
 * maximum of x over the system's units is below lim, and sets ysum to the
 * halving-tree sum of y.  The fmax tree ignores NaN unless every value is
 * NaN, so "max < lim" is exactly "every non-NaN value is below lim and at
 * least one value is not NaN"; two warp votes decide it without a max tree. */
template <int U, int G>
__device__ __forceinline__ bool grp_sum_max_below(const Sys<U, G>& S, const double (&x)[U], const double (&y)[U],
                                                  double lim, double& ysum) {
    bool ok = true, seen = false;
#pragma unroll
    for (int m = 0; m < U; m++) {
        ok = ok && (isnan(x[m]) || x[m] < lim);
        seen = seen || !isnan(x[m]);
    }
    const bool wok = __all_sync(FULL, ok), wseen = __any_sync(FULL, seen);
    if constexpr (G == 1) {
        ysum = grp_tree_sum<U, G>(S, y);
        return wok && wseen;
    } else {
        /* the sum's blocks and one flag word per warp share one exchange buffer */
        double* buf = grp_buffer(S);
        constexpr int NB = U * G;
#pragma unroll
        for (int m = 0; m < U; m++) buf[(G * m + S.wis) * 32 + S.lane] = y[m];
        if (S.lane == 0) buf[32 * NB + S.wis] = (wok ? 1.0 : 0.0) + (wseen ? 2.0 : 0.0);
        grp_sync(S);
        double a[NB];
#pragma unroll
        for (int b = 0; b < NB; b++) a[b] = buf[b * 32 + S.lane];
        ysum = warp_tree_sum<NB>(a);
        bool all_ok = true, any_seen = false;
#pragma unroll
        for (int w = 0; w < G; w++) {
            const double f = buf[32 * NB + w];
            all_ok = all_ok && (f == 1.0 || f == 3.0);
            any_seen = any_seen || f >= 2.0;
        }
        return __all_sync(FULL, all_ok && any_seen);
    }
}

/* one warp-uniform value per warp to all G warps: out[w] */
template <int U, int G>
__device__ __forceinline__ void grp_share(const Sys<U, G>& S, double v, double (&out)[G]) {
    if constexpr (G == 1) {
        out[0] = v;
    } else {
        double* buf = grp_buffer(S);
        if (S.lane == 0) buf[S.wis] = v;
        grp_sync(S);
#pragma unroll
        for (int w = 0; w < G; w++) out[w] = buf[w];
    }
}

template <int U, int G>
__device__ __forceinline__ double grp_min(const Sys<U, G>& S, double s) {
    s = warp_min(s);
    double w[G];
    grp_share(S, s, w);
#pragma unroll
    for (int k = 1; k < G; k++) w[0] = fmin(w[0], w[k]);
    return w[0];
}

/* What the step controller needs of all units, in one exchange: whether every
 * a and every b holds, whether any c does, and the minimum of s. */
template <int U, int G>
__device__ __forceinline__ void grp_step_votes(const Sys<U, G>& S, bool& a, bool& b, bool& c, double& s) {
    a = __all_sync(FULL, a);
    b = __all_sync(FULL, b);
    c = __any_sync(FULL, c);
    s = warp_min(s);
    if constexpr (G > 1) {
        double* buf = grp_buffer(S);
        if (S.lane == 0) {
            buf[2 * S.wis] = __hiloint2double(0, (a ? 0 : 1) + (b ? 0 : 2) + (c ? 4 : 0));
            buf[2 * S.wis + 1] = s;
        }
        grp_sync(S);
        int f = 0;
#pragma unroll
        for (int w = 0; w < G; w++) {
            f |= __double2loint(buf[2 * w]);
            s = w == 0 ? buf[1] : fmin(s, buf[2 * w + 1]);
        }
        a = __all_sync(FULL, (f & 1) == 0);
        b = __all_sync(FULL, (f & 2) == 0);
        c = __all_sync(FULL, (f & 4) != 0);
    }
}

template <int U, int G>
__device__ __forceinline__ bool grp_all(const Sys<U, G>& S, bool p) {
    if constexpr (G == 1) {
        return __all_sync(FULL, p);
    } else {
        double w[G];
        grp_share(S, __all_sync(FULL, p) ? 1.0 : 0.0, w);
        bool r = true;
#pragma unroll
        for (int k = 0; k < G; k++) r = r && w[k] != 0.0;
        return __all_sync(FULL, r);
    }
}

template <int U, int G>
__device__ __forceinline__ bool grp_any(const Sys<U, G>& S, bool p) {
    if constexpr (G == 1) {
        return __any_sync(FULL, p);
    } else {
        double w[G];
        grp_share(S, __any_sync(FULL, p) ? 1.0 : 0.0, w);
        bool r = false;
#pragma unroll
        for (int k = 0; k < G; k++) r = r || w[k] != 0.0;
        return __all_sync(FULL, r);
    }
}

/* A callback may change a system-scope scalar through its reference argument
 * (the reference's shared variables).  Units see the value from before the
 * callback round; afterwards the lowest unit that changed it wins
 * (first_unit: the lowest unit of this lane that changed it, or -1). */
template <int U, int G>
__device__ __forceinline__ double grp_resolve(const Sys<U, G>& S, double before, double after_lane, int first_unit) {
    const unsigned int best = __reduce_min_sync(FULL, (unsigned int)first_unit);
    const double val = __shfl_sync(FULL, after_lane, (int)(best & 31u));
    double keys[G], vals[G];
    grp_share(S, (double)best, keys);
    grp_share(S, val, vals);
    double kmin = keys[0], v = vals[0];
#pragma unroll
    for (int w = 1; w < G; w++)
        if (keys[w] < kmin) { kmin = keys[w]; v = vals[w]; }
    return kmin == 4294967295.0 ? before : v;
}

template <int U, int G>
__device__ __forceinline__ int grp_resolve_int(const Sys<U, G>& S, int before, int after_lane, int first_unit) {
    return (int)grp_resolve<U, G>(S, (double)before, (double)after_lane, first_unit);
}

/* Two sums over all 32U units of the warp, each in halving-tree order (the
 * shuffles of the two butterflies interleave); every lane gets both.  One sum is
 * shorter through shared memory (warp_sum32), two are not: 300 systems of 32
 * units with their own matrices, 250 steps with REC 1, 5.94 ms so and 5.55 with
 * the butterflies. */
template <int U>
__device__ __forceinline__ void warp_tree_sum2(const double (&v)[U], const double (&w)[U], double& sv, double& sw) {
    double a[U], b[U];
#pragma unroll
    for (int m = 0; m < U; m++) { a[m] = v[m]; b[m] = w[m]; }
#pragma unroll
    for (int h = U / 2; h >= 1; h /= 2)
#pragma unroll
        for (int m = 0; m < h; m++) { a[m] = a[m] + a[m + h]; b[m] = b[m] + b[m + h]; }
    double s = a[0], t = b[0];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const double so = __shfl_xor_sync(FULL, s, o), to = __shfl_xor_sync(FULL, t, o);
        s = s + so;
        t = t + to;
    }
    sv = s;
    sw = t;
}

/* two sums over the system's units in one group exchange (each bit-identical to grp_tree_sum) */
template <int U, int G>
__device__ __forceinline__ void grp_tree_sum2(const Sys<U, G>& S, const double (&v)[U], const double (&w)[U],
                                              double& sv, double& sw) {
    if constexpr (G == 1) {
        warp_tree_sum2<U>(v, w, sv, sw);
    } else {
        double in[2][U], a[2][U * G];
#pragma unroll
        for (int m = 0; m < U; m++) { in[0][m] = v[m]; in[1][m] = w[m]; }
        grp_gather<U, G, 2>(S, in, a);
        warp_tree_sum2<U * G>(a[0], a[1], sv, sw);
    }
}

/* the BiCG exit test alone: fmax-tree maximum of x over the system below lim
 * (same decision and NaN rule as grp_sum_max_below) */
template <int U, int G>
__device__ __forceinline__ bool grp_max_below(const Sys<U, G>& S, const double (&x)[U], double lim) {
    bool ok = true, seen = false;
#pragma unroll
    for (int m = 0; m < U; m++) {
        ok = ok && (isnan(x[m]) || x[m] < lim);
        seen = seen || !isnan(x[m]);
    }
    const bool wok = __all_sync(FULL, ok), wseen = __any_sync(FULL, seen);
    if constexpr (G == 1) {
        return wok && wseen;
    } else {
        double f[G];
        grp_share(S, (wok ? 1.0 : 0.0) + (wseen ? 2.0 : 0.0), f);
        bool all_ok = true, any_seen = false;
#pragma unroll
        for (int w = 0; w < G; w++) {
            all_ok = all_ok && (f[w] == 1.0 || f[w] == 3.0);
            any_seen = any_seen || f[w] >= 2.0;
        }
        return all_ok && any_seen;
    }
}

/* The exit test of a multi-warp group, folded into a barrier the group crosses
 * anyway: each warp posts its votes in its flag word before that barrier, and
 * after it every warp reads all flags.  The flag words are rewritten only
 * after a later group exchange, which every reader of the current flags passes
 * after reading them. */
template <int U, int G>
__device__ __forceinline__ void grp_post_max_below(const Sys<U, G>& S, const double (&x)[U], double lim) {
    bool ok = true, seen = false;
#pragma unroll
    for (int m = 0; m < U; m++) {
        ok = ok && (isnan(x[m]) || x[m] < lim);
        seen = seen || !isnan(x[m]);
    }
    const bool wok = __all_sync(FULL, ok), wseen = __any_sync(FULL, seen);
    if (S.lane == 0) S.flag[S.wis] = (wok ? 1.0 : 0.0) + (wseen ? 2.0 : 0.0);
}

template <int U, int G>
__device__ __forceinline__ bool grp_read_max_below(const Sys<U, G>& S) {
    bool all_ok = true, any_seen = false;
#pragma unroll
    for (int w = 0; w < G; w++) {
        const double f = S.flag[w];
        all_ok = all_ok && (f == 1.0 || f == 3.0);
        any_seen = any_seen || f >= 2.0;
    }
    return __all_sync(FULL, all_ok && any_seen);
}

/* ---------------------------------------------------------------------------
 * BiCG iterations (Steppers.cuh:508-561) on a system whose residual r
 * (r~ = r) and start x are set.  put(v, vt) posts this lane's entries of v and
 * vt for the other lanes, mul(v, vt, q, qt) -- after a grp_sync -- forms
 * q = A v and q~ = A^T vt, zero for slots beyond the system's units.  A put
 * needs no barrier before it when a group exchange lies between it and the last
 * read of the posted vectors (every reader is past its reads there); a single
 * warp's __syncwarp costs nothing and stays.
 *
 * REC = 0: the reference's recurrence -- per iteration the products of the
 * search directions, then alpha from one reduction and the exit test with the
 * next rho from a second.
 * REC = 1: the single-reduction form of the same iterates.  The products of
 * the residuals w = A r, w~ = A^T r~ come first; rho = r.r~ needs no product
 * and mu = r~.w does; then
 *   beta = rho / rho_prev, sigma = mu - beta^2 sigma_prev,
 *   p = r + beta p, p~ = r~ + beta p~, q = w + beta q, q~ = w~ + beta q~,
 *   alpha = rho / sigma,
 * so q = A p, q~ = A^T p~ and sigma = p~.A p (its cross terms equal
 * -rho/alpha_prev = -beta sigma_prev each, by the biorthogonality of the
 * residuals).  Same exits as the reference (|rho| < 1e-6 before the first
 * update, max |r| < 1e-6 after each, at most bicg_max_iter updates).  A single
 * warp tests the exit by votes right after the update; a group posts each
 * warp's votes with the residuals it puts for the next product, so the test
 * costs no barrier of its own.
 *
 * An iteration is one dependency chain on one warp and is bound by its length
 * and its instruction count.  Both quotients of either recurrence go on as
 * Markstein's and are proven at the end of the iteration, together with the
 * exit test, so the loop has one branch (a proof's comparison and branch on the
 * chain cost 60 cycles each, twice an iteration).  With an unproven one the
 * update is dropped and done with IEEE divisions.  The iteration is repeated for
 * that, but with REC 1, whose products do not need the quotients, a single warp
 * repeats the update only: a second copy of the iteration beside the loop cost
 * it registers (700 systems of 31 units 11.5 -> 10.7 ms without), while the
 * kernels of 128 registers lose by keeping the products until the proof (1200
 * systems of 64 units with a shared matrix: 13.3 ms, 13.8 so).
 * IN_PLACE: several units a lane have no registers for a second set of iterates
 * (148 systems of 128 units on one warp, own matrices: 292 -> 205 ms without
 * it), so each quotient is settled before it is used and the iterates are
 * updated in place.  With a shared matrix REC 0 is faster with the second set
 * all the same (239 ms, 250 in place).
 * Returns the completed iterations; sets capped when the cap ended the loop. */
template <int U, int G, int REC, bool IN_PLACE = false, class Put, class Mul>
__device__ __forceinline__ int bicg_iterate(const Sys<U, G>& S, const DeviceProblem& P, const double (&b)[U],
                                            double (&r)[U], double (&x)[U], Put&& put, Mul&& mul, bool& capped) {
    static_assert(!IN_PLACE || G == 1, "updates in place are for one warp");
    double rt[U], p[U], pt[U], ar[U];
    const int max_iter = P.bicg_max_iter;
#pragma unroll
    for (int m = 0; m < U; m++) { rt[m] = r[m]; p[m] = 0.0; pt[m] = 0.0; ar[m] = 0.0; }
    int done = 0;
    bool exited = false;
    auto reference_recurrence = [&]() {
        double prod[U], q[U], qt[U];
#pragma unroll
        for (int m = 0; m < U; m++) prod[m] = r[m] * rt[m];
        double rho1 = grp_tree_sum<U, G>(S, prod);
        if (max_iter < 1) return;
        if (__all_sync(FULL, fabs(rho1) < 1e-6)) { exited = true; return; }
        double rho2 = 1.0, y2 = 1.0;   /* y2: reciprocal estimate of rho2, formed an iteration early */
        if constexpr (IN_PLACE) {
            for (int it = 1; it <= max_iter; it++) {
                const double beta = it == 1 ? 0.0 : math::div_known(rho1, rho2, y2);   /* = rho1 / rho2; p = r first */
#pragma unroll
                for (int m = 0; m < U; m++) {
                    p[m] = fma(beta, p[m], r[m]);
                    pt[m] = fma(beta, pt[m], rt[m]);
                }
                __syncwarp();
                put(p, pt);
                __syncwarp();
                rho2 = rho1;
                y2 = math::recip_estimate(rho2);
                mul(p, pt, q, qt);
#pragma unroll
                for (int m = 0; m < U; m++) prod[m] = pt[m] * q[m];
                const double sig = grp_tree_sum<U, G>(S, prod);
                const double alpha = math::div_known(rho2, sig, math::recip_estimate(sig));   /* = rho / sigma */
#pragma unroll
                for (int m = 0; m < U; m++) {
                    x[m] = fma(alpha, p[m], x[m]);
                    r[m] = fma(-alpha, q[m], r[m]);
                    rt[m] = fma(-alpha, qt[m], rt[m]);
                    ar[m] = fabs(r[m]);
                    prod[m] = r[m] * rt[m];
                }
                done++;
                if (grp_sum_max_below<U, G>(S, ar, prod, 1e-6, rho1)) { exited = true; break; }
            }
            return;
        }
        double pn[U], ptn[U], xn[U], rn[U], rtn[U], rho_next, y1;
        bool small, proven;
        int it = 0;   /* committed iterations of this solve (done counts a redone solve's too) */
        /* one iteration into pn .. rtn, rho_next and small: nothing is committed */
        auto iteration = [&](auto ieee) {
            bool beta_ok, alpha_ok;
            double beta = decltype(ieee)::value ? math::div_ieee(rho1, rho2)
                                                : math::div_markstein(rho1, rho2, y2, beta_ok);   /* = rho1 / rho2 */
            if (it == 0) { beta = 0.0; beta_ok = true; }   /* p = r */
#pragma unroll
            for (int m = 0; m < U; m++) {
                pn[m] = fma(beta, p[m], r[m]);
                ptn[m] = fma(beta, pt[m], rt[m]);
            }
            if constexpr (G == 1) __syncwarp();
            put(pn, ptn);
            grp_sync(S);
            y1 = math::recip_estimate(rho1);   /* becomes y2 with the commit */
            mul(pn, ptn, q, qt);
#pragma unroll
            for (int m = 0; m < U; m++) prod[m] = ptn[m] * q[m];
            const double sig = grp_tree_sum<U, G>(S, prod);
            const double alpha = decltype(ieee)::value
                                     ? math::div_ieee(rho1, sig)
                                     : math::div_markstein(rho1, sig, math::recip_estimate(sig), alpha_ok);   /* = rho1 / sig */
#pragma unroll
            for (int m = 0; m < U; m++) {
                xn[m] = fma(alpha, pn[m], x[m]);
                rn[m] = fma(-alpha, q[m], r[m]);
                rtn[m] = fma(-alpha, qt[m], rt[m]);
                ar[m] = fabs(rn[m]);
                prod[m] = rn[m] * rtn[m];
            }
            small = grp_sum_max_below<U, G>(S, ar, prod, 1e-6, rho_next);
            proven = decltype(ieee)::value || __all_sync(FULL, beta_ok && alpha_ok);
        };
        auto commit = [&]() {
#pragma unroll
            for (int m = 0; m < U; m++) { p[m] = pn[m]; pt[m] = ptn[m]; x[m] = xn[m]; r[m] = rn[m]; rt[m] = rtn[m]; }
            rho2 = rho1;
            y2 = y1;
            rho1 = rho_next;
            it++;
            done++;
        };
        for (;;) {
            for (;;) {
                iteration(Const<0>{});
                if (!proven || small || it + 1 >= max_iter) break;
                commit();
            }
            if (!proven) iteration(Const<1>{});
            commit();
            exited = small;
            if (small || it >= max_iter) break;
        }
    };
    if constexpr (REC == 0) {
        reference_recurrence();
    } else {
        double r0[U], x0[U];
#pragma unroll
        for (int m = 0; m < U; m++) { r0[m] = r[m]; x0[m] = x[m]; }
        double w[U], wt[U], rw[U], prod[U], q[U], qt[U];
#pragma unroll
        for (int m = 0; m < U; m++) { q[m] = 0.0; qt[m] = 0.0; }
        double sigma = 0.0, rho_prev = 1.0, y_prev = 1.0;   /* y_prev: reciprocal estimate of rho_prev */
        if constexpr (IN_PLACE) {
            for (int it = 1; it <= max_iter; it++) {
                __syncwarp();
                put(r, rt);
                __syncwarp();
                mul(r, rt, w, wt);
#pragma unroll
                for (int m = 0; m < U; m++) { prod[m] = r[m] * rt[m]; rw[m] = rt[m] * w[m]; }
                double rho, mu;
                grp_tree_sum2<U, G>(S, prod, rw, rho, mu);
                if (it == 1 && __all_sync(FULL, fabs(rho) < 1e-6)) { exited = true; break; }
                const double beta = it == 1 ? 0.0 : math::div_known(rho, rho_prev, y_prev);   /* = rho / rho_prev */
                sigma = fma(-(beta * beta), sigma, mu);
                const double alpha = math::div_known(rho, sigma, math::recip_estimate(sigma));   /* = rho / sigma */
                rho_prev = rho;
                y_prev = math::recip_estimate(rho);
#pragma unroll
                for (int m = 0; m < U; m++) {
                    p[m] = fma(beta, p[m], r[m]);
                    pt[m] = fma(beta, pt[m], rt[m]);
                    q[m] = fma(beta, q[m], w[m]);
                    qt[m] = fma(beta, qt[m], wt[m]);
                    x[m] = fma(alpha, p[m], x[m]);
                    r[m] = fma(-alpha, q[m], r[m]);
                    rt[m] = fma(-alpha, qt[m], rt[m]);
                    ar[m] = fabs(r[m]);
                }
                done++;
                if (grp_max_below<U, G>(S, ar, 1e-6)) { exited = true; break; }
            }
        }
        double rho, mu, sg, y1, pn[U], ptn[U], qn[U], qtn[U], xn[U], rn[U], rtn[U];
        bool small = false, proven = true, early = false;
        /* the iterates pn .. rtn that the quotients lead to, and a single warp's exit test on them */
        auto update = [&](double beta, double alpha) {
#pragma unroll
            for (int m = 0; m < U; m++) {
                pn[m] = fma(beta, p[m], r[m]);
                ptn[m] = fma(beta, pt[m], rt[m]);
                qn[m] = fma(beta, q[m], w[m]);
                qtn[m] = fma(beta, qt[m], wt[m]);
                xn[m] = fma(alpha, pn[m], x[m]);
                rn[m] = fma(-alpha, qn[m], r[m]);
                rtn[m] = fma(-alpha, qtn[m], rt[m]);
                ar[m] = fabs(rn[m]);
            }
            if constexpr (G == 1) small = grp_max_below<U, G>(S, ar, 1e-6);
        };
        /* one iteration into pn .. rtn and sg: nothing is committed */
        auto iteration = [&](auto ieee) {
            if (G == 1 || done == 0) grp_sync(S);
            put(r, rt);
            if constexpr (G > 1) {
                if (done > 0 && !decltype(ieee)::value) grp_post_max_below<U, G>(S, ar, 1e-6);
            }
            grp_sync(S);
            if constexpr (G > 1) {
                early = done > 0 && !decltype(ieee)::value && grp_read_max_below<U, G>(S);
                if (early) return;
            }
#pragma unroll
            for (int m = 0; m < U; m++) prod[m] = r[m] * rt[m];
            mul(r, rt, w, wt);
#pragma unroll
            for (int m = 0; m < U; m++) rw[m] = rt[m] * w[m];
            grp_tree_sum2<U, G>(S, prod, rw, rho, mu);
            bool beta_ok, alpha_ok;
            double beta = decltype(ieee)::value ? math::div_ieee(rho, rho_prev)
                                                : math::div_markstein(rho, rho_prev, y_prev, beta_ok);   /* = rho / rho_prev */
            if (done == 0) { beta = 0.0; beta_ok = true; }   /* p = r */
            sg = fma(-(beta * beta), sigma, mu);
            const double alpha = decltype(ieee)::value
                                     ? math::div_ieee(rho, sg)
                                     : math::div_markstein(rho, sg, math::recip_estimate(sg), alpha_ok);   /* = rho / sigma */
            y1 = math::recip_estimate(rho);
            update(beta, alpha);
            proven = decltype(ieee)::value || __all_sync(FULL, beta_ok && alpha_ok);
            early = done == 0 && __all_sync(FULL, fabs(rho) < 1e-6);   /* the first rho test: the update is dropped */
        };
        auto commit = [&]() {
#pragma unroll
            for (int m = 0; m < U; m++) {
                p[m] = pn[m]; pt[m] = ptn[m]; q[m] = qn[m]; qt[m] = qtn[m];
                x[m] = xn[m]; r[m] = rn[m]; rt[m] = rtn[m];
            }
            sigma = sg;
            rho_prev = rho;
            y_prev = y1;
            done++;
        };
        if (!IN_PLACE && max_iter >= 1) {
            for (;;) {
                for (;;) {
                    iteration(Const<0>{});
                    if (early || !proven || small || done + 1 >= max_iter) break;
                    commit();
                }
                if (early) { exited = true; break; }
                if (!proven) {
                    if constexpr (G == 1) {   /* the products, rho and mu stand */
                        const double beta = done == 0 ? 0.0 : math::div_ieee(rho, rho_prev);
                        sg = fma(-(beta * beta), sigma, mu);
                        update(beta, math::div_ieee(rho, sg));
                    } else {
                        iteration(Const<1>{});   /* the previous update's exit test is not repeated */
                    }
                }
                commit();
                exited = small;
                if (small || done >= max_iter) break;
            }
        }
        if constexpr (G > 1) {
            /* the update that used up the cap has not been tested yet */
            if (!exited && done > 0 && done == max_iter && grp_max_below<U, G>(S, ar, 1e-6)) exited = true;
        }
        /* Safeguard: q is a recurrence, not a product, so r can drift from the
         * true residual (and sigma can collapse).  The solution stands when every
         * x is finite and the true residual b - A x passes the reference's exit
         * test, or when the first rho test ended the solve (x = x_u, as in the
         * reference's recurrence); otherwise the solve is redone from the start
         * with the reference's recurrence. */
        bool accept = exited;
        if (accept) {
            bool fin = true;
#pragma unroll
            for (int m = 0; m < U; m++) fin = fin && isfinite(x[m]);
            accept = grp_all<U, G>(S, fin);
        }
        if (accept && done > 0) {
            double ax[U], unused[U], zero[U], tr[U];
#pragma unroll
            for (int m = 0; m < U; m++) zero[m] = 0.0;
            if constexpr (G == 1) __syncwarp();
            put(x, zero);
            grp_sync(S);
            mul(x, zero, ax, unused);
#pragma unroll
            for (int m = 0; m < U; m++) tr[m] = fabs(b[m] - ax[m]);
            accept = grp_max_below<U, G>(S, tr, 1e-6);
        }
        if (!accept) {
            exited = false;
#pragma unroll
            for (int m = 0; m < U; m++) { r[m] = r0[m]; rt[m] = r0[m]; x[m] = x0[m]; p[m] = 0.0; pt[m] = 0.0; }
            reference_recurrence();
        }
    }
    if (!exited) capped = true;
    return done;
}

/* ---------------------------------------------------------------------------
 * Work split of the products of multi-warp systems (one unit per lane, matrix in
 * shared memory, M[i][j] at i + j LD with LD odd).  Warp w owns 32 rows; lane
 * l = 4r + c of it takes the four rows 4r .. 4r + 3 and of each the columns of
 * chain c (j = 4t + c), so an entry of a posted vector is loaded for four rows.
 * The four lanes of a quad then exchange their partial sums (three shuffles a
 * vector) and lane l keeps row l.  Both directions read 64-bit words of 32
 * different banks: 4r + c LD along rows, c + 4r LD along columns.
 *
 * A sub-partition fills registers from shared memory at 64 to 80 bytes a clock,
 * which bounds these products; with one row a lane the posted vectors were two
 * thirds of those bytes (N = 128, two vectors: 128 + 2 x 128 words a lane and
 * product, now 128 + 2 x 32), and loops of four guarded columns exposed every
 * load's latency.  Cycles per BiCG iteration of a lone system
 * on a B200: own matrix, N = 101: 7710 -> 3610, N = 48: 4130 -> 1780; shared
 * symmetric matrix, N = 128: 3840 -> 2900, N = 51: 1950 -> 1740. */

/* s[i]: this lane's chain of row i.  Returns (s0 + s1) + (s2 + s3) of its own row.
 * M0, M1: the lane bits that hold c's two bits. */
template <int M0, int M1>
__device__ __forceinline__ double quad_chains(int c, const double (&s)[4]) {
    const bool odd = c & 1, high = c & 2;
    const double k0 = odd ? s[1] : s[0], k2 = odd ? s[3] : s[2], g0 = odd ? s[0] : s[1], g2 = odd ? s[2] : s[3];
    const double a0 = k0 + __shfl_xor_sync(FULL, g0, M0), a2 = k2 + __shfl_xor_sync(FULL, g2, M0);
    return (high ? a2 : a0) + __shfl_xor_sync(FULL, high ? a0 : a2, M1);
}

/* s[i]: the halving subtree over the rows k = c (mod 4) of column i.  Returns the
 * whole tree (s0 + s2) + (s1 + s3) of this lane's own column. */
template <int M0, int M1>
__device__ __forceinline__ double quad_subtrees(int c, const double (&s)[4]) {
    const bool odd = c & 1, high = c & 2;
    const double k0 = high ? s[2] : s[0], k1 = high ? s[3] : s[1], g0 = high ? s[0] : s[2], g1 = high ? s[1] : s[3];
    const double a0 = k0 + __shfl_xor_sync(FULL, g0, M1), a1 = k1 + __shfl_xor_sync(FULL, g1, M1);
    return (odd ? a1 : a0) + __shfl_xor_sync(FULL, odd ? a0 : a1, M0);
}

/* sums of this lane's row of M against K posted vectors (columns j < N) */
template <int LD, int K>
__device__ __forceinline__ void quad_row_sums(const double* M, int row0, int c, int N, const double* const (&v)[K],
                                              double (&out)[K]) {
    double s[K][4];
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
        for (int i = 0; i < 4; i++) s[k][i] = 0.0;
    const double* m = M + row0 + c * LD;
    auto group = [&](int t) {
        double w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) w[i] = m[4 * t * LD + i];
#pragma unroll
        for (int k = 0; k < K; k++) {
            const double x = v[k][4 * t + c];
#pragma unroll
            for (int i = 0; i < 4; i++) s[k][i] = fma(w[i], x, s[k][i]);
        }
    };
    const int full = N >> 2;
#pragma unroll 8
    for (int t = 0; t < full; t++) group(t);
    if (c < (N & 3)) group(full);
#pragma unroll
    for (int k = 0; k < K; k++) out[k] = quad_chains<1, 2>(c, s[k]);
}

/* sum of this lane's column of M against a posted vector, halving tree over the NMAX rows (zero-padded) */
template <int NMAX, int LD>
__device__ __forceinline__ double quad_column_tree(const double* M, int col0, int c, const double* v) {
    double s[4];
    const double* m = M + col0 * LD + c;
    double x[NMAX / 4];
#pragma unroll
    for (int t = 0; t < NMAX / 4; t++) x[t] = v[4 * t + c];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        auto leaf = [&](int t) -> double { return m[i * LD + 4 * t] * x[t]; };
        s[i] = TreeSum<1, NMAX / 4>::run(0, leaf);
    }
    return quad_subtrees<1, 2>(c, s);
}

/* ---------------------------------------------------------------------------
 * The same split with the matrix in tensor memory.  Lane l = 8c + r takes the
 * rows r, r + 8, r + 16, r + 24 of its warp's 32 and the columns of chain c (the
 * eight lanes of a chain read one word of a posted vector, which shared memory
 * serves in one cycle a load), and keeps row l = r + 8c.  Its NMAX entries are
 * its own, so they sit in its TMEM lane, sixteen doubles a chunk: chunk k of the
 * row share holds the column groups t = 4k .. 4k + 3, four rows each; of the
 * column share the leaves 4k .. 4k + 3 of the halving tree, in bit-reversed
 * order of t, four columns each.  A chunk is loaded while the one before is
 * used; its latency is some 130 cycles, so chunks of eight doubles (40 cycles of
 * work) were slower than shared memory, and the loop is unrolled over all of
 * NMAX (guards on the chunks spilled registers).  Shared memory's 128 bytes a
 * clock were the bound before (N = 128: 1540 of the 2070 cycles of a product).
 * Cycles per BiCG iteration of a lone system on a B200: own matrix, N = 101:
 * 3610 -> 2040, N = 48: 1780 -> 1410; shared symmetric matrix, N = 128: 2900 ->
 * 1960 (two on an SM: 4290 -> 2660), N = 51: 1740 -> 1430. */

/* sums of this lane's row share against K posted vectors, entry j of vector k at v[K j + k]; all NMAX
 * columns are read, so the matrix and the vectors hold zeros from N to NMAX */
template <int K, int NMAX>
__device__ __forceinline__ void tmem_row_sums(uint32_t addr, int c, const double* v, double (&out)[K]) {
    double s[K][4];
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
        for (int i = 0; i < 4; i++) s[k][i] = 0.0;
    const double* vc = v + K * c;
    tmem::Chunk m[2];
    m[0].load(addr);
#pragma unroll
    for (int ch = 0; ch < NMAX / 16; ch++) {
        m[ch & 1].wait();
        if (ch + 1 < NMAX / 16) m[(ch + 1) & 1].load(addr + 32 * (ch + 1));
#pragma unroll
        for (int e = 0; e < 4; e++) {
            double x[K];
            if constexpr (K == 2) {
                const double2 p = *reinterpret_cast<const double2*>(vc + 8 * (4 * ch + e));
                x[0] = p.x;
                x[1] = p.y;
            } else {
                x[0] = vc[4 * (4 * ch + e)];
            }
#pragma unroll
            for (int k = 0; k < K; k++)
#pragma unroll
                for (int i = 0; i < 4; i++) s[k][i] = fma(m[ch & 1].get(4 * e + i), x[k], s[k][i]);
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++) out[k] = quad_chains<8, 16>(c, s[k]);
}

/* t of leaf m of the halving tree over T = 2^B column groups: m's bits reversed */
__host__ __device__ constexpr int tree_leaf(int m, int T) {
    int t = 0;
    for (int b = 1; b < T; b *= 2) t = 2 * t + (m / b) % 2;
    return t;
}

/* halving tree of this lane's column share against a posted vector, over all NMAX rows (zeros from N on) */
template <int NMAX>
__device__ __forceinline__ double tmem_column_tree(uint32_t addr, int c, const double* v) {
    constexpr int T = NMAX / 4, CH = T / 4;
    double part[CH][4];
    tmem::Chunk m[2];
    m[0].load(addr);
#pragma unroll
    for (int ch = 0; ch < CH; ch++) {
        m[ch & 1].wait();
        if (ch + 1 < CH) m[(ch + 1) & 1].load(addr + 32 * (ch + 1));
        double x[4];
#pragma unroll
        for (int e = 0; e < 4; e++) x[e] = v[4 * tree_leaf(4 * ch + e, T) + c];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            part[ch][i] = (m[ch & 1].get(i) * x[0] + m[ch & 1].get(4 + i) * x[1]) +
                          (m[ch & 1].get(8 + i) * x[2] + m[ch & 1].get(12 + i) * x[3]);
            /* join the subtrees that this chunk completes */
#pragma unroll
            for (int w = 1; w < CH; w *= 2)
                if ((ch + 1) % (2 * w) == 0) part[ch + 1 - 2 * w][i] = part[ch + 1 - 2 * w][i] + part[ch + 1 - w][i];
        }
    }
    return quad_subtrees<8, 16>(c, part[0]);
}

/* ---------------------------------------------------------------------------
 * Coupled right-hand side with the operator W in tensor memory and one unit
 * per lane on G warps (Steppers.cuh:432-562): a lane forms its row share and its
 * column share of W_ij = (rD_i C_ij) X1sq_j once per right-hand side from the
 * system's matrix, which is staged in shared memory once per system (zero-padded,
 * C[i][j] at (i ^ f(j)) + j NMAX with f(j) = j's low three bits reversed onto
 * bits 3, 2, 1: neither reads along rows nor along columns meet bank conflicts).
 * From L2 on every right-hand side the forming took 8080 cycles of a
 * 101-bubble system, now 4560. */
__device__ __forceinline__ int quad_swizzle(int j) { return ((j & 1) << 3) | ((j & 2) << 1) | ((j & 4) >> 1); }

template <int G, int REC>
__device__ __forceinline__ int coupled_rhs_quad(const Sys<1, G>& S, const DeviceProblem& P, double T,
                                                double (&Xs)[1][UD], double (&F)[1][UD], double (&ua)[1][NUAa],
                                                int (&iua)[1][NIUAa], bool& capped) {
    constexpr int NMAX = WarpSmem<1, G>::NMAX;
    const int N = S.N;
    const int i = S.unit(0);
    const bool valid = i < N;
    const int c = S.lane >> 3, r0 = S.lane & 7, row0 = 32 * S.wis + r0;
    double xu = 0.0, rd = 0.0;
    grp_sync(S);
    if (valid) {
        double Fl[UD], cpt, cpf;
        CoupledSystems_PerBlock_OdeFunction<double>(S.sid, i, Fl, Xs[0], T, S.upsh + i * NUPa, S.sPAR, S.gPAR,
                                                    S.igPAR, ua[0], iua[0], S.sACC, S.isACC, &cpt, &cpf);
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = Fl[k];
        xu = Fl[IC];
        rd = cpf;
        S.vcpt[i] = cpt;
        S.vx1[i] = Xs[0][0] * Xs[0][0];
        S.vxu[i] = xu;
    } else {
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = 0.0;
        S.vcpt[i] = 0.0;
        S.vx1[i] = 0.0;
        S.vxu[i] = 0.0;
    }
    S.vrd[i] = rd;
    grp_sync(S);
    /* b = rD (C CPT) + x_u, r = b - A x_u, and W (C and the posted vectors are zeros beyond N) */
    double bs[4] = {0.0, 0.0, 0.0, 0.0}, as[4] = {0.0, 0.0, 0.0, 0.0}, rd4[4], x14[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        rd4[k] = S.vrd[row0 + 8 * k];
        x14[k] = S.vx1[row0 + 8 * k];
    }
    const double* C = S.W;
    const int flip = quad_swizzle(c);
#pragma unroll 2
    for (int ch = 0; ch < NMAX / 16; ch++) {
        tmem::Chunk m;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int j = 16 * ch + 4 * e + c;
            const double x1 = S.vx1[j], cp = S.vcpt[j], xj = S.vxu[j];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double cij = C[((row0 + 8 * k) ^ (flip | ((e & 1) << 1))) + j * NMAX];
                bs[k] = fma(cij, cp, bs[k]);
                as[k] = fma(cij * x1, xj, as[k]);
                m.set(4 * e + k, (rd4[k] * cij) * x1);
            }
        }
        m.store(S.tm + 32 * ch);
    }
    const int cflip = quad_swizzle(r0);
#pragma unroll 2
    for (int ch = 0; ch < NMAX / 16; ch++) {
        tmem::Chunk m;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            /* leaf 4 ch + e: its bits reversed are t (tree_leaf) */
            const int t = (int)(__brev(4u * (unsigned)ch + (unsigned)e) >> (32 - (G == 2 ? 4 : 5)));
            const int j = 4 * t + c;
            const double rdj = S.vrd[j];
#pragma unroll
            for (int k = 0; k < 4; k++)
                m.set(4 * e + k, (rdj * C[(j ^ cflip) + (row0 + 8 * k) * NMAX]) * x14[k]);
        }
        m.store(S.tm + 2 * NMAX + 32 * ch);
    }
    const double bsum = quad_chains<8, 16>(c, bs), asum = quad_chains<8, 16>(c, as);
    tmem::wait_stores();
    double r = 0.0, bval = 0.0;
    if (valid) {
        const double b = fma(rd, bsum, xu);
        const double ax = fma(rd, asum, xu);
        r = b - ax;
        bval = b;
    }
    auto put = [&](const double (&v)[1], const double (&vt)[1]) {
        S.vp[i] = v[0];
        S.vpt[i] = vt[0];
    };
    /* q = A v (row sums of W), q~ = A^T vt (column tree of W) */
    auto mul = [&](const double (&v)[1], const double (&vt)[1], double (&q)[1], double (&qt)[1]) {
        double qs[1];
        tmem_row_sums<1, NMAX>(S.tm, c, S.vp, qs);
        const double qts = tmem_column_tree<NMAX>(S.tm + 2 * NMAX, c, S.vpt);
        q[0] = valid ? v[0] + qs[0] : 0.0;
        qt[0] = valid ? vt[0] + qts : 0.0;
    };
    double rr[1] = {r}, xx[1] = {xu};
    const double bb[1] = {bval};
    const int done = bicg_iterate<1, G, REC>(S, P, bb, rr, xx, put, mul, capped);
    F[0][IC] = xx[0];
    return done;
}

/* ---------------------------------------------------------------------------
 * Coupled right-hand side with the operator W in shared memory and two or four
 * units per lane of one warp (Steppers.cuh:432-562). */
template <int U, int G, int REC>
__device__ __forceinline__ int coupled_rhs(const Sys<U, G>& S, const DeviceProblem& P, double T,
                                           double (&Xs)[U][UD], double (&F)[U][UD],
                                           double (&up)[U][NUPa], double (&ua)[U][NUAa],
                                           int (&iua)[U][NIUAa], bool& capped) {
    constexpr int NMAX = WarpSmem<U, G>::NMAX;
    constexpr int LDW = WarpSmem<U, G>::LDW;
    const int N = S.N;
    double xu[U], rd[U], r[U], x[U], bv[U];
    grp_sync(S);
#pragma unroll
    for (int m = 0; m < U; m++) {
        const int i = S.unit(m);
        if (i < N) {
            double Fl[UD], cpt, cpf;
            CoupledSystems_PerBlock_OdeFunction<double>(S.sid, i, Fl, Xs[m], T, U == 1 ? S.upsh + i * NUPa : up[m],
                                                        S.sPAR, S.gPAR, S.igPAR,
                                                        ua[m], iua[m], S.sACC, S.isACC, &cpt, &cpf);
#pragma unroll
            for (int k = 0; k < UD; k++) F[m][k] = Fl[k];
            xu[m] = Fl[IC];
            rd[m] = cpf;
            S.vcpt[i] = cpt;
            S.vx1[i] = Xs[m][0] * Xs[m][0];
            S.vxu[i] = Fl[IC];
        } else {
#pragma unroll
            for (int k = 0; k < UD; k++) F[m][k] = 0.0;
            xu[m] = 0.0;
            rd[m] = 0.0;
        }
    }
    grp_sync(S);
    /* b = rD (C CPT) + x_u, r = b - A x_u, W_ij = (rD_i C_ij) X1sq_j */
#pragma unroll
    for (int m = 0; m < U; m++) {
        const int i = S.unit(m);
        if (i < N) {
            double b0 = 0.0, b1 = 0.0, b2 = 0.0, b3 = 0.0, a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
            const double* Ci = S.C + i;
            double* Wi = S.W + i;
            const double rdm = rd[m];
            /* one column: chain k of the four interleaved chains */
            auto col = [&](int j, double& bk, double& ak) {
                const double cij = __ldg(Ci + (int64_t)j * N);
                const double x1 = S.vx1[j];
                bk = fma(cij, S.vcpt[j], bk);
                ak = fma(cij * x1, S.vxu[j], ak);
                Wi[j * LDW] = (rdm * cij) * x1;
            };
            int j = 0;
            for (; j + 3 < N; j += 4) {
                col(j, b0, a0);
                col(j + 1, b1, a1);
                col(j + 2, b2, a2);
                col(j + 3, b3, a3);
            }
            if (j < N) col(j, b0, a0);
            if (j + 1 < N) col(j + 1, b1, a1);
            if (j + 2 < N) col(j + 2, b2, a2);
            double b = fma(rdm, (b0 + b1) + (b2 + b3), xu[m]);
            double ax = fma(rdm, (a0 + a1) + (a2 + a3), xu[m]);
            r[m] = b - ax;
            bv[m] = b;
        } else {
            r[m] = 0.0;
            bv[m] = 0.0;
        }
        x[m] = xu[m];
    }
    /* q = A v (row sums of W), q~ = A^T vt (column tree of W) */
    auto put = [&](const double (&v)[U], const double (&vt)[U]) {
#pragma unroll
        for (int m = 0; m < U; m++) {
            const int i = S.unit(m);
            S.vp[i] = v[m];
            S.vpt[i] = vt[m];
        }
    };
    auto mul = [&](const double (&v)[U], const double (&vt)[U], double (&q)[U], double (&qt)[U]) {
#pragma unroll
        for (int m = 0; m < U; m++) {
            const int i = S.unit(m);
            if (i < N) {
                double q0 = 0.0, q1 = 0.0, q2 = 0.0, q3 = 0.0;
                const double* Wi = S.W + i;
                int j = 0;
                for (; j + 3 < N; j += 4) {
                    q0 = fma(Wi[j * LDW], S.vp[j], q0);
                    q1 = fma(Wi[(j + 1) * LDW], S.vp[j + 1], q1);
                    q2 = fma(Wi[(j + 2) * LDW], S.vp[j + 2], q2);
                    q3 = fma(Wi[(j + 3) * LDW], S.vp[j + 3], q3);
                }
                if (j < N) q0 = fma(Wi[j * LDW], S.vp[j], q0);
                if (j + 1 < N) q1 = fma(Wi[(j + 1) * LDW], S.vp[j + 1], q1);
                if (j + 2 < N) q2 = fma(Wi[(j + 2) * LDW], S.vp[j + 2], q2);
                q[m] = v[m] + ((q0 + q1) + (q2 + q3));
                const double* Wc = S.W + (int64_t)i * LDW;
                const double* vpt = S.vpt;
                auto leaf = [&](int j) -> double { return j < N ? Wc[j] * vpt[j] : 0.0; };
                qt[m] = vt[m] + TreeSum<1, NMAX>::run(0, leaf);
            } else {
                q[m] = 0.0;
                qt[m] = 0.0;
            }
        }
    };
    const int done = bicg_iterate<U, G, REC, (U > 1)>(S, P, bv, r, x, put, mul, capped);
#pragma unroll
    for (int m = 0; m < U; m++) F[m][IC] = x[m];
    return done;
}

/* ---------------------------------------------------------------------------
 * Work split of the one-warp products (N <= 32).  Lane l owns unit l, but a
 * product gives lane l = 2r + h two rows, 2r and 2r + 1, and of each the columns
 * of chains 2h and 2h + 1 (j = 4t + 2h + e, e < 2): the lane pair then exchanges
 * one partial sum a vector, and lane l keeps row l.  With a whole row per lane
 * every entry of a broadcast vector is loaded for one fma, and a sub-partition
 * fills registers from shared memory at 64 bytes a clock: 32 double2 loads a
 * product took 270 cycles against 160 for the fmas.  Two rows a lane halve the
 * loads; the sums are the same chains in the same order. */
__device__ __forceinline__ double pair_exchange(int h, double own0, double own1) {
    const double keep = h ? own1 : own0, give = h ? own0 : own1;
    return keep + __shfl_xor_sync(FULL, give, 1);
}

/* f(t) for the column groups t < ceil(N / 4), unrolled, in three runs so that
 * systems of up to 8 and up to 16 units skip the rest */
template <int NFIX, class Fn>
__device__ __forceinline__ void column_groups(int N, Fn&& f) {
#pragma unroll
    for (int t = 0; t < 2; t++) f(t);
    if (NFIX != 0 || N > 8) {
#pragma unroll
        for (int t = 2; t < 4; t++) f(t);
    }
    if (NFIX != 0 || N > 16) {
#pragma unroll
        for (int t = 4; t < 8; t++) f(t);
    }
}

/* ---------------------------------------------------------------------------
 * Coupled right-hand side with the operator in registers (N <= 32, one unit
 * per lane).  A lane holds the entries of W that its share of A v reads (two
 * rows, two chains: 32 doubles in registers) and those its share of A^T vt
 * reads: for the two columns 2r and 2r + 1 the rows of parity h, because the
 * halving tree over the rows splits into its even and its odd subtree until its
 * last addition: 32 doubles of its own, in shared memory (lane-consecutive
 * double2) or with TMEM in tensor memory; in registers as well they spill.  With
 * a warp to itself on each sub-partition tensor memory is the faster place (256
 * systems of 32: 322 -> 292 ms), with two the slower (1024: 287 -> 331 ms).  The system's coupling matrix is
 * staged once per system, zero-padded (leading dimension 33); the vector of the
 * transposed product is posted split by parity.
 * NFIX = 32 drops the N guards for full warps.  Same arithmetic, in the same
 * order, as the shared-memory variant. */
template <int NFIX, int REC, bool TMEM>
__device__ __forceinline__ int coupled_rhs_regw(const Sys<1>& S, const DeviceProblem& P, double T,
                                                double (&Xs)[1][UD], double (&F)[1][UD],
                                                double (&up)[1][NUPa], double (&ua)[1][NUAa],
                                                int (&iua)[1][NIUAa], bool& capped) {
    constexpr int LDC = WarpSmem<1>::LDW;
    const int N = NFIX ? NFIX : S.N;
    const int i = S.lane;
    const int h = i & 1, r0 = i & ~1;   /* rows (and columns) r0, r0 + 1; chains 2h, 2h + 1; row parity h */
    const bool valid = i < N;
    double xu = 0.0, rd = 0.0, x1 = 0.0;
    __syncwarp();
    if (valid) {
        double Fl[UD], cpt, cpf;
        CoupledSystems_PerBlock_OdeFunction<double>(S.sid, i, Fl, Xs[0], T, S.upsh + i * NUPa, S.sPAR, S.gPAR,
                                                    S.igPAR, ua[0], iua[0], S.sACC, S.isACC, &cpt, &cpf);
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = Fl[k];
        xu = Fl[IC];
        rd = cpf;
        x1 = Xs[0][0] * Xs[0][0];
        S.vcpt[i] = cpt;
    } else {
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = 0.0;
        S.vcpt[i] = 0.0;
    }
    S.vx1[i] = x1;
    S.vxu[i] = xu;
    S.vrd[i] = rd;
    S.rdpar[par_slot(i)] = rd;
    __syncwarp();
    double wr[2][16];
    /* the column share, entry k of columns r0, r0 + 1: at wc[32 k], or 2k and 2k + 1 of the chunks */
    double2* wc = reinterpret_cast<double2*>(S.W + 32 * LDC) + i;
    tmem::Chunk tc[2];
    double bs[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, as[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    const double* C = S.W;   /* C[i][j] at i + j * LDC */
    const double2* vx1_2 = reinterpret_cast<const double2*>(S.vx1);
    const double2* vcpt2 = reinterpret_cast<const double2*>(S.vcpt);
    const double2* vxu2 = reinterpret_cast<const double2*>(S.vxu);
    const double2* rdp2 = reinterpret_cast<const double2*>(S.rdpar + h * RED_RUN);
    const double2 rd2 = reinterpret_cast<const double2*>(S.vrd)[i >> 1], x12 = vx1_2[i >> 1];
#pragma unroll
    for (int t = 0; t < 16; t++) {
        wr[0][t] = wr[1][t] = 0.0;
        tc[t >> 3].set(2 * (t & 7), 0.0);
        tc[t >> 3].set(2 * (t & 7) + 1, 0.0);
    }
    column_groups<NFIX>(N, [&](int t) {
        const double2 x1p = vx1_2[2 * t + h], cpp = vcpt2[2 * t + h], xup = vxu2[2 * t + h];
        const double2 rdk = rdp2[t];   /* rows k = 4t + h and 4t + 2 + h */
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int j = 4 * t + 2 * h + e;
            const double c0 = C[r0 + j * LDC], c1 = C[r0 + 1 + j * LDC];
            const double x1j = e ? x1p.y : x1p.x, cpj = e ? cpp.y : cpp.x, xuj = e ? xup.y : xup.x;
            /* columns beyond N hold zeros in C and in every vector: their terms are +0 */
            bs[0][e] = fma(c0, cpj, bs[0][e]);
            bs[1][e] = fma(c1, cpj, bs[1][e]);
            as[0][e] = fma(c0 * x1j, xuj, as[0][e]);
            as[1][e] = fma(c1 * x1j, xuj, as[1][e]);
            wr[0][2 * t + e] = (rd2.x * c0) * x1j;
            wr[1][2 * t + e] = (rd2.y * c1) * x1j;
            const int k = 4 * t + 2 * e + h;   /* the row with index 2t + e among those of parity h */
            const double rk = e ? rdk.y : rdk.x;
            const double wk0 = (rk * C[k + r0 * LDC]) * x12.x, wk1 = (rk * C[k + (r0 + 1) * LDC]) * x12.y;
            if constexpr (TMEM) {
                tc[t >> 2].set(2 * (2 * (t & 3) + e), wk0);
                tc[t >> 2].set(2 * (2 * (t & 3) + e) + 1, wk1);
            } else {
                wc[32 * (2 * t + e)] = make_double2(wk0, wk1);
            }
        }
    });
    if constexpr (TMEM) {
        tc[0].store(S.tm);
        tc[1].store(S.tm + 32);
        tmem::wait_stores();
    }
    double r = 0.0, bval = 0.0;
    {
        const double bsum = pair_exchange(h, bs[0][0] + bs[0][1], bs[1][0] + bs[1][1]);
        const double asum = pair_exchange(h, as[0][0] + as[0][1], as[1][0] + as[1][1]);
        if (valid) {
            const double b = fma(rd, bsum, xu);
            const double ax = fma(rd, asum, xu);
            r = b - ax;
            bval = b;
        }
    }
    const double2* vp2 = reinterpret_cast<const double2*>(S.vp);
    const double2* tp2 = reinterpret_cast<const double2*>(S.tpar + h * RED_RUN);
    const int tslot = par_slot(i);
    auto put = [&](const double (&v)[1], const double (&vt)[1]) {
        S.vp[i] = v[0];
        S.tpar[tslot] = vt[0];
    };
    /* q = A v (this lane's chains of two rows), q~ = A^T vt (this lane's subtree of two columns) */
    auto mul = [&](const double (&v)[1], const double (&vt)[1], double (&qo)[1], double (&qto)[1]) {
        double qs[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
        double u[2][16];
#pragma unroll
        for (int k = 0; k < 16; k++) u[0][k] = u[1][k] = 0.0;
        /* from tensor memory the column share arrives in two chunks, the first beside the row sums */
        tmem::Chunk m;
        if constexpr (TMEM) m.load(S.tm);
        column_groups<NFIX>(N, [&](int t) {
            const double2 a = vp2[2 * t + h];
            qs[0][0] = fma(wr[0][2 * t], a.x, qs[0][0]);
            qs[1][0] = fma(wr[1][2 * t], a.x, qs[1][0]);
            qs[0][1] = fma(wr[0][2 * t + 1], a.y, qs[0][1]);
            qs[1][1] = fma(wr[1][2 * t + 1], a.y, qs[1][1]);
            if constexpr (!TMEM) {
                const double2 c = tp2[t], w0 = wc[32 * (2 * t)], w1 = wc[32 * (2 * t + 1)];
                u[0][2 * t] = w0.x * c.x;
                u[1][2 * t] = w0.y * c.x;
                u[0][2 * t + 1] = w1.x * c.y;
                u[1][2 * t + 1] = w1.y * c.y;
            }
        });
        if constexpr (TMEM) {
            auto products = [&](int ch) {
#pragma unroll
                for (int t = 4 * ch; t < 4 * ch + 4; t++) {
                    const double2 c = tp2[t];
                    u[0][2 * t] = m.get(4 * (t & 3)) * c.x;
                    u[1][2 * t] = m.get(4 * (t & 3) + 1) * c.x;
                    u[0][2 * t + 1] = m.get(4 * (t & 3) + 2) * c.y;
                    u[1][2 * t + 1] = m.get(4 * (t & 3) + 3) * c.y;
                }
            };
            m.wait();
            products(0);
            if (NFIX != 0 || N > 16) {
                m.load(S.tm + 32);
                m.wait();
                products(1);
            }
        }
        const double q = v[0] + pair_exchange(h, qs[0][0] + qs[0][1], qs[1][0] + qs[1][1]);
        auto leaf0 = [&](int k) -> double { return u[0][k]; };
        auto leaf1 = [&](int k) -> double { return u[1][k]; };
        const double qt = vt[0] + pair_exchange(h, TreeSum<1, 16>::run(0, leaf0), TreeSum<1, 16>::run(0, leaf1));
        qo[0] = valid ? q : 0.0;
        qto[0] = valid ? qt : 0.0;
    };
    double rr[1] = {r}, xx[1] = {xu};
    const double bb[1] = {bval};
    const int done = bicg_iterate<1, 1, REC>(S, P, bb, rr, xx, put, mul, capped);
    const double x = xx[0];
    F[0][IC] = x;
    return done;
}

/* ---------------------------------------------------------------------------
 * Coupled right-hand side with the launch's shared coupling matrix staged once
 * per CTA (RHS = 3, 64 or 128 units).  A system's coupling matrix is
 * C = diag(a) G diag(b) with G the staged matrix and a, b unit-scope factors
 * (1 unless the caller sets them: one shared geometry, per-system radii).
 * With u = b X1sq and v = rD a the products apply G to scaled vectors,
 *   A x0 = v (G (u x0)),  A p = p + v (G (u p)),  A^T p~ = p~ + u (G^T (v p~)),
 *   right-hand side v (G (b CPT)) + x_u,
 * with G row sums as four interleaved fma chains and G column sums in the
 * halving-tree order over 32UG; the oracle's shared-matrix association
 * computes the same (a = b = 1 reproduces the unscaled products bit for bit). */
template <int U, int G, bool SYM, int REC>
__device__ __forceinline__ int coupled_rhs_sharedc(const Sys<U, G>& S, const DeviceProblem& P, double T,
                                                   double (&Xs)[U][UD], double (&F)[U][UD],
                                                   double (&up)[U][NUPa], double (&ua)[U][NUAa],
                                                   int (&iua)[U][NIUAa], const double (&ra)[U],
                                                   const double (&cb)[U], bool& capped) {
    using SM = SharedCSmem<U, G, SYM>;
    constexpr int NMAX = SM::NMAX;
    constexpr int LDC = SM::LDC;
    constexpr int H = NMAX / 2;
    static_assert(U > 1 || !SYM, "the symmetric matrix of one-unit-per-lane systems is in tensor memory");
    const int N = S.N;
    /* with C = diag(a) G diag(b): x1 holds u = b X1sq (applied before G), rd holds v = rD a (after G) */
    double xu[U], rd[U], x1[U], r[U], x[U], bv[U];
    grp_sync(S);
#pragma unroll
    for (int m = 0; m < U; m++) {
        const int i = S.unit(m);
        if (i < N) {
            double Fl[UD], cpt, cpf;
            CoupledSystems_PerBlock_OdeFunction<double>(S.sid, i, Fl, Xs[m], T, U == 1 ? S.upsh + i * NUPa : up[m],
                                                        S.sPAR, S.gPAR, S.igPAR,
                                                        ua[m], iua[m], S.sACC, S.isACC, &cpt, &cpf);
#pragma unroll
            for (int k = 0; k < UD; k++) F[m][k] = Fl[k];
            xu[m] = Fl[IC];
            rd[m] = cpf * ra[m];
            x1[m] = cb[m] * (Xs[m][0] * Xs[m][0]);
            S.vcpt[i] = cb[m] * cpt;
            S.vp[i] = x1[m] * xu[m];   /* z0 = b X1sq x0 */
        } else {
#pragma unroll
            for (int k = 0; k < UD; k++) F[m][k] = 0.0;
            xu[m] = 0.0;
            rd[m] = 0.0;
            x1[m] = 0.0;
            S.vcpt[i] = 0.0;
            S.vp[i] = 0.0;
        }
    }
    grp_sync(S);
    const double2* cpt2 = reinterpret_cast<const double2*>(S.vcpt);
    const double2* z2 = reinterpret_cast<const double2*>(S.vp);
    const double2* zt2 = reinterpret_cast<const double2*>(S.vpt);
    const int c = S.lane & 3, row0 = S.unit(0) & ~3;   /* the quad's rows (U = 1) */
    /* rowsum_m = sum_j C[i_m][j] v[j], four interleaved chains */
    auto row_sums = [&](const double2* v2, double (&out)[U]) {
        if constexpr (U == 1) {
            const double* const vec[1] = {reinterpret_cast<const double*>(v2)};
            quad_row_sums<LDC, 1>(S.W, row0, c, N, vec, out);
        } else {
            double a0[U], a1[U], a2[U], a3[U];
#pragma unroll
            for (int m = 0; m < U; m++) { a0[m] = 0.0; a1[m] = 0.0; a2[m] = 0.0; a3[m] = 0.0; }
#pragma unroll 4
            for (int j = 0; j < NMAX; j += 4) {
                const double2 va = v2[j / 2], vb = v2[j / 2 + 1];
#pragma unroll
                for (int m = 0; m < U; m++) {
                    const double* Crow = S.W + S.unit(m);
                    if (j < N) a0[m] = fma(Crow[j * LDC], va.x, a0[m]);
                    if (j + 1 < N) a1[m] = fma(Crow[(j + 1) * LDC], va.y, a1[m]);
                    if (j + 2 < N) a2[m] = fma(Crow[(j + 2) * LDC], vb.x, a2[m]);
                    if (j + 3 < N) a3[m] = fma(Crow[(j + 3) * LDC], vb.y, a3[m]);
                }
            }
#pragma unroll
            for (int m = 0; m < U; m++) out[m] = (a0[m] + a1[m]) + (a2[m] + a3[m]);
        }
    };
    /* the same row sums for two vectors at once: each matrix entry read from
     * shared memory once (the kernel is bound by shared-memory reads), the
     * chains and their order per vector as in row_sums */
    auto row_sums2 = [&](const double2* v2, const double2* w2, double (&outv)[U], double (&outw)[U]) {
        if constexpr (U == 1) {
            const double* const vec[2] = {reinterpret_cast<const double*>(v2), reinterpret_cast<const double*>(w2)};
            double o[2];
            quad_row_sums<LDC, 2>(S.W, row0, c, N, vec, o);   /* the right-hand side's sums only */
            outv[0] = o[0];
            outw[0] = o[1];
        } else {
            double a0[U], a1[U], a2[U], a3[U], b0[U], b1[U], b2[U], b3[U];
#pragma unroll
            for (int m = 0; m < U; m++) {
                a0[m] = 0.0; a1[m] = 0.0; a2[m] = 0.0; a3[m] = 0.0;
                b0[m] = 0.0; b1[m] = 0.0; b2[m] = 0.0; b3[m] = 0.0;
            }
#pragma unroll 2
            for (int j = 0; j < NMAX; j += 4) {
                const double2 va = v2[j / 2], vb = v2[j / 2 + 1];
                const double2 wa = w2[j / 2], wb = w2[j / 2 + 1];
#pragma unroll
                for (int m = 0; m < U; m++) {
                    const double* Crow = S.W + S.unit(m);
                    if (j < N) { const double c = Crow[j * LDC]; a0[m] = fma(c, va.x, a0[m]); b0[m] = fma(c, wa.x, b0[m]); }
                    if (j + 1 < N) {
                        const double c = Crow[(j + 1) * LDC];
                        a1[m] = fma(c, va.y, a1[m]);
                        b1[m] = fma(c, wa.y, b1[m]);
                    }
                    if (j + 2 < N) {
                        const double c = Crow[(j + 2) * LDC];
                        a2[m] = fma(c, vb.x, a2[m]);
                        b2[m] = fma(c, wb.x, b2[m]);
                    }
                    if (j + 3 < N) {
                        const double c = Crow[(j + 3) * LDC];
                        a3[m] = fma(c, vb.y, a3[m]);
                        b3[m] = fma(c, wb.y, b3[m]);
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < U; m++) {
                outv[m] = (a0[m] + a1[m]) + (a2[m] + a3[m]);
                outw[m] = (b0[m] + b1[m]) + (b2[m] + b3[m]);
            }
        }
    };
    double bsum[U], asum[U];
    row_sums2(cpt2, z2, bsum, asum);
#pragma unroll
    for (int m = 0; m < U; m++) {
        if (S.unit(m) < N) {
            const double b = fma(rd[m], bsum[m], xu[m]);
            const double ax = fma(rd[m], asum[m], xu[m]);
            r[m] = b - ax;
            bv[m] = b;
        } else {
            r[m] = 0.0;
            bv[m] = 0.0;
        }
        x[m] = xu[m];
    }
    /* q = A v = v + rD a (G (b X1sq v)), q~ = A^T vt = vt + b X1sq (G^T (rD a vt)) */
    auto put = [&](const double (&v)[U], const double (&vt)[U]) {
#pragma unroll
        for (int m = 0; m < U; m++) {
            const int i = S.unit(m);
            S.vp[i] = x1[m] * v[m];    /* z  = X1sq v  */
            S.vpt[i] = rd[m] * vt[m];  /* z~ = rD vt   */
        }
    };
    auto mul = [&](const double (&v)[U], const double (&vt)[U], double (&q)[U], double (&qt)[U]) {
        double qs[U], qts[U];
        if constexpr (SYM) {
            /* C = C^T: the transposed product is a row sum too, from the same reads */
            row_sums2(z2, zt2, qs, qts);
        } else if constexpr (U == 1) {
            row_sums(z2, qs);
            qts[0] = quad_column_tree<NMAX, LDC>(S.W, row0, c, S.vpt);
        } else {
        row_sums(z2, qs);
#pragma unroll
        for (int m = 0; m < U; m++) {
            /* column i_m of C against z~: the first tree levels on the loads, then the halving tree over 32 */
            const double2* Ccol2 = reinterpret_cast<const double2*>(S.W + (S.unit(m)) * LDC);
            double u[32];
#pragma unroll
            for (int k = 0; k < 32; k += 2) {
                double2 c0 = Ccol2[k / 2], z0 = zt2[k / 2];
                double s0 = c0.x * z0.x, s1 = c0.y * z0.y;
                if constexpr (H >= 32) {
                    const double2 c1 = Ccol2[(k + 32) / 2], z1 = zt2[(k + 32) / 2];
                    if constexpr (H == 64) {
                        const double2 c2 = Ccol2[(k + 64) / 2], zz2 = zt2[(k + 64) / 2];
                        const double2 c3 = Ccol2[(k + 96) / 2], z3 = zt2[(k + 96) / 2];
                        s0 = (s0 + c2.x * zz2.x) + (c1.x * z1.x + c3.x * z3.x);
                        s1 = (s1 + c2.y * zz2.y) + (c1.y * z1.y + c3.y * z3.y);
                    } else {
                        s0 = s0 + c1.x * z1.x;
                        s1 = s1 + c1.y * z1.y;
                    }
                }
                u[k] = s0;
                u[k + 1] = s1;
            }
            auto leaf = [&](int k) -> double { return u[k]; };
            qts[m] = TreeSum<1, 32>::run(0, leaf);
        }
        }
#pragma unroll
        for (int m = 0; m < U; m++) {
            const bool vld = S.unit(m) < N;
            q[m] = vld ? fma(rd[m], qs[m], v[m]) : 0.0;
            qt[m] = vld ? fma(x1[m], qts[m], vt[m]) : 0.0;
        }
    };
    const int done = bicg_iterate<U, G, REC, (U > 1 && REC == 1)>(S, P, bv, r, x, put, mul, capped);
#pragma unroll
    for (int m = 0; m < U; m++) F[m][IC] = x[m];
    return done;
}

/* ---------------------------------------------------------------------------
 * Coupled right-hand side with the launch's shared symmetric matrix and one unit
 * per lane on G warps (RHS = 4): the scaled products of coupled_rhs_sharedc, both
 * as row sums of the lane's share of G in tensor memory (stored once per CTA)
 * against two vectors posted side by side. */
template <int G, int REC>
__device__ __forceinline__ int coupled_rhs_symquad(const Sys<1, G>& S, const DeviceProblem& P, double T,
                                                   double (&Xs)[1][UD], double (&F)[1][UD], double (&ua)[1][NUAa],
                                                   int (&iua)[1][NIUAa], const double (&ra)[1], const double (&cb)[1],
                                                   bool& capped) {
    const int N = S.N;
    const int i = S.unit(0);
    const bool valid = i < N;
    const int c = S.lane >> 3;
    double2* post = reinterpret_cast<double2*>(S.vp) + i;   /* vp and vpt: the pairs of all NMAX units */
    double xu = 0.0, rd = 0.0, x1 = 0.0;
    grp_sync(S);
    if (valid) {
        double Fl[UD], cpt, cpf;
        CoupledSystems_PerBlock_OdeFunction<double>(S.sid, i, Fl, Xs[0], T, S.upsh + i * NUPa, S.sPAR, S.gPAR,
                                                    S.igPAR, ua[0], iua[0], S.sACC, S.isACC, &cpt, &cpf);
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = Fl[k];
        xu = Fl[IC];
        rd = cpf * ra[0];                       /* v = rD a  */
        x1 = cb[0] * (Xs[0][0] * Xs[0][0]);     /* u = b X1sq */
        *post = make_double2(cb[0] * cpt, x1 * xu);
    } else {
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = 0.0;
        *post = make_double2(0.0, 0.0);
    }
    grp_sync(S);
    double sums[2];
    tmem_row_sums<2, 32 * G>(S.tm, c, S.vp, sums);
    double r = 0.0, bval = 0.0;
    if (valid) {
        const double b = fma(rd, sums[0], xu);
        const double ax = fma(rd, sums[1], xu);
        r = b - ax;
        bval = b;
    }
    /* q = A v = v + v_f (G (u v)), q~ = A^T vt = vt + u (G (v_f vt)) with u = b X1sq, v_f = rD a */
    auto put = [&](const double (&v)[1], const double (&vt)[1]) {
        *post = valid ? make_double2(x1 * v[0], rd * vt[0]) : make_double2(0.0, 0.0);
    };
    auto mul = [&](const double (&v)[1], const double (&vt)[1], double (&q)[1], double (&qt)[1]) {
        double qs[2];
        tmem_row_sums<2, 32 * G>(S.tm, c, S.vp, qs);
        q[0] = valid ? fma(rd, qs[0], v[0]) : 0.0;
        qt[0] = valid ? fma(x1, qs[1], vt[0]) : 0.0;
    };
    double rr[1] = {r}, xx[1] = {xu};
    const double bb[1] = {bval};
    const int done = bicg_iterate<1, G, REC>(S, P, bb, rr, xx, put, mul, capped);
    F[0][IC] = xx[0];
    return done;
}

/* ---------------------------------------------------------------------------
 * Coupled right-hand side for N <= 32 when the launch shares one symmetric
 * matrix G (RHS = 5; 6 drops the N guards when every system has 32 units):
 * a lane's share of G (two rows, two chains: 32 entries) is staged in shared
 * memory once per system, lane-consecutive, and taken into registers for a
 * right-hand side -- nothing is formed -- and both BiCG products are row sums of
 * those entries against posted vectors, with the unit factors a, b as in
 * coupled_rhs_sharedc<.., SYM = true> and the same arithmetic order.  Held in
 * registers for the whole system the share left too few of them outside the
 * products: the compiler kept part of it in local memory, whose loads miss the
 * small L1 that 230 KB of shared memory leave (300 systems of 31 units, 250
 * steps: 7.7 -> 6.75 ms, with REC 1 8.7 -> 6.95). */
template <int NFIX, int REC>
__device__ __forceinline__ int coupled_rhs_regsym(const Sys<1>& S, const DeviceProblem& P, double T,
                                                  double (&Xs)[1][UD], double (&F)[1][UD], double (&ua)[1][NUAa],
                                                  int (&iua)[1][NIUAa], const double (&ra)[1], const double (&cb)[1],
                                                  bool& capped) {
    const int N = NFIX ? NFIX : S.N;
    const int i = S.lane;
    const int h = i & 1;
    const bool valid = i < N;
    double xu = 0.0, rd = 0.0, x1 = 0.0;
    __syncwarp();
    double g[32];   /* this lane's share of G */
    const double2* share = reinterpret_cast<const double2*>(S.W) + i;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const double2 t = share[32 * k];
        g[2 * k] = t.x;
        g[2 * k + 1] = t.y;
    }
    if (valid) {
        double Fl[UD], cpt, cpf;
        CoupledSystems_PerBlock_OdeFunction<double>(S.sid, i, Fl, Xs[0], T, S.upsh + i * NUPa, S.sPAR, S.gPAR,
                                                    S.igPAR, ua[0], iua[0], S.sACC, S.isACC, &cpt, &cpf);
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = Fl[k];
        xu = Fl[IC];
        rd = cpf * ra[0];                       /* v = rD a  */
        x1 = cb[0] * (Xs[0][0] * Xs[0][0]);     /* u = b X1sq */
        S.vcpt[i] = cb[0] * cpt;
        S.vp[i] = x1 * xu;
    } else {
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = 0.0;
        S.vcpt[i] = 0.0;
        S.vp[i] = 0.0;
    }
    __syncwarp();
    /* row sums of G against two posted vectors: this lane's chains of two rows, g = their entries
     * (columns beyond N hold zeros in G and in the vectors: their terms are +0) */
    auto row_sums2 = [&](const double* v, const double* w, double& outv, double& outw) {
        const double2* v2 = reinterpret_cast<const double2*>(v) + h;
        const double2* w2 = reinterpret_cast<const double2*>(w) + h;
        double a[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, b[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
        column_groups<NFIX>(N, [&](int t) {
            const double2 vv = v2[2 * t], ww = w2[2 * t];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const double vj = e ? vv.y : vv.x, wj = e ? ww.y : ww.x;
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    a[m][e] = fma(g[16 * m + 2 * t + e], vj, a[m][e]);
                    b[m][e] = fma(g[16 * m + 2 * t + e], wj, b[m][e]);
                }
            }
        });
        outv = pair_exchange(h, a[0][0] + a[0][1], a[1][0] + a[1][1]);
        outw = pair_exchange(h, b[0][0] + b[0][1], b[1][0] + b[1][1]);
    };
    double bsum, asum;
    row_sums2(S.vcpt, S.vp, bsum, asum);
    double r = 0.0, bval = 0.0;
    if (valid) {
        const double b = fma(rd, bsum, xu);
        const double ax = fma(rd, asum, xu);
        r = b - ax;
        bval = b;
    }
    /* q = A v = v + v_f (G (u v)), q~ = A^T vt = vt + u (G (v_f vt)) with u = b X1sq, v_f = rD a */
    auto put = [&](const double (&v)[1], const double (&vt)[1]) {
        S.vp[i] = valid ? x1 * v[0] : 0.0;     /* z  = u v  */
        S.vpt[i] = valid ? rd * vt[0] : 0.0;   /* z~ = v_f vt */
    };
    auto mul = [&](const double (&v)[1], const double (&vt)[1], double (&qo)[1], double (&qto)[1]) {
        double qs, qts;
        row_sums2(S.vp, S.vpt, qs, qts);
        qo[0] = valid ? fma(rd, qs, v[0]) : 0.0;
        qto[0] = valid ? fma(x1, qts, vt[0]) : 0.0;
    };
    double rr[1] = {r}, xx[1] = {xu};
    const double bb[1] = {bval};
    const int done = bicg_iterate<1, 1, REC>(S, P, bb, rr, xx, put, mul, capped);
    const double x = xx[0];
    F[0][IC] = x;
    return done;
}

/* ---------------------------------------------------------------------------
 * Systems of up to 32 units on a team of four warps, for launches of so few
 * systems that warps are to spare (RHS 11, 12: own matrix; 15, 16: shared symmetric
 * matrix with unit factors; the even ones without N guards).  Every warp of the
 * team integrates the whole system, in private registers and shared memory, from
 * the same values to the same bits -- every decision included -- and only the
 * products, half of a BiCG iteration on one warp, are divided: warps 0 and 1 form
 * q, warps 2 and 3 q~, each over two of its four chains (of the column tree: one
 * parity of the rows), lane l for unit l.  Each posts its partial sums in the
 * team's exchange buffer, one named barrier, and all read them.  The two buffers
 * alternate, so one is rewritten only after a later exchange's barrier.  The
 * host's rule (team_pays) says for how many systems. */
__device__ __forceinline__ double* team_buffer(const Sys<1>& S) {
    double* b = S.xt + (S.tsel & 1) * (TEAM * 32);
    S.tsel++;
    return b;
}
__device__ __forceinline__ void team_sync(const Sys<1>& S) {
    asm volatile("bar.sync %0, %1;" ::"r"(S.bar), "r"(32 * TEAM) : "memory");
}
/* warp 0's value to the whole team */
__device__ __forceinline__ int team_share(const Sys<1>& S, int v) {
    double* x = team_buffer(S);
    if (S.tw == 0 && S.lane == 0) x[0] = (double)v;
    team_sync(S);
    return (int)x[0];
}
/* the partial sums of the four warps: first = (warp 0's + warp 1's), second = (warp 2's + warp 3's) */
__device__ __forceinline__ void team_exchange(const Sys<1>& S, double partial, double& first, double& second) {
    double* x = team_buffer(S);
    x[32 * S.tw + S.lane] = partial;
    team_sync(S);
    first = x[S.lane] + x[32 + S.lane];
    second = x[64 + S.lane] + x[96 + S.lane];
}

template <bool SYM, int NFIX, int REC>
__device__ __forceinline__ int coupled_rhs_team(const Sys<1>& S, const DeviceProblem& P, double T, double (&Xs)[1][UD],
                                                double (&F)[1][UD], double (&ua)[1][NUAa], int (&iua)[1][NIUAa],
                                                const double (&ra)[1], const double (&cb)[1], const double (&g)[16],
                                                bool& capped) {
    constexpr int LDC = WarpSmem<1>::LDW;
    const int N = NFIX ? NFIX : S.N;
    const int i = S.lane;
    const int h = S.tw & 1;           /* chains 2h, 2h + 1, or the rows of parity h */
    const bool second = S.tw >= 2;    /* forms q~ */
    const bool valid = i < N;
    double xu = 0.0, rd = 0.0, x1 = 0.0, cp = 0.0;
    __syncwarp();
    if (valid) {
        double Fl[UD], cpt, cpf;
        CoupledSystems_PerBlock_OdeFunction<double>(S.sid, i, Fl, Xs[0], T, S.upsh + i * NUPa, S.sPAR, S.gPAR,
                                                    S.igPAR, ua[0], iua[0], S.sACC, S.isACC, &cpt, &cpf);
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = Fl[k];
        xu = Fl[IC];
        rd = SYM ? cpf * ra[0] : cpf;                                          /* v = rD a  */
        x1 = SYM ? cb[0] * (Xs[0][0] * Xs[0][0]) : Xs[0][0] * Xs[0][0];        /* u = b X1sq */
        cp = SYM ? cb[0] * cpt : cpt;
    } else {
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = 0.0;
    }
    const double2* vp2 = reinterpret_cast<const double2*>(S.vp) + h;
    const double2* tp2 = reinterpret_cast<const double2*>(S.tpar + h * RED_RUN);
    const int tslot = par_slot(i);
    double w[16] = {};   /* this lane's 16 entries of G or of W */
    /* this warp's chains of row i of w against the vector posted at vp */
    auto row_part = [&]() -> double {
        double s[2] = {0.0, 0.0};
        column_groups<NFIX>(N, [&](int t) {
            const double2 a = vp2[2 * t];
            s[0] = fma(w[2 * t], a.x, s[0]);
            s[1] = fma(w[2 * t + 1], a.y, s[1]);
        });
        return s[0] + s[1];
    };
    double bsum, asum;
    if constexpr (SYM) {
#pragma unroll
        for (int k = 0; k < 16; k++) w[k] = g[k];
        S.vp[i] = second ? x1 * xu : cp;
        __syncwarp();
        team_exchange(S, row_part(), bsum, asum);
    } else {
        S.vx1[i] = x1;
        S.vxu[i] = xu;
        S.vcpt[i] = cp;
        S.rdpar[tslot] = rd;
        __syncwarp();
        const double* C = S.W;   /* C[i][j] at i + j * LDC, zero-padded */
        double bs[2] = {0.0, 0.0}, as[2] = {0.0, 0.0};
        if (!second) {
            const double2* vx1_2 = reinterpret_cast<const double2*>(S.vx1) + h;
            const double2* vcpt2 = reinterpret_cast<const double2*>(S.vcpt) + h;
            const double2* vxu2 = reinterpret_cast<const double2*>(S.vxu) + h;
            column_groups<NFIX>(N, [&](int t) {
                const double2 x1p = vx1_2[2 * t], cpp = vcpt2[2 * t], xup = vxu2[2 * t];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const double c = C[i + (4 * t + 2 * h + e) * LDC];
                    const double x1j = e ? x1p.y : x1p.x;
                    bs[e] = fma(c, e ? cpp.y : cpp.x, bs[e]);
                    as[e] = fma(c * x1j, e ? xup.y : xup.x, as[e]);
                    w[2 * t + e] = (rd * c) * x1j;
                }
            });
        } else {
            const double2* rdp2 = reinterpret_cast<const double2*>(S.rdpar + h * RED_RUN);
            column_groups<NFIX>(N, [&](int t) {
                const double2 rdk = rdp2[t];
#pragma unroll
                for (int e = 0; e < 2; e++)
                    w[2 * t + e] = ((e ? rdk.y : rdk.x) * C[4 * t + 2 * e + h + i * LDC]) * x1;
            });
        }
        double* x = team_buffer(S);
        if (!second) {
            x[32 * h + i] = bs[0] + bs[1];
            x[64 + 32 * h + i] = as[0] + as[1];
        }
        team_sync(S);
        bsum = x[i] + x[32 + i];
        asum = x[64 + i] + x[96 + i];
    }
    double r = 0.0, bval = 0.0;
    if (valid) {
        const double b = fma(rd, bsum, xu);
        const double ax = fma(rd, asum, xu);
        r = b - ax;
        bval = b;
    }
    auto put = [&](const double (&v)[1], const double (&vt)[1]) {
        if constexpr (SYM) S.vp[i] = valid ? (second ? rd * vt[0] : x1 * v[0]) : 0.0;
        else if (!second) S.vp[i] = v[0];
        else S.tpar[tslot] = vt[0];
    };
    auto mul = [&](const double (&v)[1], const double (&vt)[1], double (&qo)[1], double (&qto)[1]) {
        double part, qs, qts;
        if (SYM || !second) {
            part = row_part();
        } else {
            double u[16];
#pragma unroll
            for (int k = 0; k < 16; k++) u[k] = 0.0;
            column_groups<NFIX>(N, [&](int t) {
                const double2 c = tp2[t];
                u[2 * t] = w[2 * t] * c.x;
                u[2 * t + 1] = w[2 * t + 1] * c.y;
            });
            auto leaf = [&](int k) -> double { return u[k]; };
            part = TreeSum<1, 16>::run(0, leaf);
        }
        team_exchange(S, part, qs, qts);
        if constexpr (SYM) {
            qo[0] = valid ? fma(rd, qs, v[0]) : 0.0;
            qto[0] = valid ? fma(x1, qts, vt[0]) : 0.0;
        } else {
            qo[0] = valid ? v[0] + qs : 0.0;
            qto[0] = valid ? vt[0] + qts : 0.0;
        }
    };
    double rr[1] = {r}, xx[1] = {xu};
    const double bb[1] = {bval};
    const int done = bicg_iterate<1, 1, REC>(S, P, bb, rr, xx, put, mul, capped);
    F[0][IC] = xx[0];
    return done;
}

/* ---------------------------------------------------------------------------
 * Coupled right-hand side for banded coupling storage (RHS = 7; the
 * reference's CBW modes, Steppers.cuh:586-641, whose implicit products read
 * full storage, :660,692): only the wrapping band of nd = min(2 bw + 1, N)
 * diagonals j = i + d - bw (mod N) couples, so every product costs O(N nd)
 * instead of O(N^2).  Lane i holds unit i; the system's band Cb[d][i] was
 * staged at the start of the system, the operator Wb[d][i] = (rD_i C_ij) X1sq_j
 * is formed per right-hand side, A v sums Wb[d][i] v[j] over d and A^T vt sums
 * Wb[d][k] vt[k] over k = i + bw - d (mod N), each as four chains over d
 * (d mod 4) combined (s0 + s1) + (s2 + s3) -- the oracle's banded association.
 *
 * Bound by the latency of each BiCG iteration's chain.  The chains are four
 * named accumulators, so they stay in registers whatever the run-time band (a
 * loop that indexes them by d mod 4 puts them in local memory), and the
 * operator's first BAND_REGS diagonals -- all of them up to bw = 3, the rings
 * and chains in use -- stay in registers for the whole right-hand side, in
 * both directions, so an iteration reads only the two vectors: 512 rings of
 * 128 bubbles with bw = 1, 4000 steps each, 445 -> 348 ms on a B200.
 * WIDE (RHS 10): more diagonals than that.  The rest is read from shared memory,
 * four diagonals a group without guards and two groups at once, so that sixteen
 * entries are on their way together (a guard on each entry exposed every load's
 * latency).  A kernel of its own: with the loop in the kernel of narrow bands,
 * those lose 3 %. */

template <int G, bool WIDE, int REC>
__device__ __forceinline__ int coupled_rhs_band(const Sys<1, G>& S, const DeviceProblem& P, double T,
                                                double (&Xs)[1][UD], double (&F)[1][UD], double (&ua)[1][NUAa],
                                                int (&iua)[1][NIUAa], bool& capped) {
    constexpr int NMAX = 32 * G;
    const int N = S.N;
    const int bw = P.band_width;
    const int ND = BandSmem<G, WIDE>::diagonals(bw);
    const int nd = ND < N ? ND : N;
    const int i = S.unit(0);
    const bool valid = i < N;
    const double* Cb = S.W;
    double* Wb = S.W + (size_t)ND * NMAX;
    /* first column of unit i's band and first row of its transposed band */
    const int j0 = valid ? ((i - bw) % N + N) % N : 0;
    const int k0 = valid ? ((i + bw) % N + N) % N : 0;
    double xu = 0.0, rd = 0.0;
    grp_sync(S);
    if (valid) {
        double Fl[UD], cpt, cpf;
        CoupledSystems_PerBlock_OdeFunction<double>(S.sid, i, Fl, Xs[0], T, S.upsh + i * NUPa, S.sPAR, S.gPAR,
                                                    S.igPAR, ua[0], iua[0], S.sACC, S.isACC, &cpt, &cpf);
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = Fl[k];
        xu = Fl[IC];
        rd = cpf;
        S.vcpt[i] = cpt;
        S.vx1[i] = Xs[0][0] * Xs[0][0];
        S.vxu[i] = Fl[IC];
    } else {
#pragma unroll
        for (int k = 0; k < UD; k++) F[0][k] = 0.0;
    }
    grp_sync(S);
    /* column of diagonal d (0 <= d < nd <= N, so one wrap at most) and row of its transposed entry */
    auto col = [&](int d) -> int { return j0 + d >= N ? j0 + d - N : j0 + d; };
    auto row = [&](int d) -> int { return k0 - d < 0 ? k0 - d + N : k0 - d; };
    double wr[BAND_REGS], wt[BAND_REGS];
    double r = 0.0, bval = 0.0;
    if (valid) {
        double bs[4] = {0.0, 0.0, 0.0, 0.0}, as[4] = {0.0, 0.0, 0.0, 0.0};
        auto form = [&](int d, double& bk, double& ak) -> double {
            const double c = Cb[d * NMAX + i];
            const int j = col(d);
            const double x1 = S.vx1[j];
            bk = fma(c, S.vcpt[j], bk);
            ak = fma(c * x1, S.vxu[j], ak);
            const double w = (rd * c) * x1;
            Wb[d * NMAX + i] = w;
            return w;
        };
#pragma unroll
        for (int d = 0; d < BAND_REGS; d++) wr[d] = d < nd ? form(d, bs[d & 3], as[d & 3]) : 0.0;
        if constexpr (WIDE) {
            int d = BAND_REGS;
#pragma unroll 2
            for (; d + 3 < nd; d += 4) {
#pragma unroll
                for (int e = 0; e < 4; e++) form(d + e, bs[e], as[e]);
            }
#pragma unroll
            for (int e = 0; e < 3; e++)
                if (d + e < nd) form(d + e, bs[e], as[e]);
        }
        const double b = fma(rd, (bs[0] + bs[1]) + (bs[2] + bs[3]), xu);
        const double ax = fma(rd, (as[0] + as[1]) + (as[2] + as[3]), xu);
        r = b - ax;
        bval = b;
    }
    grp_sync(S);
#pragma unroll
    for (int d = 0; d < BAND_REGS; d++) wt[d] = valid && d < nd ? Wb[d * NMAX + row(d)] : 0.0;
    auto put = [&](const double (&v)[1], const double (&vt)[1]) {
        S.vp[i] = v[0];
        S.vpt[i] = vt[0];
    };
    auto mul = [&](const double (&v)[1], const double (&vt)[1], double (&qo)[1], double (&qto)[1]) {
        double q = 0.0, qt = 0.0;
        if (valid) {
            double qs[4] = {0.0, 0.0, 0.0, 0.0}, ts[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int d = 0; d < BAND_REGS; d++)
                if (d < nd) {
                    qs[d & 3] = fma(wr[d], S.vp[col(d)], qs[d & 3]);
                    ts[d & 3] = fma(wt[d], S.vpt[row(d)], ts[d & 3]);
                }
            if constexpr (WIDE) {
                auto entry = [&](int d, double& qk, double& tk) {
                    const int kk = row(d);
                    qk = fma(Wb[d * NMAX + i], S.vp[col(d)], qk);
                    tk = fma(Wb[d * NMAX + kk], S.vpt[kk], tk);
                };
                int d = BAND_REGS;
#pragma unroll 2
                for (; d + 3 < nd; d += 4) {
#pragma unroll
                    for (int e = 0; e < 4; e++) entry(d + e, qs[e], ts[e]);
                }
#pragma unroll
                for (int e = 0; e < 3; e++)
                    if (d + e < nd) entry(d + e, qs[e], ts[e]);
            }
            q = v[0] + ((qs[0] + qs[1]) + (qs[2] + qs[3]));
            qt = vt[0] + ((ts[0] + ts[1]) + (ts[2] + ts[3]));
        }
        qo[0] = q;
        qto[0] = qt;
    };
    double rr[1] = {r}, xx[1] = {xu};
    const double bb[1] = {bval};
    const int done = bicg_iterate<1, G, REC>(S, P, bb, rr, xx, put, mul, capped);
    F[0][IC] = xx[0];
    return done;
}

/* the right-hand side a kernel variant uses */
template <int U, int RHS, int G, int REC>
__device__ __forceinline__ int rhs_eval(const Sys<U, G>& S, const DeviceProblem& P, double T, double (&Xs)[U][UD],
                                        double (&F)[U][UD], double (&up)[U][NUPa], double (&ua)[U][NUAa],
                                        int (&iua)[U][NIUAa], const double (&ra)[U], const double (&cb)[U],
                                        const double (&grow)[16], bool& capped) {
    if constexpr (RHS == 0 && U == 1) {
        return coupled_rhs_quad<G, REC>(S, P, T, Xs, F, ua, iua, capped);
    } else if constexpr (RHS == 0) {
        return coupled_rhs<U, G, REC>(S, P, T, Xs, F, up, ua, iua, capped);
    } else if constexpr (RHS == 4 && U == 1) {
        return coupled_rhs_symquad<G, REC>(S, P, T, Xs, F, ua, iua, ra, cb, capped);
    } else if constexpr (RHS == 3 || RHS == 4) {
        return coupled_rhs_sharedc<U, G, RHS == 4, REC>(S, P, T, Xs, F, up, ua, iua, ra, cb, capped);
    } else if constexpr (RHS > 10) {
        return coupled_rhs_team<(RHS > 14), RHS % 2 == 0 ? 32 : 0, REC>(S, P, T, Xs, F, ua, iua, ra, cb, grow, capped);
    } else if constexpr (RHS == 5 || RHS == 6) {
        static_assert(U == 1 && G == 1, "the register-resident operator needs one unit per lane");
        return coupled_rhs_regsym<RHS == 6 ? 32 : 0, REC>(S, P, T, Xs, F, ua, iua, ra, cb, capped);
    } else if constexpr (RHS == 7 || RHS == 10) {
        static_assert(U == 1, "the banded operator runs one unit per lane");
        return coupled_rhs_band<G, RHS == 10, REC>(S, P, T, Xs, F, ua, iua, capped);
    } else {
        static_assert(U == 1, "the register-resident operator needs one unit per lane");
        return coupled_rhs_regw<RHS == 2 || RHS == 9 ? 32 : 0, REC, (RHS > 7)>(S, P, T, Xs, F, up, ua, iua, capped);
    }
}

/* per-lane state of the units it owns */
template <int U>
struct Lane {
    double X[U][UD];
    double up[U][NUPa];
    double ua[U][NUAa];
    int iua[U][NIUAa];
    double ev_a[U][NEa], ev_n[U][NEa];
    double ra[U], cb[U];   /* coupling factors a_i, b_i of the shared-matrix kernels */
    double grow[16];       /* this lane's share of the shared symmetric matrix (teams) */
};

struct Counters {
    unsigned long long acc, rej, bicg, rhs;
    int status;
};

template <int U, int G>
__device__ __forceinline__ bool valid_unit(const Sys<U, G>& S, int m) { return S.unit(m) < S.N; }

/* the parameter array a callback gets for slot m of this lane */
template <int U, int RHS, int G>
__device__ __forceinline__ double* upar_of(const Sys<U, G>& S, Lane<U>& L, int m) {
    if constexpr (U == 1) return S.upsh + (S.unit(m)) * NUPa;
    else return L.up[m];
}

/* the shared-memory layout of a one-system-at-a-time variant */
template <int U, int RHS, int G>
using OwnSmem = WarpSmem<U, G, (RHS > 10 ? TEAM : RHS > 7 ? 0 : 1)>;

/* are a variant's stage derivatives in shared memory */
template <int U, int RHS, int G>
__device__ constexpr bool stages_shared() {
    if constexpr (RHS == 3 || RHS == 4) return SharedCSmem<U, G, RHS == 4>::K_DOUBLES > 0;
    else if constexpr (RHS == 7 || RHS == 10) return BandSmem<G, RHS == 10>::K_DOUBLES > 0;
    else return OwnSmem<U, RHS, G>::K_DOUBLES > 0;
}

/* The stage derivatives K_j of this lane's units: SHARED in shared memory (each
 * is written once and read a few times a step, while the BiCG needs the
 * registers).  Else, with one unit per lane, in local memory for the same reason
 * (wide bands with REC 1 lack registers: 512 systems of 128 units, CBW 8, 100
 * steps 15.9 ms in registers, 14.2 so; 148 of 60 units, CBW 4, 5.8 and 4.3); with
 * several in registers. */
template <int U, int G, int J, bool SHARED>
struct Stages {
    double k[SHARED ? 1 : J][U][UD];
    __device__ __forceinline__ void set(const Sys<U, G>& S, int st, const double (&F)[U][UD]) {
        if constexpr (SHARED) {
#pragma unroll
            for (int c = 0; c < UD; c++) S.ks[(st * UD + c) * 32 * G + S.unit(0)] = F[0][c];
        } else if constexpr (U == 1) {
#pragma unroll
            for (int c = 0; c < UD; c++) k[st][0][c] = F[0][c];   /* st varies at run time: local memory */
        } else {
#pragma unroll
            for (int j = 0; j < J; j++)
#pragma unroll
                for (int m = 0; m < U; m++)
#pragma unroll
                    for (int c = 0; c < UD; c++)
                        if (j == st) k[j][m][c] = F[m][c];
        }
    }
    __device__ __forceinline__ double get(const Sys<U, G>& S, int j, int m, int c) const {
        if constexpr (SHARED) return S.ks[(j * UD + c) * 32 * G + S.unit(0)];
        else return k[j][m][c];
    }
};

/* Cash-Karp tableau (Steppers.cuh:197-370): stage nodes and coefficients,
 * each entry the double nearest to the reference's literal fraction. */
__constant__ double kCK_A[6][5] = {
    {0.0, 0.0, 0.0, 0.0, 0.0},
    {1.0 / 5.0, 0.0, 0.0, 0.0, 0.0},
    {3.0 / 40.0, 9.0 / 40.0, 0.0, 0.0, 0.0},
    {3.0 / 10.0, -9.0 / 10.0, 6.0 / 5.0, 0.0, 0.0},
    {-11.0 / 54.0, 5.0 / 2.0, -70.0 / 27.0, 35.0 / 27.0, 0.0},
    {1631.0 / 55296.0, 175.0 / 512.0, 575.0 / 13824.0, 44275.0 / 110592.0, 253.0 / 4096.0}};
__constant__ double kCK_C[6] = {0.0, 1.0 / 5.0, 3.0 / 10.0, 3.0 / 5.0, 1.0, 7.0 / 8.0};
/* classical RK4 */
__constant__ double kRK4_A[4] = {0.0, 0.5, 0.5, 1.0};

/* ---------------------------------------------------------------------------
 * RKCK45 step (Steppers.cuh:94-425); returns whether y5 and the error of this lane's units are finite.
 * The six stages run as one loop so the coupled right-hand side is inlined
 * once; stage s evaluates at X + dt * (sum_j<s a_sj K_j) with the terms
 * accumulated in the reference's order (first a product, then fmas). */
template <int U, int RHS, int G, int REC>
__device__ __forceinline__ bool step_rkck45(const Sys<U, G>& S, const DeviceProblem& P, Lane<U>& L,
                                            double T, double dt, double (&Yn)[U][UD], double (&E)[U][UD],
                                            Counters& cnt, bool& capped) {
    Stages<U, G, 6, stages_shared<U, RHS, G>()> K;
    if constexpr (!stages_shared<U, RHS, G>()) {
#pragma unroll
        for (int j = 0; j < 6; j++)
#pragma unroll
            for (int m = 0; m < U; m++)
#pragma unroll
                for (int c = 0; c < UD; c++) K.k[j][m][c] = 0.0;
    }
#pragma unroll 1
    for (int st = 0; st < 6; st++) {
        double Xs[U][UD], F[U][UD];
        double Ts;
        if (st == 0) {
            Ts = T;
#pragma unroll
            for (int m = 0; m < U; m++)
#pragma unroll
                for (int c = 0; c < UD; c++) Xs[m][c] = L.X[m][c];
        } else {
            Ts = st == 4 ? T + dt : fma(kCK_C[st], dt, T);
#pragma unroll
            for (int m = 0; m < U; m++)
#pragma unroll
                for (int c = 0; c < UD; c++) {
                    double acc = K.get(S, 0, m, c) * kCK_A[st][0];
#pragma unroll
                    for (int j = 1; j < 5; j++)
                        if (j < st) acc = fma(K.get(S, j, m, c), kCK_A[st][j], acc);
                    Xs[m][c] = fma(acc, dt, L.X[m][c]);
                }
        }
        cnt.bicg += rhs_eval<U, RHS, G, REC>(S, P, Ts, Xs, F, L.up, L.ua, L.iua, L.ra, L.cb, L.grow, capped);
        K.set(S, st, F);
    }
    cnt.rhs += 6;
    bool finite = true;
#pragma unroll
    for (int m = 0; m < U; m++)
#pragma unroll
        for (int c = 0; c < UD; c++) {
            double s = K.get(S, 0, m, c) * (37.0 / 378.0);
            s = fma(K.get(S, 2, m, c), 250.0 / 621.0, s);
            s = fma(K.get(S, 3, m, c), 125.0 / 594.0, s);
            s = fma(K.get(S, 5, m, c), 512.0 / 1771.0, s);
            Yn[m][c] = fma(s, dt, L.X[m][c]);
            double e = K.get(S, 0, m, c) * (37.0 / 378.0 - 2825.0 / 27648.0);
            e = fma(K.get(S, 2, m, c), 250.0 / 621.0 - 18575.0 / 48384.0, e);
            e = fma(K.get(S, 3, m, c), 125.0 / 594.0 - 13525.0 / 55296.0, e);
            e = fma(K.get(S, 4, m, c), 0.0 - 277.0 / 14336.0, e);
            e = fma(K.get(S, 5, m, c), 512.0 / 1771.0 - 1.0 / 4.0, e);
            E[m][c] = fma(dt, fabs(e), 1e-18);
            if (valid_unit(S, m) && (!isfinite(Yn[m][c]) || !isfinite(E[m][c]))) finite = false;
        }
    return finite;
}

/* classical RK4 step (the reference has only its fixed-step controller,
 * ErrorControllers.cuh:424-450); returns whether this lane's new states are finite */
template <int U, int RHS, int G, int REC>
__device__ __forceinline__ bool step_rk4(const Sys<U, G>& S, const DeviceProblem& P, Lane<U>& L,
                                         double T, double dt, double (&Yn)[U][UD], Counters& cnt, bool& capped) {
    Stages<U, G, 4, stages_shared<U, RHS, G>()> K;
    if constexpr (!stages_shared<U, RHS, G>()) {
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int m = 0; m < U; m++)
#pragma unroll
                for (int c = 0; c < UD; c++) K.k[j][m][c] = 0.0;
    }
#pragma unroll 1
    for (int st = 0; st < 4; st++) {
        double Xs[U][UD], F[U][UD];
        double Ts;
        if (st == 0) {
            Ts = T;
#pragma unroll
            for (int m = 0; m < U; m++)
#pragma unroll
                for (int c = 0; c < UD; c++) Xs[m][c] = L.X[m][c];
        } else {
            Ts = st == 3 ? T + dt : fma(0.5, dt, T);
#pragma unroll
            for (int m = 0; m < U; m++)
#pragma unroll
                for (int c = 0; c < UD; c++) {
                    double kprev = 0.0;
#pragma unroll
                    for (int j = 0; j < 3; j++)
                        if (j == st - 1) kprev = K.get(S, j, m, c);
                    /* stage 3 uses K3 itself (a = 1): fma(K3, dt, X); stages 1, 2 use K*0.5 */
                    Xs[m][c] = st == 3 ? fma(kprev, dt, L.X[m][c]) : fma(kprev * kRK4_A[st], dt, L.X[m][c]);
                }
        }
        cnt.bicg += rhs_eval<U, RHS, G, REC>(S, P, Ts, Xs, F, L.up, L.ua, L.iua, L.ra, L.cb, L.grow, capped);
        K.set(S, st, F);
    }
    cnt.rhs += 4;
    bool finite = true;
#pragma unroll
    for (int m = 0; m < U; m++)
#pragma unroll
        for (int c = 0; c < UD; c++) {
            double s = K.get(S, 0, m, c) * (1.0 / 6.0);
            s = fma(K.get(S, 1, m, c), 1.0 / 3.0, s);
            s = fma(K.get(S, 2, m, c), 1.0 / 3.0, s);
            s = fma(K.get(S, 3, m, c), 1.0 / 6.0, s);
            Yn[m][c] = fma(s, dt, L.X[m][c]);
            if (valid_unit(S, m) && !isfinite(Yn[m][c])) finite = false;
        }
    return finite;
}

/* dense-output store (DenseOutput.cuh:312-361), bounds-checked at the slot */
template <int U, int G>
__device__ __forceinline__ void store_dense(const Sys<U, G>& S, const DeviceProblem& P, const Lane<U>& L,
                                            int& idx, int update_do, int update, int& skipped,
                                            double& do_time, double T, double TD1) {
    if (update_do == 1 && idx < P.ndo && S.lead) {
#pragma unroll
        for (int m = 0; m < U; m++) {
            const int i = S.unit(m);
            if (i < S.N) {
#pragma unroll
                for (int c = 0; c < UD; c++)
                    P.dense_state[(int64_t)idx * UD * S.tot + (int64_t)c * S.tot + S.off + i] = L.X[m][c];
            }
        }
        if (S.lane == 0 && S.wis == 0) P.dense_time[(int64_t)idx * P.n_systems + S.sid] = T;
    }
    if (update_do == 1) {
        idx++;
        skipped = 0;
        do_time = fmin(T + P.do_min_dt, TD1);
    }
    if (update_do == 0 && update == 1) skipped++;
}

/* ---------------------------------------------------------------------------
 * One reference Solve() of one system (Solver.cuh:82-648). */
template <int U, int RHS, int G, int REC>
__device__ __forceinline__ void run_period(const Sys<U, G>& S, const DeviceProblem& P, Lane<U>& L, Counters& cnt,
                           double (&TD)[2], double& T, int& do_idx) {
    const double TD1 = TD[1];
    double dt = P.dt0, newdt = P.dt0;
    int update_do = 1, skipped = 0;
    double do_time = 0.0;
    int udt = 0;
    double rtol[UD], atol[UD];
#pragma unroll
    for (int c = 0; c < UD; c++) {
        rtol[c] = P.rtol[(int64_t)c * P.n_systems + S.sid];
        atol[c] = P.atol[(int64_t)c * P.n_systems + S.sid];
    }
    double evtol[NEa];
    int evdir[NEa];
#pragma unroll
    for (int e = 0; e < NE; e++) { evtol[e] = P.event_tol[e]; evdir[e] = P.event_dir[e]; }

    /* Initialization callback (Solver.cuh:262-280) */
    {
        double Tl = T, dTl = dt;
        int DOl = do_idx;
        int firstT = -1, firstD = -1, firstO = -1;
        double TnewL = T, dTnewL = dt;
        int DOnewL = do_idx;
#pragma unroll
        for (int m = 0; m < U; m++) {
            const int i = S.unit(m);
            if (i < S.N) {
                double Tu = Tl, dTu = dTl;
                int DOu = DOl;
                CoupledSystems_PerBlock_Initialization<double>(S.sid, i, DOu, Tu, dTu, TD, L.X[m], upar_of<U, RHS, G>(S, L, m), S.sPAR,
                                                               S.gPAR, S.igPAR, L.ua[m], L.iua[m], S.sACC, S.isACC);
                if (firstT < 0 && Tu != Tl) { firstT = i; TnewL = Tu; }
                if (firstD < 0 && dTu != dTl) { firstD = i; dTnewL = dTu; }
                if (firstO < 0 && DOu != DOl) { firstO = i; DOnewL = DOu; }
            }
        }
        T = grp_resolve<U, G>(S, T, TnewL, firstT < 0 ? -1 : firstT);
        dt = grp_resolve<U, G>(S, dt, dTnewL, firstD < 0 ? -1 : firstD);
        newdt = dt;
        do_idx = grp_resolve_int<U, G>(S, do_idx, DOnewL, firstO < 0 ? -1 : firstO);
    }
    /* first event values (Solver.cuh:283-305) */
    if (NE > 0) {
#pragma unroll
        for (int m = 0; m < U; m++)
            if (valid_unit(S, m))
                CoupledSystems_PerBlock_EventFunction<double>(S.sid, S.unit(m), L.ev_a[m], T, dt, TD, L.X[m],
                                                              upar_of<U, RHS, G>(S, L, m), S.sPAR, S.gPAR, S.igPAR, L.ua[m], L.iua[m],
                                                              S.sACC, S.isACC);
    }
    if (P.ndo > 0) store_dense<U, G>(S, P, L, do_idx, update_do, 1, skipped, do_time, T, TD1);

    long long attempted = 0;
    bool terminate = false;
    while (!terminate) {
        int update = 1, end = 0;
        dt = newdt;
        if (dt > (TD1 - T)) { dt = TD1 - T; end = 1; }
        if (attempted >= P.max_steps_per_period) { cnt.status |= BES_STATUS_STEP_BUDGET; break; }
        attempted++;
        bool capped = false;
        double Yn[U][UD], E[U][UD];
        bool finite;
        if (P.algorithm == 1) {
            finite = step_rkck45<U, RHS, G, REC>(S, P, L, T, dt, Yn, E, cnt, capped);
            /* ErrorController_RKCK45 (ErrorControllers.cuh:454-542) */
            double rr = 1e30;
            bool within = true;
#pragma unroll
            for (int m = 0; m < U; m++) {
                if (valid_unit(S, m)) {
                    double et[UD], ratio[UD];
                    bool ok = true;
#pragma unroll
                    for (int c = 0; c < UD; c++) {
                        et[c] = fmax(rtol[c] * fmax(fabs(Yn[m][c]), fabs(L.X[m][c])), atol[c]);
                        within = within && E[m][c] < et[c];
                        ratio[c] = math::div_try(et[c], E[m][c], ok);
                    }
                    if (!ok) {
#pragma unroll
                        for (int c = 0; c < UD; c++) ratio[c] = math::div_ieee(et[c], E[m][c]);
                    }
#pragma unroll
                    for (int c = 0; c < UD; c++) rr = fmin(rr, ratio[c]);
                }
            }
            grp_step_votes<U, G>(S, finite, within, capped, rr);
            update = within ? 1 : 0;
            const double expo = within ? 1.0 / 5.0 : 1.0 / 4.0;
            bool ok = true;
            double mult = math::pow_try(rr, expo, ok);
            if (!__all_sync(FULL, ok)) mult = math::pow_general(rr, expo);
            mult = 0.8 * mult;
            if (!isfinite(mult)) finite = false;
            if (!finite) {
                mult = P.shrink;
                update = 0;
                if (dt < P.dtmin * 1.01) { cnt.status |= BES_STATUS_NONFINITE; terminate = true; }
            } else if (dt < P.dtmin * 1.01) {
                cnt.status |= BES_STATUS_MIN_STEP;
                update = 1;
            }
            mult = fmin(mult, P.grow);
            mult = fmax(mult, P.shrink);
            newdt = dt * mult;
            newdt = fmin(newdt, P.dtmax);
            newdt = fmax(newdt, P.dtmin);
        } else {
            finite = step_rk4<U, RHS, G, REC>(S, P, L, T, dt, Yn, cnt, capped);
            bool unused = true;
            double none = 0.0;
            grp_step_votes<U, G>(S, finite, unused, capped, none);
            if (!finite) { cnt.status |= BES_STATUS_NONFINITE; terminate = true; update = 0; }
            newdt = P.dt0;
        }
        if (capped) cnt.status |= BES_STATUS_BICG_CAP;

        if (!terminate && NE > 0) {
            /* next event values at the trial state (Solver.cuh:393-414) */
#pragma unroll
            for (int m = 0; m < U; m++)
                if (valid_unit(S, m))
                    CoupledSystems_PerBlock_EventFunction<double>(S.sid, S.unit(m), L.ev_n[m], T + dt, newdt, TD,
                                                                  Yn[m], upar_of<U, RHS, G>(S, L, m), S.sPAR, S.gPAR, S.igPAR, L.ua[m],
                                                                  L.iua[m], S.sACC, S.isACC);
            if (update == 1) {
                /* EventTimeStepControl (EventHandling.cuh:216-268) */
                double evdt = dt;
                int corrected = 0;
#pragma unroll
                for (int m = 0; m < U; m++) {
                    if (valid_unit(S, m)) {
#pragma unroll
                        for (int e = 0; e < NE; e++) {
                            double a = L.ev_a[m][e], n = L.ev_n[m][e];
                            if ((a > evtol[e] && n < -evtol[e] && evdir[e] <= 0) ||
                                (a < -evtol[e] && n > evtol[e] && evdir[e] >= 0)) {
                                double cand = (-a) / (n - a) * dt;
                                evdt = fmin(evdt, cand);
                                corrected = 1;
                            }
                        }
                    }
                }
                if (grp_any<U, G>(S, corrected)) {
                    evdt = grp_min<U, G>(S, evdt);
                    if (evdt < P.dtmin) {
                        cnt.status |= BES_STATUS_EVENT_MISSED;
                    } else {
                        newdt = evdt;
                        update = 0;
                    }
                }
            }
        }

        if (update == 1) {
            T = T + dt;
#pragma unroll
            for (int m = 0; m < U; m++)
#pragma unroll
                for (int c = 0; c < UD; c++) L.X[m][c] = Yn[m][c];
            cnt.acc++;
            /* ActionAfterSuccessfulTimeStep (Solver.cuh:443-463) */
            {
                double Tl = T, dTl = dt;
                int firstT = -1, firstD = -1, anyU = 0;
                double TnewL = T, dTnewL = dt;
#pragma unroll
                for (int m = 0; m < U; m++) {
                    const int i = S.unit(m);
                    if (i < S.N) {
                        double Tu = Tl, dTu = dTl;
                        int Uu = udt;
                        CoupledSystems_PerBlock_ActionAfterSuccessfulTimeStep<double>(
                            S.sid, i, Uu, Tu, dTu, TD, L.X[m], upar_of<U, RHS, G>(S, L, m), S.sPAR, S.gPAR, S.igPAR, L.ua[m], L.iua[m],
                            S.sACC, S.isACC);
                        if (firstT < 0 && Tu != Tl) { firstT = i; TnewL = Tu; }
                        if (firstD < 0 && dTu != dTl) { firstD = i; dTnewL = dTu; }
                        if (Uu != udt) anyU = 1;
                    }
                }
                if (grp_any<U, G>(S, firstT >= 0 || firstD >= 0 || anyU != 0)) {
                    T = grp_resolve<U, G>(S, T, TnewL, firstT);
                    dt = grp_resolve<U, G>(S, dt, dTnewL, firstD);
                    if (grp_any<U, G>(S, anyU)) udt = 1;
                }
            }
            if (NE > 0) {
                /* ActionAfterEventDetection when an event lands within tolerance (Solver.cuh:465-495) */
                double Tl = T, dTl = dt;
                int firstT = -1, firstD = -1, anyU = 0;
                double TnewL = T, dTnewL = dt;
#pragma unroll
                for (int m = 0; m < U; m++) {
                    const int i = S.unit(m);
                    if (i < S.N) {
#pragma unroll
                        for (int e = 0; e < NE; e++) {
                            double a = L.ev_a[m][e], n = L.ev_n[m][e];
                            if ((a > evtol[e] && fabs(n) < evtol[e] && evdir[e] <= 0) ||
                                (a < -evtol[e] && fabs(n) < evtol[e] && evdir[e] >= 0)) {
                                double Tu = Tl, dTu = dTl;
                                int Uu = udt;
                                CoupledSystems_PerBlock_ActionAfterEventDetection<double>(
                                    S.sid, i, e, Uu, Tu, dTu, TD, L.X[m], upar_of<U, RHS, G>(S, L, m), S.sPAR, S.gPAR, S.igPAR, L.ua[m],
                                    L.iua[m], S.sACC, S.isACC);
                                if (firstT < 0 && Tu != Tl) { firstT = i; TnewL = Tu; }
                                if (firstD < 0 && dTu != dTl) { firstD = i; dTnewL = dTu; }
                                if (Uu != udt) anyU = 1;
                            }
                        }
                    }
                }
                if (grp_any<U, G>(S, firstT >= 0 || firstD >= 0 || anyU != 0)) {
                    T = grp_resolve<U, G>(S, T, TnewL, firstT);
                    dt = grp_resolve<U, G>(S, dt, dTnewL, firstD);
                    if (grp_any<U, G>(S, anyU)) udt = 1;
                }
                /* refresh event values at the accepted state (Solver.cuh:497-525) */
#pragma unroll
                for (int m = 0; m < U; m++)
                    if (valid_unit(S, m))
                        CoupledSystems_PerBlock_EventFunction<double>(S.sid, S.unit(m), L.ev_a[m], T, newdt, TD,
                                                                      L.X[m], upar_of<U, RHS, G>(S, L, m), S.sPAR, S.gPAR, S.igPAR,
                                                                      L.ua[m], L.iua[m], S.sACC, S.isACC);
            }
        } else {
            cnt.rej++;
        }
        if (P.ndo > 0) {
            /* DenseOutputStorageCondition (DenseOutput.cuh:372-395) */
            if (update == 1) {
                update_do = (do_idx < P.ndo && do_time < T && skipped >= (P.do_save_frequency - 1)) ? 1 : 0;
                if (do_idx < P.ndo && (end == 1 || udt == 1)) update_do = 1;
            } else {
                update_do = 0;
            }
            store_dense<U, G>(S, P, L, do_idx, update_do, update, skipped, do_time, T, TD1);
        }
        if (update == 1 && (end == 1 || udt == 1)) terminate = true;
    }
    /* Finalization callback (Solver.cuh:577-595) */
    {
        double Tl = T, dTl = dt;
        int DOl = do_idx;
        int firstT = -1, firstD = -1, firstO = -1;
        double TnewL = T, dTnewL = dt;
        int DOnewL = do_idx;
#pragma unroll
        for (int m = 0; m < U; m++) {
            const int i = S.unit(m);
            if (i < S.N) {
                double Tu = Tl, dTu = dTl;
                int DOu = DOl;
                CoupledSystems_PerBlock_Finalization<double>(S.sid, i, DOu, Tu, dTu, TD, L.X[m], upar_of<U, RHS, G>(S, L, m), S.sPAR,
                                                             S.gPAR, S.igPAR, L.ua[m], L.iua[m], S.sACC, S.isACC);
                if (firstT < 0 && Tu != Tl) { firstT = i; TnewL = Tu; }
                if (firstD < 0 && dTu != dTl) { firstD = i; dTnewL = dTu; }
                if (firstO < 0 && DOu != DOl) { firstO = i; DOnewL = DOu; }
            }
        }
        T = grp_resolve<U, G>(S, T, TnewL, firstT);
        do_idx = grp_resolve_int<U, G>(S, do_idx, DOnewL, firstO);
    }
}

/* ---------------------------------------------------------------------------
 * Per-period analysis (BubbleEnsemble.cu:174-216, moved onto the device): at
 * the start of a call each unit's state is the reference point and the
 * running maximum starts from the unit accessory; after every period the
 * unit's state component 0 goes to that period's Poincare section, the first
 * period whose end state lies within period_tol (Euclidean over the state
 * components) of the reference point is recorded 1-based, and the maximum is
 * raised when the accessory exceeds it.  Everything lives in HBM between
 * periods, so nothing stays in registers across a period. */
template <int U, int G>
__device__ __forceinline__ void analysis_start(const Sys<U, G>& S, const DeviceProblem& P, const Lane<U>& L) {
    if (!S.lead) return;
#pragma unroll
    for (int m = 0; m < U; m++) {
        const int i = S.unit(m);
        if (i >= S.N) continue;
        const int64_t g = S.off + i;
#pragma unroll
        for (int c = 0; c < UD; c++) P.period_ref[(int64_t)c * S.tot + g] = L.X[m][c];
        P.period_number[g] = 0;
        double a = 0.0;
        for (int c = 0; c < NUA; c++)
            if (c == P.max_accessory_index) a = L.ua[m][c];
        P.max_accessory[g] = a;
    }
}

template <int U, int G>
__device__ __forceinline__ void analysis_period_end(const Sys<U, G>& S, const DeviceProblem& P, const Lane<U>& L,
                                                    int per) {
    if (!S.lead) return;
#pragma unroll
    for (int m = 0; m < U; m++) {
        const int i = S.unit(m);
        if (i >= S.N) continue;
        const int64_t g = S.off + i;
        if (per < P.n_sections) P.poincare[(int64_t)per * S.tot + g] = L.X[m][0];
        double d2 = 0.0;
#pragma unroll
        for (int c = 0; c < UD; c++) {
            const double d = P.period_ref[(int64_t)c * S.tot + g] - L.X[m][c];
            d2 = c == 0 ? d * d : d2 + d * d;   /* products rounded, then summed, in component order */
        }
        if (sqrt(d2) < P.period_tol && P.period_number[g] == 0) P.period_number[g] = per + 1;
        double a = 0.0;
        for (int c = 0; c < NUA; c++)
            if (c == P.max_accessory_index) a = L.ua[m][c];
        if (a > P.max_accessory[g]) P.max_accessory[g] = a;
    }
}

/* ---------------------------------------------------------------------------
 * The kernel: groups of G warps pull systems from the work counter.
 * G > 1 runs one unit per lane (U = 1) and exchanges the group's values through
 * shared memory and a named barrier per system slot (barrier 0 is left to
 * __syncthreads).
 * RHS = 0: operator W of the system's own matrix, in tensor memory (G > 1) or in
 * shared memory (several units a lane on one warp); RHS = 1 / 2: U = 1, G = 1,
 * half of W in registers, the column share in shared memory (2 = every system of
 * the launch has exactly 32 units), RHS = 8 / 9 the same with the column share in
 * tensor memory; RHS = 3: every system of the launch shares one coupling matrix,
 * staged in shared memory once per CTA (up to 8 warps per CTA), RHS = 4 the same
 * for a symmetric matrix (both BiCG products as row sums from one read of each
 * entry), in tensor memory for U = 1; RHS = 5 / 6: as 1 / 2 for a shared
 * symmetric matrix; RHS = 7 and 10: the banded operator of narrow and of wide
 * bands; 10 < RHS < 17: the variant RHS - 10 of a system of up to 32 units on a
 * team of warps (coupled_rhs_team).  V > 20 is RHS V - 20 compiled for sixteen
 * warps an SM (128 registers a thread), V = RHS otherwise. */
template <int U, int V, int G, int REC>
__global__ void __launch_bounds__(V > 20 ? 512 : V == 3 || V == 4 || V == 7 || V >= 10 || G > 1 ? 256 : 128, 1)
    bes_ensemble_kernel(DeviceProblem P) {
    constexpr int RHS = V > 20 ? V - 20 : V;
    constexpr bool BAND = RHS == 7 || RHS == 10;
    static_assert(G == 1 || U == 1, "multi-warp systems run one unit per lane");
    static_assert(G == 1 || (RHS != 1 && RHS != 2 && RHS != 5 && RHS != 6),
                  "the register-resident operators are single-warp");
    extern __shared__ double smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int slot = wib / G;
    Sys<U, G> S;
    S.lane = lane;
    S.wis = wib % G;
    S.tw = RHS > 10 ? wib % TEAM : 0;
    S.lead = S.tw == 0;
    S.xt = nullptr;
    S.tsel = 0;
    S.bar = 1u + (unsigned)(RHS > 10 ? wib / TEAM : slot);
    S.xsel = 0;
    S.tot = P.total_units;
    constexpr bool TMEM = tmem_columns<U, RHS, G>(G) > 0;
    __shared__ uint32_t tmem_base;
    const uint32_t tmem_cols = tmem_columns<U, RHS, G>((int)blockDim.x >> 5);
    S.tm = 0;
    if constexpr (TMEM) {
        if (wib == 0) tmem::alloc(&tmem_base, tmem_cols);
        tmem::fence_before_sync();
        __syncthreads();
        tmem::fence_after_sync();
        /* the lanes of this warp's quarter; four warps lie side by side, with RHS 0 the next four behind them */
        S.tm = tmem_base + ((uint32_t)(32 * (wib & 3)) << 16) + (RHS == 0 ? (uint32_t)(4 * 32 * G * (wib >> 2)) : 0u);
    }
    if constexpr (RHS == 4 && U == 1) {
        /* this lane's share of the launch's shared matrix, zero-padded: stored by the CTA's first four warps */
        const int s0 = P.order[0];
        const int n0 = P.units[s0];
        const double* Cg = P.coupling + P.coupling_offset[s0];
        const int c = lane >> 3, row0 = 32 * S.wis + (lane & 7);
        if (wib < 4) {
            for (int ch = 0; ch < 32 * G / 16; ch++) {
                tmem::Chunk m;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int j = 16 * ch + 4 * e + c;
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        m.set(4 * e + k,
                              row0 + 8 * k < n0 && j < n0 ? __ldg(Cg + row0 + 8 * k + (int64_t)j * n0) : 0.0);
                }
                m.store(S.tm + 32 * ch);
            }
            tmem::wait_stores();
        }
        tmem::fence_before_sync();
        __syncthreads();
        tmem::fence_after_sync();
    }
    if constexpr (RHS == 3 || RHS == 4) {
        /* one copy of the launch's shared coupling matrix per CTA, zero-padded (none in shared memory with TMEM) */
        using SM = SharedCSmem<U, G, RHS == 4>;
        constexpr int LDC = SM::LDC;
        const int s0 = P.order[0];
        const int n0 = P.units[s0];
        const double* Cg = P.coupling + P.coupling_offset[s0];
        for (int idx = threadIdx.x; idx < SM::C_DOUBLES; idx += blockDim.x) {
            const int r = idx % LDC, c = idx / LDC;
            smem[idx] = (r < n0 && c < n0) ? __ldg(Cg + r + (int64_t)c * n0) : 0.0;
        }
        __syncthreads();
        constexpr int NM = SM::NMAX;
        double* base = smem + SM::C_DOUBLES + (size_t)slot * SM::WARP_DOUBLES;
        S.W = smem;
        S.vp = base;
        S.vpt = base + NM;
        S.vcpt = base + 2 * NM;
        S.vx1 = base + 3 * NM;
        S.vxu = base + 4 * NM;
        S.vrd = nullptr;
        S.xch = base + 5 * NM;
        S.flag = S.xch + 2 * XCH_BUF;
        S.sPAR = S.xch + SM::XCH_DOUBLES;
        S.upsh = S.sPAR + NSPa + NSAa + NISAa;
    } else if constexpr (BAND) {
        using SM = BandSmem<G, RHS == 10>;
        constexpr int NM = SM::NMAX;
        const int ND = SM::diagonals(P.band_width);
        double* base = smem + (size_t)slot * SM::doubles(P.band_width);
        S.W = base;                                   /* Cb, then Wb */
        S.vp = base + 2 * (size_t)ND * NM;
        S.vpt = S.vp + NM;
        S.vcpt = S.vpt + NM;
        S.vx1 = S.vcpt + NM;
        S.vxu = S.vx1 + NM;
        S.vrd = S.vxu + NM;
        S.xch = S.vrd + NM;
        S.flag = S.xch + 2 * XCH_BUF;
        S.sPAR = S.xch + SM::XCH_DOUBLES + SM::RED_DOUBLES;
        S.upsh = S.sPAR + NSPa + NSAa + NISAa;
    } else {
        using SM = OwnSmem<U, RHS, G>;
        double* base = smem + (size_t)slot * SM::DOUBLES;
        if constexpr (RHS > 10) S.xt = base - (size_t)S.tw * SM::DOUBLES + SM::DOUBLES - SM::XT_DOUBLES;
        S.W = base;
        S.vp = base + SM::W_DOUBLES + SM::WT_DOUBLES;
        S.vpt = S.vp + SM::NMAX;
        S.vcpt = S.vpt + SM::NMAX;
        S.vx1 = S.vcpt + SM::NMAX;
        S.vxu = S.vx1 + SM::NMAX;
        S.vrd = S.vxu + SM::NMAX;
        S.xch = S.vrd + SM::NMAX;
        S.tpar = S.xch + 2 * RED_BUF;   /* U = G = 1 */
        S.rdpar = S.tpar + RED_BUF;
        S.flag = S.xch + 2 * XCH_BUF;
        S.sPAR = S.xch + SM::XCH_DOUBLES + SM::RED_DOUBLES;
        S.upsh = S.sPAR + SM::SYS_DOUBLES;
    }
    S.ks = S.upsh + 32 * U * G * NUPa;
    S.sACC = S.sPAR + NSPa;
    S.isACC = reinterpret_cast<int*>(S.sACC + NSAa);
    S.gPAR = P.gpar;
    S.igPAR = P.igpar;
    /* system-scope loads and stores are done by the group's first warp */
    const bool leader = S.wis == 0;

    Lane<U> L;
    for (;;) {
        int k = 0;
        if (lane == 0 && leader && S.lead) k = atomicAdd(P.work_counter, 1);
        k = __shfl_sync(FULL, k, 0);
        if constexpr (RHS > 10) k = team_share(S, k);
        if constexpr (G > 1) {
            double kk[G];
            grp_share(S, (double)k, kk);
            k = (int)kk[0];
        }
        if (k >= P.n_active) break;
        const int sid = P.order ? P.order[k] : k;
        if (sid < 0 || sid >= P.n_systems) continue;   /* an order slot left unfilled */
        S.sid = sid;
        S.N = P.units[sid];
        S.off = P.unit_offset[sid];
        S.C = P.coupling + P.coupling_offset[sid];
        /* unit-scope loads into registers / local memory (Solver.cuh:234-257) */
#pragma unroll
        for (int m = 0; m < U; m++) {
            const int i = S.unit(m);
            const bool v = i < S.N;
            const int64_t g = S.off + i;
#pragma unroll
            for (int c = 0; c < UD; c++) L.X[m][c] = v ? P.state[(int64_t)c * S.tot + g] : 0.0;
            if constexpr (U == 1) {
                for (int c = 0; c < NUP; c++) S.upsh[i * NUPa + c] = v ? __ldg(P.upar + (int64_t)c * S.tot + g) : 0.0;
            } else {
#pragma unroll
                for (int c = 0; c < NUP; c++) L.up[m][c] = v ? __ldg(P.upar + (int64_t)c * S.tot + g) : 0.0;
            }
            if constexpr ((RHS >= 3 && RHS <= 6) || RHS > 14) {   /* the shared-matrix kernels */
                L.ra[m] = v ? (P.coupling_row_scale ? __ldg(P.coupling_row_scale + g) : 1.0) : 0.0;
                L.cb[m] = v ? (P.coupling_col_scale ? __ldg(P.coupling_col_scale + g) : 1.0) : 0.0;
            } else {
                L.ra[m] = 1.0;
                L.cb[m] = 1.0;
            }
            for (int c = 0; c < NUA; c++) L.ua[m][c] = v ? P.uacc[(int64_t)c * S.tot + g] : 0.0;
#pragma unroll
            for (int c = 0; c < NIUA; c++) L.iua[m][c] = v ? P.iuacc[(int64_t)c * S.tot + g] : 0;
        }
        /* system-scope loads (Solver.cuh:82-130) */
        if (leader) {
            for (int c = lane; c < NSP; c += 32) S.sPAR[c] = P.spar[(int64_t)c * P.n_systems + sid];
            for (int c = lane; c < NSA; c += 32) S.sACC[c] = P.sacc[(int64_t)c * P.n_systems + sid];
            for (int c = lane; c < NISA; c += 32) S.isACC[c] = P.isacc[(int64_t)c * P.n_systems + sid];
        }
        if constexpr (RHS == 0 && U == 1) {
            /* stage the system's coupling matrix, zero-padded and swizzled (see coupled_rhs_quad) */
            constexpr int NM = 32 * G;
            const int r = 32 * S.wis + lane;
#pragma unroll 8
            for (int c = 0; c < NM; c++)
                S.W[(r ^ quad_swizzle(c)) + c * NM] = (r < S.N && c < S.N) ? __ldg(S.C + r + (int64_t)c * S.N) : 0.0;
        }
        if constexpr (RHS > 14) {
            /* row `lane` of the shared symmetric matrix at the columns of this warp's two chains, zero-padded */
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const int j = 4 * (k >> 1) + 2 * (S.tw & 1) + (k & 1);
                L.grow[k] = (lane < S.N && j < S.N) ? __ldg(S.C + lane + (int64_t)j * S.N) : 0.0;
            }
        }
        if constexpr (RHS == 5 || RHS == 6) {
            /* rows 2r, 2r + 1 of the shared symmetric matrix at the columns 4t + 2h + e for lane 2r + h, zero-padded,
             * its entries k and k + 1 as one double2 among the lanes' */
#pragma unroll
            for (int k = 0; k < 32; k++) {
                const int row = (lane & ~1) + (k >> 4), j = 4 * ((k & 15) >> 1) + 2 * (lane & 1) + (k & 1);
                S.W[2 * (32 * (k >> 1) + lane) + (k & 1)] =
                    (row < S.N && j < S.N) ? __ldg(S.C + row + (int64_t)j * S.N) : 0.0;
            }
        }
        if constexpr (BAND) {
            /* stage the system's band: Cb[d][i] = C[i][(i + d - bw) mod N] */
            using SM = BandSmem<G, RHS == 10>;
            constexpr int NM = SM::NMAX;
            const int ND = SM::diagonals(P.band_width);
            const int nd = ND < S.N ? ND : S.N;
            for (int idx = 32 * S.wis + lane; idx < nd * NM; idx += 32 * G) {
                const int d = idx / NM, r = idx % NM;
                const int c = ((r + d - P.band_width) % S.N + S.N) % S.N;
                S.W[idx] = r < S.N ? __ldg(S.C + r + (int64_t)c * S.N) : 0.0;
            }
        }
        if constexpr (RHS == 1 || RHS == 2 || RHS == 8 || RHS == 9 || RHS == 11 || RHS == 12) {
            /* stage the system's coupling matrix, zero-padded to 32 x 33 */
            constexpr int LDC = WarpSmem<1>::LDW;
            for (int idx = lane; idx < 32 * LDC; idx += 32) {
                const int r = idx % LDC, c = idx / LDC;
                S.W[idx] = (r < S.N && c < S.N) ? __ldg(S.C + r + (int64_t)c * S.N) : 0.0;
            }
        }
        double TD[2] = {P.time_domain[sid], P.time_domain[P.n_systems + sid]};
        double T = P.actual_time[sid];
        int do_idx = P.ndo > 0 ? P.dense_index[sid] : 0;
        grp_sync(S);
        Counters cnt = {0ull, 0ull, 0ull, 0ull, 0};
        if (P.period_ref) analysis_start<U, G>(S, P, L);
        for (int per = 0; per < P.n_periods; per++) {
            if (per == P.reset_at) {
#pragma unroll
                for (int m = 0; m < U; m++) {
                    const bool v = S.unit(m) < S.N;
                    for (int c = 0; c < NUA; c++) L.ua[m][c] = v ? P.uacc_reset[c] : 0.0;
#pragma unroll
                    for (int c = 0; c < NIUA; c++) L.iua[m][c] = v ? P.iuacc_reset[c] : 0;
                }
            }
            run_period<U, RHS, G, REC>(S, P, L, cnt, TD, T, do_idx);
            if (P.period_ref) analysis_period_end<U, G>(S, P, L, per);
        }
        /* write-back (Solver.cuh:599-648) */
        grp_sync(S);
#pragma unroll
        for (int m = 0; m < U; m++) {
            const int i = S.unit(m);
            if (i < S.N && S.lead) {
                const int64_t g = S.off + i;
#pragma unroll
                for (int c = 0; c < UD; c++) P.state[(int64_t)c * S.tot + g] = L.X[m][c];
                for (int c = 0; c < NUA; c++) P.uacc[(int64_t)c * S.tot + g] = L.ua[m][c];
#pragma unroll
                for (int c = 0; c < NIUA; c++) P.iuacc[(int64_t)c * S.tot + g] = L.iua[m][c];
            }
        }
        if (leader && S.lead) {
            for (int c = lane; c < NSA; c += 32) P.sacc[(int64_t)c * P.n_systems + sid] = S.sACC[c];
            for (int c = lane; c < NISA; c += 32) P.isacc[(int64_t)c * P.n_systems + sid] = S.isACC[c];
            if (lane == 0) {
                P.actual_time[sid] = T;
                P.time_domain[sid] = TD[0];
                P.time_domain[P.n_systems + sid] = TD[1];
                if (P.ndo > 0) P.dense_index[sid] = do_idx;
                P.n_accepted[sid] += cnt.acc;
                P.n_rejected[sid] += cnt.rej;
                P.n_bicg_iter[sid] += cnt.bicg;
                P.n_rhs[sid] += cnt.rhs;
                P.status[sid] |= cnt.status;
            }
        }
        grp_sync(S);
    }
    if constexpr (TMEM) {
        /* every warp's loads have been waited for */
        tmem::fence_before_sync();
        __syncthreads();
        if (wib == 0) {
            tmem::fence_after_sync();
            tmem::dealloc(tmem_base, tmem_cols);
        }
    }
}

}  // namespace bes

#endif
