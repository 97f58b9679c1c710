/* bes_kernel_inst.cuh -- host entry points (shared-memory size, occupancy,
 * launch) of one solver kernel instantiation; each bes_kernel_*.cu unit
 * instantiates the variants of one layout class with one BiCG recurrence, so
 * the units compile in parallel. */
#ifndef BES_KERNEL_INST_CUH
#define BES_KERNEL_INST_CUH

#include "bes_kernel.cuh"
#include "bes_launch.h"

/* SMEM: dynamic shared memory of a CTA of `warps` warps (`band`: the band width of the banded variant) */
#define BES_KERNEL_VARIANT(U_, RHS_, G_, REC_, SMEM)                                                          \
    template <>                                                                                               \
    size_t cta_smem_t<U_, RHS_, G_, REC_>(int warps, int band) {                                              \
        (void)band;                                                                                           \
        return (SMEM);                                                                                        \
    }                                                                                                         \
    template <>                                                                                               \
    cudaError_t occupancy_t<U_, RHS_, G_, REC_>(int warps, int band, int* ctas_per_sm) {                      \
        const size_t smem = cta_smem_t<U_, RHS_, G_, REC_>(warps, band);                                      \
        if (smem > 48 * 1024) {                                                                               \
            cudaError_t e = cudaFuncSetAttribute(bes_ensemble_kernel<U_, RHS_, G_, REC_>,                     \
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);     \
            if (e != cudaSuccess) return e;                                                                   \
        }                                                                                                     \
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, bes_ensemble_kernel<U_, RHS_, G_, REC_>, \
                                                             32 * warps, smem);                               \
    }                                                                                                         \
    template <>                                                                                               \
    cudaError_t launch_t<U_, RHS_, G_, REC_>(const DeviceProblem& P, int grid, int warps, cudaStream_t stream) { \
        bes_ensemble_kernel<U_, RHS_, G_, REC_><<<grid, 32 * warps, cta_smem_t<U_, RHS_, G_, REC_>(warps, P.band_width), \
                                                  stream>>>(P);                                               \
        return cudaGetLastError();                                                                            \
    }

/* at least the share of an SM's shared memory (228 KB, 1 KB reserved and a few words static per
 * CTA) that the CTA takes of its 512 columns of tensor memory: whatever launches share an SM, the
 * columns of the CTAs that fit are there, and an allocation never waits for another CTA */
inline size_t tmem_fit(size_t smem, int columns) {
    if (columns == 0) return smem;
    size_t least = (size_t)228 * 1024 * columns / 512 - 1024 - 256;
    if (least > 226 * 1024) least = 226 * 1024;
    return smem > least ? smem : least;
}

/* per-system shared memory (operator or staged matrix per system) */
#define BES_SMEM_WARP(U_, G_) \
    tmem_fit((size_t)(warps / (G_)) * WarpSmem<U_, G_>::BYTES, tmem_columns<U_, ((U_) == 1 && (G_) > 1 ? 0 : 1), G_>(warps))
/* one warp a system, its column share of W in tensor memory */
#define BES_SMEM_WARP_TMEM(RHS_) \
    tmem_fit((size_t)warps * WarpSmem<1, 1, 0>::BYTES, tmem_columns<1, RHS_, 1>(warps))
/* a team's warps, each with its own region */
#define BES_SMEM_TEAM (size_t)warps * WarpSmem<1, 1, TEAM>::BYTES
/* per-system band of the coupling matrix, sized by the run-time band width */
#define BES_SMEM_BAND(G_, WIDE_) (size_t)(warps / (G_)) * (size_t)BandSmem<G_, WIDE_>::doubles(band) * 8
/* one staged matrix per CTA plus per-system vectors */
#define BES_SMEM_SHARED(U_, G_, SYM_)                                    \
    tmem_fit((size_t)SharedCSmem<U_, G_, SYM_>::C_BYTES +                \
                 (size_t)(warps / (G_)) * SharedCSmem<U_, G_, SYM_>::WARP_BYTES, \
             tmem_columns<U_, (SYM_) ? 4 : 3, G_>(warps))

#endif
