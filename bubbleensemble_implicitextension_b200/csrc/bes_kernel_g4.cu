/* bes_kernel_g4.cu -- solver kernel variants for systems of up to 128 units
 * (one unit per lane, four warps), the reference's BiCG recurrence. */
#include "bes_kernel_inst.cuh"

namespace bes {
BES_KERNEL_VARIANT(1, 0, 4, 0, BES_SMEM_WARP(1, 4))
BES_KERNEL_VARIANT(1, 3, 4, 0, BES_SMEM_SHARED(1, 4, false))
BES_KERNEL_VARIANT(1, 4, 4, 0, BES_SMEM_SHARED(1, 4, true))
BES_KERNEL_VARIANT(1, 7, 4, 0, BES_SMEM_BAND(4, false))
BES_KERNEL_VARIANT(1, 10, 4, 0, BES_SMEM_BAND(4, true))
}  // namespace bes
