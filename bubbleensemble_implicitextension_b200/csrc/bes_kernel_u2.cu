/* bes_kernel_u2.cu -- solver kernel variants for systems of up to 64 units
 * on one warp (two units per lane), the reference's BiCG recurrence. */
#include "bes_kernel_inst.cuh"

namespace bes {
BES_KERNEL_VARIANT(2, 0, 1, 0, BES_SMEM_WARP(2, 1))
BES_KERNEL_VARIANT(2, 3, 1, 0, BES_SMEM_SHARED(2, 1, false))
BES_KERNEL_VARIANT(2, 4, 1, 0, BES_SMEM_SHARED(2, 1, true))
}  // namespace bes
