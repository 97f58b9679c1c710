/* bes_kernel_t4_r1.cu -- solver kernel variants for systems of up to 32 units
 * (one unit per lane) on a team of four warps, the single-reduction BiCG recurrence. */
#include "bes_kernel_inst.cuh"

namespace bes {
BES_KERNEL_VARIANT(1, 11, 1, 1, BES_SMEM_TEAM)
BES_KERNEL_VARIANT(1, 12, 1, 1, BES_SMEM_TEAM)
BES_KERNEL_VARIANT(1, 15, 1, 1, BES_SMEM_TEAM)
BES_KERNEL_VARIANT(1, 16, 1, 1, BES_SMEM_TEAM)
}  // namespace bes
