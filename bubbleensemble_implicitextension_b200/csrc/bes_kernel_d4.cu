/* bes_kernel_d4.cu -- solver kernel variants for systems of up to 128 units
 * at sixteen warps an SM (one unit per lane, four warps), the reference's BiCG recurrence. */
#include "bes_kernel_inst.cuh"

namespace bes {
BES_KERNEL_VARIANT(1, 24, 4, 0, BES_SMEM_SHARED(1, 4, true))
BES_KERNEL_VARIANT(1, 27, 4, 0, BES_SMEM_BAND(4, false))
}  // namespace bes
