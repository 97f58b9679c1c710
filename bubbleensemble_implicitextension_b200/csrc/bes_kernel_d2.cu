/* bes_kernel_d2.cu -- solver kernel variants for systems of up to 64 units
 * at sixteen warps an SM (one unit per lane, two warps), the reference's BiCG recurrence. */
#include "bes_kernel_inst.cuh"

namespace bes {
BES_KERNEL_VARIANT(1, 24, 2, 0, BES_SMEM_SHARED(1, 2, true))
BES_KERNEL_VARIANT(1, 27, 2, 0, BES_SMEM_BAND(2, false))
}  // namespace bes
