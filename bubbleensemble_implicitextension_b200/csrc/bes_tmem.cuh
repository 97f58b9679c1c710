/*
 * bes_tmem.cuh -- tensor memory (TMEM, 128 lanes x 512 columns of 32 bits per
 * SM) as per-lane operand storage of the FP64 products.
 *
 * A warp reaches the 32 TMEM lanes of its quarter (warp index mod 4), one per
 * thread, so each thread has up to 256 doubles of its own there, read at four
 * times the rate of shared memory and beside it.  Only the 32x32b shape is used
 * (thread l of the warp: lane l of the quarter), sixteen doubles at a time.
 */
#ifndef BES_TMEM_CUH
#define BES_TMEM_CUH

#include <stdint.h>

namespace bes {
namespace tmem {

/* One warp allocates `columns` (a power of two, 32 to 512) for the CTA; the base address goes to
 * *base in shared memory.  Every CTA that can be resident on the SM has to fit. */
__device__ __forceinline__ void alloc(uint32_t* base, uint32_t columns) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(base);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(a), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void dealloc(uint32_t base, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns));
}
/* around a CTA barrier between one warp's stores and another's loads */
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

/* sixteen doubles of this thread, columns addr .. addr + 31 */
struct Chunk {
    uint32_t r[32];
    __device__ __forceinline__ void set(int k, double v) {
        r[2 * k] = (uint32_t)__double2loint(v);
        r[2 * k + 1] = (uint32_t)__double2hiint(v);
    }
    __device__ __forceinline__ double get(int k) const { return __hiloint2double((int)r[2 * k + 1], (int)r[2 * k]); }
    __device__ __forceinline__ void store(uint32_t addr) const {
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
            "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(addr),
            "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
            "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
            "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
            "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]));
    }
    /* starts the load; the values are there after wait(), which has to follow every load */
    __device__ __forceinline__ void load(uint32_t addr) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(addr));
    }
    /* the registers pass through the wait, so nothing that reads them moves before it */
    __device__ __forceinline__ void wait() {
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                       "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                       "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                       "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                     ::"memory");
    }
};
__device__ __forceinline__ void wait_stores() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

}  // namespace tmem
}  // namespace bes

#endif
