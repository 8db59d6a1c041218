// tmem.cuh -- tensor memory (TMEM, sm_100a) as per-thread storage.
//
// TMEM is 128 lanes x 512 columns of 32-bit cells per SM.  A warp reaches only the 32 lanes of
// its quadrant (warp id mod 4): with the 32x32b shape each thread reads or writes its own lane,
// `num` consecutive columns starting at the address's column.  Address: lane << 16 | column.
// These helpers keep thread-private data (a kernel's accumulator) there, off shared memory.
// Every call is warp-collective (.sync.aligned): all 32 lanes execute it with the same address.
#pragma once

#include <cstdint>

namespace cbs {

// allocate ncols columns (a power of two, 32..512) for this CTA; the base address lands in
// *slot (shared memory).  Executed by one whole warp.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(slot));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(a), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

// free what tmem_alloc returned; one whole warp, after every thread's last access (ordered by
// tmem_fence_before / a CTA barrier / tmem_fence_after)
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// the TMEM address of column `col` in the calling warp's lane quadrant
__device__ __forceinline__ uint32_t tmem_quadrant_addr(uint32_t base, uint32_t col) {
    const uint32_t quadrant = (threadIdx.x >> 5) & 3u;
    return base + ((quadrant * 32u) << 16) + col;
}

// 16 consecutive columns of this thread's lane <-> r[0..15]; the load waits for its data
__device__ __forceinline__ void tmem_load16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_store16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// 32 consecutive columns into r[0..31]; the load waits for its data
__device__ __forceinline__ void tmem_load32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// four columns into r[0..3], without the wait (tmem_wait_load before r is used)
__device__ __forceinline__ void tmem_load4_nowait(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}
template <int COUNT>
__device__ __forceinline__ void tmem_wait_load(uint32_t (&r)[COUNT][4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < COUNT; ++k)  // later uses of r stay behind the wait
        asm volatile("" : "+r"(r[k][0]), "+r"(r[k][1]), "+r"(r[k][2]), "+r"(r[k][3]));
}

// one complex value in four columns
__device__ __forceinline__ void tmem_store_complex(uint32_t taddr, double2 a) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr),
                 "r"(__double2loint(a.x)), "r"(__double2hiint(a.x)), "r"(__double2loint(a.y)),
                 "r"(__double2hiint(a.y))
                 : "memory");
}
// complex value k of loaded words
template <int WORDS>
__device__ __forceinline__ double2 tmem_complex(const uint32_t (&r)[WORDS], int k) {
    return make_double2(__hiloint2double(static_cast<int>(r[4 * k + 1]), static_cast<int>(r[4 * k])),
                        __hiloint2double(static_cast<int>(r[4 * k + 3]), static_cast<int>(r[4 * k + 2])));
}
// 8 consecutive columns into r[0..7]; the load waits for its data
__device__ __forceinline__ void tmem_load8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr)
        : "memory");
}

// the stores issued so far by this thread have completed (before TMEM is read again or freed)
__device__ __forceinline__ void tmem_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

}  // namespace cbs
