/*
 * Tensor memory (TMEM) as a register extension: helpers that move D 32-bit
 * words per thread between registers and consecutive TMEM columns of the
 * thread's own lane (tcgen05.ld / tcgen05.st, shape 32x32b). A warp reaches
 * only the 32 lanes 32 * (warp index mod 4) .. + 31, all 512 columns.
 *
 * tcgen05.ld and .st are asynchronous: the loaded registers are passed
 * through the wait (tm_wait_ld) so that no use of them can be scheduled
 * before it, and a store is visible to a later load of the same columns
 * after tm_wait_st. Every function is warp-collective.
 */
#ifndef WLDPC_TMEM_CUH
#define WLDPC_TMEM_CUH

#include <cstdint>
#include "device_util.cuh"

namespace wldpc {

__device__ __forceinline__ void tm_ld1(uint32_t* r, uint32_t a)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r[0]) : "r"(a) : "memory");
}
__device__ __forceinline__ void tm_ld2(uint32_t* r, uint32_t a)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void tm_ld4(uint32_t* r, uint32_t a)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void tm_ld8(uint32_t* r, uint32_t a)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(a) : "memory");
}
__device__ __forceinline__ void tm_st1(const uint32_t* r, uint32_t a)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(a), "r"(r[0]) : "memory");
}
__device__ __forceinline__ void tm_st2(const uint32_t* r, uint32_t a)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(a), "r"(r[0]), "r"(r[1]) : "memory");
}
__device__ __forceinline__ void tm_st4(const uint32_t* r, uint32_t a)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
                 ::"r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void tm_st8(const uint32_t* r, uint32_t a)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

/* D columns from a on, in pieces of 8, 4, 2 and 1 */
template <int D>
__device__ __forceinline__ void tm_ld(uint32_t* r, uint32_t a)
{
    constexpr int P = D >= 8 ? 8 : D >= 4 ? 4 : D >= 2 ? 2 : 1;
    if constexpr (P == 8) tm_ld8(r, a);
    else if constexpr (P == 4) tm_ld4(r, a);
    else if constexpr (P == 2) tm_ld2(r, a);
    else tm_ld1(r, a);
    if constexpr (D > P) tm_ld<D - P>(r + P, a + P);
}
template <int D>
__device__ __forceinline__ void tm_st(const uint32_t* r, uint32_t a)
{
    constexpr int P = D >= 8 ? 8 : D >= 4 ? 4 : D >= 2 ? 2 : 1;
    if constexpr (P == 8) tm_st8(r, a);
    else if constexpr (P == 4) tm_st4(r, a);
    else if constexpr (P == 2) tm_st2(r, a);
    else tm_st1(r, a);
    if constexpr (D > P) tm_st<D - P>(r + P, a + P);
}

/* wait for this thread's loads; the D loaded words are tied to the wait (volatile
 * asm statements keep their order), so no use of them moves before it */
template <int D, int N>
__device__ __forceinline__ void tm_wait_ld(uint32_t (&r)[N])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < D; i++) asm volatile("" : "+r"(r[i])::"memory");
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

/* one whole warp; blocks until the columns are free on the SM */
template <int COLS>
__device__ __forceinline__ void tm_alloc(uint32_t* dst_smem)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_smem)), "n"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int COLS>
__device__ __forceinline__ void tm_dealloc(uint32_t base)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(COLS) : "memory");
}
__device__ __forceinline__ void tm_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tm_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

}  // namespace wldpc

#endif
