/*
 * What the warps of a unit (unit_decode.cuh) share: their barrier, their
 * votes, and the place and clearing of their messages in tensor memory.
 */
#ifndef WLDPC_UNIT_SYNC_CUH
#define WLDPC_UNIT_SYNC_CUH

#include <cstdint>
#include "codes.h"
#include "device_util.cuh"
#include "tmem.cuh"

namespace wldpc {

/* a unit's barrier and votes. Words: four per unit in shared memory, zero at
 * the start; a vote's word is cleared two votes later. Votes are barriers that
 * order shared memory like sync(): the vote and reduce instructions of a warp
 * order none, so a unit of one warp synchronises before them. */
template <int UW>
struct UnitSync {
    unsigned* words;
    int unit, thread;   /* unit of the CTA, thread of the unit */
    int turn = 0;
    __device__ __forceinline__ void sync() const
    {
        if constexpr (UW == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(unit + 1), "n"(32 * UW) : "memory");
    }
    /* bitwise OR over the unit's threads; a barrier */
    __device__ __forceinline__ unsigned vote(unsigned bits)
    {
        if constexpr (UW == 1) __syncwarp();
        bits = __reduce_or_sync(0xffffffffu, bits);
        if constexpr (UW == 1) {
            return bits;
        } else {
            unsigned* const w = words + (turn & 3);
            if ((thread & 31) == 0 && bits) atomicOr(w, bits);
            sync();
            bits = *(volatile unsigned*)w;
            if (thread == 0) words[(turn + 2) & 3] = 0;
            turn++;
            return bits;
        }
    }
    /* whether any thread's flag is set; a barrier */
    __device__ __forceinline__ unsigned any(bool flag)
    {
        if constexpr (UW == 1) {
            __syncwarp();
            return __any_sync(0xffffffffu, flag) ? 1u : 0u;
        } else {
            unsigned o;
            asm volatile("{\n\t.reg .pred p, s;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred s, %2, %3, p;\n\t"
                         "selp.u32 %0, 1, 0, s;\n\t}"
                         : "=r"(o) : "r"((unsigned)flag), "r"(unit + 1), "n"(32 * UW) : "memory");
            return o;
        }
    }
};

/* the messages of a warp: NBLK columns of its 32 lanes */
__device__ __forceinline__ uint32_t unit_tmem(uint32_t base, int warp, int nblk)
{
    return base + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * nblk);
}
/* ... set to zero, and layer 0's loaded. Nothing orders two stores to a column
 * but a wait between them, so the last layer's, still in flight when a unit
 * starts its next frames, are waited for first. */
template <int R>
__device__ __forceinline__ void unit_clear_messages(uint32_t (&M)[kMaxDeg], uint32_t tm)
{
    constexpr int NBLK = num_blocks(R);
    const uint32_t zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    tm_wait_ld<layer_degree(R, 0)>(M);
    tm_wait_st();
    static_for<(NBLK + 7) / 8>([&](auto C) {
        constexpr int c = 8 * decltype(C)::value;
        tm_st8(zero, tm + (c + 8 <= NBLK ? c : NBLK - 8));
    });
    tm_wait_st();
    tm_ld<layer_degree(R, 0)>(M, tm);
}

}  // namespace wldpc

#endif
