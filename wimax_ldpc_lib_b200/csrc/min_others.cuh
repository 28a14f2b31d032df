/*
 * For a check row, the minimum over the other edges of every edge. A min-sum
 * message needs, per edge e, mu_e = min over q != e of |L_q|. Tracking the
 * row's two smallest values costs about 2.3 minima per edge and then a
 * compare and a select per edge to choose between them. Here the edges are
 * taken in groups of three: the group minima (one three-input minimum each)
 * go through the same function, which gives every group the minimum of the
 * other groups, and an edge's result is the three-input minimum of that and
 * its two neighbours. sm_100a's three-input minimum costs as much as a
 * two-input one (2 cycles per warp on the ALU pipe, measured), so a row of 6
 * takes 8 of them, of 7 11, of 10 16, of 20 38: 1.3 to 1.9 per edge, no
 * compares and no selects.
 *
 * For values without NaN mu_e equals the tracked form's (|L_e| == min1 ?
 * min2 : min1), ties included. A NaN is never a minimum (fmin rule), unless
 * an edge's others all are.
 */
#ifndef WLDPC_MIN_OTHERS_CUH
#define WLDPC_MIN_OTHERS_CUH

#include <cstdint>
#include "device_util.cuh"

namespace wldpc {

/* f32 minima */
struct MinF32 {
    using T = float;
    static __device__ __forceinline__ float min2(float a, float b) { return fminf(a, b); }
    static __device__ __forceinline__ float min3(float a, float b, float c)
    {
        float d;
        asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
        return d;
    }
};

/* ... the three-input minimum left to the compiler */
struct MinF32Plain : MinF32 {
    static __device__ __forceinline__ float min3(float a, float b, float c) { return fminf(fminf(a, b), c); }
};

/* two binary16 minima per word */
struct MinH2 {
    using T = uint32_t;
    static __device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b)
    {
        uint32_t d;
        asm("min.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
        return d;
    }
    static __device__ __forceinline__ uint32_t min3(uint32_t a, uint32_t b, uint32_t c) { return min2(min2(a, b), c); }
};

/* out[e] = min of v[q] over q != e (and, with CLAMP and D > 4, of bound) */
template <typename Op, int D, bool CLAMP = false, typename T = typename Op::T>
__device__ __forceinline__ void min_others(const T (&v)[D], T (&out)[D], T bound = T{})
{
    static_assert(D >= 2 && (!CLAMP || D > 4), "rows of two edges or more; clamped ones of five or more");
    if constexpr (D == 2) {
        out[0] = v[1];
        out[1] = v[0];
    } else if constexpr (D == 3) {
        out[0] = Op::min2(v[1], v[2]);
        out[1] = Op::min2(v[0], v[2]);
        out[2] = Op::min2(v[0], v[1]);
    } else if constexpr (D == 4) {
        out[0] = Op::min3(v[1], v[2], v[3]);
        out[1] = Op::min3(v[0], v[2], v[3]);
        out[2] = Op::min3(v[0], v[1], v[3]);
        out[3] = Op::min3(v[0], v[1], v[2]);
    } else {
        constexpr int Q = (D + 2) / 3;
        T group[Q], rest[Q];
        static_for<Q>([&](auto I) {
            constexpr int b = 3 * decltype(I)::value;
            if constexpr (b + 2 < D) group[I] = Op::min3(v[b], v[b + 1], v[b + 2]);
            else if constexpr (b + 1 < D) group[I] = Op::min2(v[b], v[b + 1]);
            else group[I] = v[b];
        });
        min_others<Op, Q>(group, rest);
        static_for<Q>([&](auto I) {
            constexpr int b = 3 * decltype(I)::value;
            if constexpr (CLAMP) rest[I] = Op::min2(rest[I], bound);
            if constexpr (b + 2 < D) {
                out[b] = Op::min3(v[b + 1], v[b + 2], rest[I]);
                out[b + 1] = Op::min3(v[b], v[b + 2], rest[I]);
                out[b + 2] = Op::min3(v[b], v[b + 1], rest[I]);
            } else if constexpr (b + 1 < D) {
                out[b] = Op::min2(v[b + 1], rest[I]);
                out[b + 1] = Op::min2(v[b], rest[I]);
            } else {
                out[b] = rest[I];
            }
        });
    }
}

}  // namespace wldpc

#endif
