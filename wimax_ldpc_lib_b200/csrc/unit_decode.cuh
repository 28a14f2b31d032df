/*
 * Decoders for large batches: persistent CTAs whose check-to-variable
 * messages live in tensor memory.
 *
 * What bounded the one-frame-per-CTA decoders (nms_decode.cuh, lms.cuh,
 * lms16.cuh) was the register file: 76 to 88 message registers per thread
 * left 15 warps on an SM (9 at some z), too few to cover the dependent chain
 * of a layer, and a CTA of several frames (z not a multiple of 32) ran until
 * its slowest frame stopped. Here a thread keeps its messages, one word per
 * non-zero block, in its own lane of TMEM (512 columns x 128 lanes = 256 KB
 * per SM, otherwise idle): 80 registers per thread, 24 warps on an SM (20 for
 * the 88 blocks of rate 3/4B, 16 for rate 5/6). A layer's messages are loaded while the layer
 * before runs (tcgen05.ld) and stored as they are made (tcgen05.st).
 *
 * One CTA per SM, all its warps cut into units: G frames (frame pairs for binary16) on UW = ceil(G z / 32)
 * warps, with a barrier of their own (a named barrier; __syncwarp for one
 * warp). Units never wait for one another. unit_frames() picks G so that few
 * lanes of a unit idle.
 *
 * A CTA takes frames blockIdx.x, + gridDim.x, ... in order; a slot (frame
 * group of Z threads) draws the next one from a shared counter, one frame
 * ahead, and has it staged by a TMA bulk copy while it decodes. The plain
 * decoder's slots start their next frame as soon as one stops; the learned
 * decoders' units restart together, because their weights go by iteration
 * (one row for the whole unit).
 *
 * Measured against the one-frame-per-CTA kernels of the same arithmetic (ms,
 * outputs identical): r1/2 z=96, 65,536 frames: plain 2.18 -> 2.05, learned
 * fp32 1.32 -> 1.31, binary16 (131,072) 1.66 -> 1.48; r2/3B z=44, 20,011
 * frames: plain 0.326 -> 0.261, learned 0.26 -> 0.19; r3/4B z=28, 30,001
 * frames: 0.255 -> 0.193, 0.19 -> 0.14, binary16 0.17 -> 0.095. What binds
 * now: the ALU and XU pipes for plain (77% and 67% busy, 70% of the issue
 * slots), issue for learned (79-82%), the ALU pipe for binary16 (68%).
 *
 * Every wait on a copy is bounded: when one expires the unit records
 * kErrWaitTimeout, waits (bounded) for the copies it has in flight and ends.
 */
#ifndef WLDPC_UNIT_DECODE_CUH
#define WLDPC_UNIT_DECODE_CUH

#include <cstdint>
#include "codes.h"
#include "device_util.cuh"
#include "lms.cuh"
#include "lms16.cuh"
#include "min_others.cuh"
#include "nms_decode.cuh"
#include "tmem.cuh"
#include "unit_launch.cuh"
#include "unit_sync.cuh"

namespace wldpc {

/* Frames (frame pairs) side by side in a unit. More of them leave fewer lanes
 * idle, but tie more frames to one barrier and, without refill, to the slowest
 * of them: timed at rates 1/2 and 3/4A, 30,000 frames, for every z and one to
 * five frames; the best or within 1% of it for all three decoders. */
constexpr int unit_frames(int z, bool refill)
{
    switch (z) {
    case 24: return refill ? 4 : 1;
    case 36: case 40: return 3;
    case 44: case 48: case 68: case 72: case 76: case 80: return 2;
    default: return 1;
    }
}

template <int R, int Z, bool REFILL>
struct UnitShape {
    static constexpr int MB = kMb[R];
    static constexpr int NBLK = num_blocks(R);
    static constexpr int N = kNB * Z;
    static constexpr int G = unit_frames(Z, REFILL);
    static constexpr int ROWS = G * Z;               /* threads of a unit that own a row */
    static constexpr int UW = (ROWS + 31) / 32;      /* warps of a unit */
    /* as many warps as TMEM holds the messages of; at degree 20 (rate 5/6) 16,
     * whose 128 registers hold a row without spills (r5/6 z=60, 40,000 frames,
     * 24 / 20 / 16 / 12 warps: plain 0.60 / 0.46 / 0.42 / 0.44 ms, learned 0.33 /
     * 0.29 / 0.29 / 0.31), or 12 for plain units of three warps (z=96: 0.75 /
     * 0.77 / 0.75 / 0.71: 15 warps load the SM's four schedulers unevenly). Rows of
     * degree 10 to 15 spill too in 80 or 96 registers, plain rate 3/4A most (124 to
     * 328 bytes per thread); fewer warps were not timed there. */
    static constexpr int WARPS = R == 5 ? (REFILL && UW == 3 ? 12 : 16) : 4 * (512 / NBLK);
    static constexpr int U = UW == 1 ? WARPS : WARPS / UW < 15 ? WARPS / UW : 15;   /* 16 named barriers */
    static constexpr int THREADS = 32 * UW * U;
    static constexpr int SLOTS = U * G;
    static constexpr int SMEM = SLOTS * 2 * N * 4;    /* posteriors and the next frame's LLRs */
    static constexpr int SMEM16 = SLOTS * 3 * N * 4;  /* binary16 pairs and the next pair's LLRs */
    static_assert(SMEM16 <= 226 * 1024, "shared memory of an SM");
};

/* ------------------------------------------------------ what a row does */

/* learned min-sum in fp32: the arithmetic of lms.cuh, so that a frame's outputs
 * do not depend on the batch it comes in. w: (a, b) of the iteration. */
struct LearnedRow {
    using Args = LmsArgs;
    static constexpr UnitKind kKind = kUnitLearned;
    static constexpr bool kLockstep = true;
    const float2* w;
    static __device__ __forceinline__ int cap(const LmsArgs& a) { return a.iters; }
    __device__ __forceinline__ void iteration(const LmsArgs& a, int t)
    {
        /* a uniform row (by a shuffle from lane 0) turned the weights into uniform
         * registers, of which an instruction takes one: 7% more instructions, 2.7% slower */
        w = a.wab[t < a.wrows ? t : a.wrows - 1];
    }
    /* x: posteriors, m: old messages in, new ones out, pn: new posteriors.
     * loaded() is called once the old messages have been read. */
    template <int R, int I, typename F>
    __device__ __forceinline__ void row(const float* x, uint32_t* m, float* pn, F&& loaded) const
    {
        constexpr int d = layer_degree(R, I);
        constexpr int b0 = block_index(R, I, 0);
        float L[d], v[d], mu[d];
        uint32_t sgn = 0;
        static_for<d>([&](auto E) {
            L[E] = __fsub_rn(x[E], __uint_as_float(m[E]));
            v[E] = fabsf(L[E]);
            sgn ^= __float_as_uint(L[E]);
        });
        loaded();
        min_others<MinF32, d>(v, mu);
        /* positive LLR = bit 1: the extrinsic sign flips on odd-degree rows */
        const uint32_t one = ((sgn ^ ((uint32_t)(d & 1) << 31)) & 0x80000000u) | 0x3f800000u;
        static_for<d>([&](auto E) {
            const float2 ab = w[b0 + E];
            const float mag = fmaxf(__fmaf_rn(ab.x, mu[E], -ab.y), 0.0f);
            const float msg = __fmul_rn(mag, __uint_as_float((__float_as_uint(L[E]) & 0x80000000u) ^ one));
            m[E] = __float_as_uint(msg);
            pn[E] = __fadd_rn(L[E], msg);
        });
    }
};

/* plain normalized min-sum in the reference's arithmetic (nms_decode.cuh) */
struct PlainRow {
    using Args = DecodeArgs;
    static constexpr UnitKind kKind = kUnitPlain;
    static constexpr bool kLockstep = false;
    static __device__ __forceinline__ int cap(const DecodeArgs& a) { return a.max_iter; }
    __device__ __forceinline__ void iteration(const DecodeArgs&, int) {}
    template <int R, int I, typename F>
    __device__ __forceinline__ void row(const float* x, uint32_t* m, float* pn, F&& loaded) const
    {
        constexpr int d = layer_degree(R, I);
        float L[d];
        uint32_t LC[d];
        uint32_t sgn = 0;
        float m1, m2;
        static_for<d>([&](auto E) {
            L[E] = __fsub_rn(x[E], __uint_as_float(m[E]));
            LC[E] = __float_as_uint(canon(L[E]));
            sgn ^= LC[E];
        });
        loaded();
        two_min_abs<0, d>(L, m1, m2);
        m1 = fminf(m1, 10000.0f);
        m2 = fminf(m2, 10000.0f);
        const uint32_t fb = (sgn ^ ((uint32_t)(d & 1) << 31)) & 0x80000000u;
        const double D1 = __dmul_rn((double)m1, 0.815), D2 = __dmul_rn((double)m2, 0.815);
        const uint32_t f1 = __float_as_uint(__double2float_rn(D1)) | fb, f2 = __float_as_uint(__double2float_rn(D2)) | fb;
        const int h1 = __double2hiint(D1) ^ (int)fb, l1 = __double2loint(D1);
        const int h2 = __double2hiint(D2) ^ (int)fb, l2 = __double2loint(D2);
        static_for<d>([&](auto E) {
            const bool is_min = fabsf(L[E]) == m1;
            const uint32_t sb = LC[E] & 0x80000000u;
            int hi = is_min ? h2 : h1;
            const int lo = is_min ? l2 : l1;
            hi ^= (int)sb;
            pn[E] = __double2float_rn(__dadd_rn((double)L[E], __hiloint2double(hi, lo)));
            m[E] = (is_min ? f2 : f1) ^ sb;
        });
    }
};

/* ------------------------------------------------------- fp32 posteriors */

template <int R, int Z, class Row>
__global__ void __launch_bounds__(UnitShape<R, Z, !Row::kLockstep>::THREADS, 1)
unit_decode_kernel(const __grid_constant__ typename Row::Args a)
{
    using S = UnitShape<R, Z, !Row::kLockstep>;
    constexpr int MB = S::MB, N = S::N, G = S::G, UT = 32 * S::UW;
    constexpr bool REFILL = !Row::kLockstep || G == 1;   /* a slot starts its next frame by itself */
    constexpr bool FULL = S::ROWS == UT;                 /* every thread owns a row */
    constexpr bool AGES = REFILL && G > 1;               /* slots of a unit at different iterations */
    constexpr unsigned ALL = (1u << G) - 1u;
    extern __shared__ __align__(128) float smem_unit[];
    __shared__ __align__(8) uint64_t s_bar[S::SLOTS][2];
    __shared__ int s_next[S::SLOTS][2];      /* frame in each buffer of a slot, -1 = none */
    __shared__ unsigned s_vote[S::U][4];
    __shared__ uint32_t s_tmem;
    __shared__ int s_ticket;

    const int tid = threadIdx.x, warp = tid >> 5;
    const int u = S::UW == 1 ? warp : tid / UT;
    const int q = tid - u * UT;
    /* the other lanes compute along and store nothing: what they read, maybe while
     * its row's owner writes it, reaches no posterior, vote or output */
    const bool owner = FULL || q < S::ROWS;
    const int g = G == 1 || !owner ? 0 : q / Z;
    const int r = owner ? q - g * Z : (q - S::ROWS) % Z;
    const int slot = u * G + g;
    const bool leader = owner && r == 0;

    if (warp == 0) tm_alloc<512>(&s_tmem);
    for (int k = tid; k < S::SLOTS; k += S::THREADS) {
        mbar_init(&s_bar[k][0], 1);
        mbar_init(&s_bar[k][1], 1);
    }
    for (int k = tid; k < S::U * 4; k += S::THREADS) s_vote[k / 4][k % 4] = 0;
    if (tid == 0) s_ticket = S::SLOTS;   /* the slots' first frames are dealt out, a unit after the other */
    fence_mbar_init();
    tm_fence_before_sync();
    __syncthreads();
    tm_fence_after_sync();
    const uint32_t tm0 = s_tmem;
    const uint32_t tm = unit_tmem(tm0, warp, S::NBLK);
    UnitSync<S::UW> unit{s_vote[u], u, q};

    float* const buf = smem_unit + slot * 2 * N;
    unsigned pend = 0;        /* leader: buffers whose copy it has not waited for */
    /* leader: the ticket's frame, if there is one, into buffer b */
    auto stage = [&](int b, int ticket) {
        const long long f = (long long)blockIdx.x + (long long)ticket * gridDim.x;
        const bool any = f < a.frames;
        s_next[slot][b] = any ? (int)f : -1;
        if (any) {
            pend |= 1u << b;
            fence_proxy_async_smem();   /* the buffer's earlier generic reads come first */
            mbar_arrive_expect_tx(&s_bar[slot][b], N * 4);
            bulk_g2s(buf + b * N, a.llr + f * N, N * 4, &s_bar[slot][b]);
        }
    };
    float* P = buf;           /* the frame's posteriors */
    float *Pr = buf, *Prz = buf;
    int frame = -1;
    auto rows_fail = [&](auto FIRST, auto END) -> bool {
        return tdmp_rows_fail<R, decltype(FIRST)::value, decltype(END)::value>([&](auto I, auto E) {
            return edge_ptr<R, Z, decltype(I)::value, decltype(E)::value>(Pr, Prz, r);
        }) != 0;
    };
    auto fails = [&](bool flag) -> unsigned {   /* failing slots; a barrier */
        if constexpr (G == 1) return unit.any(flag);
        else return unit.vote(flag ? 1u << g : 0u);
    };
    auto write = [&](int iterations, unsigned failed) {
        int8_t* const hard = a.hard + (long long)frame * N;
#pragma unroll
        for (int s = 0; s < 6; s++) {
            const int v4 = r + s * Z;
            const float4 p = reinterpret_cast<const float4*>(P)[v4];
            reinterpret_cast<uint32_t*>(hard)[v4] = (p.x >= 0.0f ? 1u : 0u) | (p.y >= 0.0f ? 1u << 8 : 0u) |
                                                    (p.z >= 0.0f ? 1u << 16 : 0u) | (p.w >= 0.0f ? 1u << 24 : 0u);
            if (a.post) reinterpret_cast<float4*>(a.post + (long long)frame * N)[v4] = p;
        }
        if (a.status && r == 0) a.status[frame] = iterations | (int)(failed << 16);
    };
    using L0 = std::integral_constant<int, 0>;
    using L1 = std::integral_constant<int, 1>;
    using LM = std::integral_constant<int, MB - 1>;
    using LH = std::integral_constant<int, (MB - 1) / 2>;
    using LE = std::integral_constant<int, MB>;

    int b = 1, iters = 0;
    unsigned phase = 0;       /* bit b: parity the next wait on buffer b expects */
    bool fresh = false, warp_fresh = false, aborted = false;
    unsigned act = 0;         /* slots that are decoding */
    unsigned start = ALL;     /* slots to start */
    const int cap = Row::cap(a);
    if (leader) stage(0, g * S::U + u);
    unit.sync();
    Row row;
    uint32_t M[kMaxDeg];      /* the next layer's messages */
#pragma unroll
    for (int e = 0; e < kMaxDeg; e++) M[e] = 0;

    while (true) {
        if (start) {
            if constexpr (!AGES) iters = 0;   /* of every thread: the whole unit starts over */
            unsigned bits = 0;
            if (owner && ((start >> g) & 1u)) {
                const int nb = b ^ 1;
                frame = s_next[slot][nb];
                if (frame >= 0) {
                    if (mbar_wait_bounded(&s_bar[slot][nb], (phase >> nb) & 1u, a.wait_limit_us)) {
                        phase ^= 1u << nb;
                        pend &= ~(1u << nb);
                        b = nb;
                        P = buf + b * N;
                        Pr = P + r;
                        Prz = Pr - Z;
                        iters = 0;
                        fresh = true;
                        if (leader) stage(b ^ 1, atomicAdd(&s_ticket, 1));
                        bits = 1u << (16 + g);
                        if (rows_fail(L0{}, L1{})) bits |= 1u << g;
                    } else {
                        bits = 1u << 31;
                    }
                }
            }
            /* initial syndrome (reference lib/ldpc_decoder.cc:127-139): layer
             * 0's rows first; only frames that pass there check the others */
            bits = unit.vote(bits);
            if (bits >> 31) {
                aborted = true;
                break;
            }
            const unsigned started = (bits >> 16) & ALL;
            unsigned fm = bits & ALL;
            if (started & ~fm) {
                const bool mine = owner && (((started & ~fm) >> g) & 1u);
                fm |= unit.vote(mine && rows_fail(L1{}, LE{}) ? 1u << g : 0u);
            }
            act |= started;
            start = 0;
            const unsigned done = cap == 0 ? started : started & ~fm;
            if (done) {
                if (owner && ((done >> g) & 1u)) write(0, (fm >> g) & 1u);
                act &= ~done;
                if (REFILL || act == 0) {
                    start = REFILL ? done : ALL;
                    unit.sync();   /* the posteriors are read before their buffer is staged again */
                    continue;
                }
            }
            if (act == 0) break;
            if constexpr (AGES) {
                warp_fresh = __any_sync(0xffffffffu, fresh);
                tm_wait_ld<layer_degree(R, 0)>(M);
                tm_ld<layer_degree(R, 0)>(M, tm);
            } else {
                unit_clear_messages<R>(M, tm);
            }
        }
        const bool busy = owner && ((act >> g) & 1u);
        row.iteration(a, iters);
        bool last_odd = false;
        static_for<MB>([&](auto I) {
            constexpr int i = decltype(I)::value;
            constexpr int d = layer_degree(R, i);
            constexpr bool LAST = i == MB - 1;
            constexpr int ni = (i + 1) % MB;
            float x[d], pn[d];
            float* ptr[d];
            static_for<d>([&](auto E) {
                ptr[E] = edge_ptr<R, Z, i, decltype(E)::value>(Pr, Prz, r);
                x[E] = *ptr[E];
            });
            tm_wait_ld<d>(M);
            /* the stores before a layer's next load: those of the iteration
             * before by layer 0, layer 0's own by the last layer */
            if constexpr (i == 0 || LAST) tm_wait_st();
            uint32_t m[d];
            static_for<d>([&](auto E) { m[E] = M[E]; });
            if constexpr (AGES) {
                if (warp_fresh) static_for<d>([&](auto E) { m[E] = fresh ? 0u : m[E]; });
            }
            row.template row<R, i>(x, m, pn, [&]() { tm_ld<layer_degree(R, ni)>(M, tm + block_index(R, ni, 0)); });
            static_for<d>([&](auto E) {
                if ((FULL && G == 1) || busy) *ptr[E] = pn[E];
                if constexpr (LAST) last_odd = last_odd != (pn[E] < 0.0f);
            });
            if constexpr (LAST) last_odd = last_odd != ((d & 1) != 0);
            tm_st<d>(m, tm + block_index(R, i, 0));
            if constexpr (!LAST) unit.sync();
        });
        iters++;
        if constexpr (AGES) {
            fresh = false;
            warp_fresh = false;
        }
        /* stopping rule, as in nms_decode.cuh: the last layer's rows vote on
         * the posteriors they wrote, then the others in two halves */
        unsigned fm, capped;
        if constexpr (AGES) {
            const unsigned v = unit.vote(busy ? (last_odd ? 1u << g : 0u) | (iters >= cap ? 1u << (16 + g) : 0u) : 0u);
            fm = v & ALL;
            capped = v >> 16;
        } else {
            fm = fails(busy && last_odd);
            capped = iters >= cap ? ALL : 0u;
        }
        if (act & ~fm) fm |= fails(owner && (((act & ~fm) >> g) & 1u) && rows_fail(L0{}, LH{}));
        if (act & ~fm) fm |= fails(owner && (((act & ~fm) >> g) & 1u) && rows_fail(LH{}, LM{}));
        const unsigned done = act & (~fm | capped);
        if (done) {
            if (owner && ((done >> g) & 1u)) write(iters, (fm >> g) & 1u);
            act &= ~done;
            if (REFILL || act == 0) {
                start = REFILL ? done : ALL;
                unit.sync();   /* as above */
            }
        }
    }
    tm_wait_ld<layer_degree(R, 0)>(M);
    tm_wait_st();
    if (aborted && leader) {
        atomicOr(a.err, kErrWaitTimeout);
        for (int k = 0; k < 2; k++)   /* let the copies in flight land before the CTA ends */
            if ((pend >> k) & 1u) mbar_wait_bounded(&s_bar[slot][k], (phase >> k) & 1u, kWaitLimitUs);
    }
    tm_fence_before_sync();
    __syncthreads();
    tm_fence_after_sync();
    if (warp == 0) tm_dealloc<512>(tm0);
}

/* ----------------------------------------- binary16 pairs (lms16.cuh) */

/* The packed-binary16 learned decoder in the same frame: a slot is a pair of
 * frames, one per 16-bit lane, and a unit's pairs restart together. A frame
 * that stops is written at once; its lane then runs on unread until the
 * unit's last frame stops, so nothing has to freeze it. */
template <int R, int Z>
__global__ void __launch_bounds__(UnitShape<R, Z, false>::THREADS, 1)
unit_decode16_kernel(const __grid_constant__ Lms16Args a)
{
    using S = UnitShape<R, Z, false>;
    constexpr int MB = S::MB, N = S::N, G = S::G, UT = 32 * S::UW;
    constexpr bool FULL = S::ROWS == UT;
    extern __shared__ __align__(128) float smem_unit[];
    __shared__ __align__(8) uint64_t s_bar[S::SLOTS];
    __shared__ int s_next[S::SLOTS];         /* first frame of the staged pair, -1 = none */
    __shared__ unsigned s_vote[S::U][4];
    __shared__ uint32_t s_tmem;
    __shared__ int s_ticket;

    const int tid = threadIdx.x, warp = tid >> 5;
    const int u = S::UW == 1 ? warp : tid / UT;
    const int q = tid - u * UT;
    const bool owner = FULL || q < S::ROWS;
    const int g = G == 1 || !owner ? 0 : q / Z;
    const int r = owner ? q - g * Z : (q - S::ROWS) % Z;
    const int slot = u * G + g;
    const bool leader = owner && r == 0;

    if (warp == 0) tm_alloc<512>(&s_tmem);
    for (int k = tid; k < S::SLOTS; k += S::THREADS) mbar_init(&s_bar[k], 1);
    for (int k = tid; k < S::U * 4; k += S::THREADS) s_vote[k / 4][k % 4] = 0;
    if (tid == 0) s_ticket = S::SLOTS;
    fence_mbar_init();
    tm_fence_before_sync();
    __syncthreads();
    tm_fence_after_sync();
    const uint32_t tm0 = s_tmem;
    const uint32_t tm = unit_tmem(tm0, warp, S::NBLK);
    UnitSync<S::UW> unit{s_vote[u], u, q};

    uint32_t* const P = reinterpret_cast<uint32_t*>(smem_unit) + slot * N;
    float* const llr = smem_unit + S::SLOTS * N + slot * 2 * N;
    float* const Pr = reinterpret_cast<float*>(P) + (owner ? r : 0);
    float* const Prz = owner ? Pr - Z : Pr;
    auto at = [&](auto I, auto E) -> uint32_t* {
        return reinterpret_cast<uint32_t*>(edge_ptr<R, Z, decltype(I)::value, decltype(E)::value>(Pr, Prz, r));
    };
    bool pend = false;
    auto stage = [&](int ticket) {
        const long long f = 2 * ((long long)blockIdx.x + (long long)ticket * gridDim.x);
        const long long left = a.frames - f;
        s_next[slot] = left > 0 ? (int)f : -1;
        if (left > 0) {
            const uint32_t bytes = (left > 1 ? 2 : 1) * N * 4;
            pend = true;
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(&s_bar[slot], bytes);
            bulk_g2s(llr, a.llr + f * N, bytes, &s_bar[slot]);
        }
    };
    /* failing frames of this thread's rows in layers FIRST .. END-1: bit 2g + lane */
    auto rows_fail = [&](auto FIRST, auto END) -> unsigned {
        uint32_t acc = 0;
        static_for<decltype(END)::value - decltype(FIRST)::value>([&](auto I_) {
            using I = std::integral_constant<int, decltype(FIRST)::value + decltype(I_)::value>;
            constexpr int d = layer_degree(R, I::value);
            uint32_t x = (d & 1) ? kH2Sign : 0u;   /* parity of the hard bits: d minus the negatives */
            static_for<d>([&](auto E_) { x ^= *at(I{}, E_); });
            acc |= x;
        });
        return acc;
    };
    auto bits_of = [&](uint32_t acc) -> unsigned { return (((acc >> 15) & 1u) | ((acc >> 30) & 2u)) << (2 * g); };
    int frame = -1;
    auto write = [&](unsigned lanes, int iterations, unsigned failed) {
#pragma unroll
        for (int s = 0; s < 6; s++) {
            const int v4 = r + s * Z;
            const uint4 w = reinterpret_cast<const uint4*>(P)[v4];
#pragma unroll
            for (int lane = 0; lane < 2; lane++) {
                if (!((lanes >> lane) & 1u)) continue;
                const long long f = frame + lane;
                const int sh = 15 + 16 * lane;
                reinterpret_cast<uint32_t*>(a.hard + f * N)[v4] =
                    ((~w.x >> sh) & 1u) | (((~w.y >> sh) & 1u) << 8) | (((~w.z >> sh) & 1u) << 16) |
                    (((~w.w >> sh) & 1u) << 24);
                if (a.post)
                    reinterpret_cast<float4*>(a.post + f * N)[v4] =
                        make_float4(h2_lane_to_float(w.x, lane), h2_lane_to_float(w.y, lane),
                                    h2_lane_to_float(w.z, lane), h2_lane_to_float(w.w, lane));
            }
        }
        if (a.status && r == 0)
            for (int lane = 0; lane < 2; lane++)
                if ((lanes >> lane) & 1u) a.status[frame + lane] = iterations | (int)(((failed >> lane) & 1u) << 16);
    };
    using L0 = std::integral_constant<int, 0>;
    using L1 = std::integral_constant<int, 1>;
    using LM = std::integral_constant<int, MB - 1>;
    using LH = std::integral_constant<int, (MB - 1) / 2>;
    using LE = std::integral_constant<int, MB>;

    unsigned phase = 0, act = 0;   /* act: frames that are decoding */
    bool aborted = false;
    int t = 0;
    if (leader) stage(g * S::U + u);
    unit.sync();
    uint32_t M[kMaxDeg];
#pragma unroll
    for (int e = 0; e < kMaxDeg; e++) M[e] = 0;

    while (true) {
        if (act == 0) {
            /* the next pairs: wait for their LLRs, clamp and round them into P */
            unsigned bits = 0;
            if (owner) {
                frame = s_next[slot];
                if (frame >= 0) {
                    if (mbar_wait_bounded(&s_bar[slot], phase, a.wait_limit_us)) {
                        const bool two = frame + 1 < a.frames;
                        phase ^= 1u;
                        pend = false;
#pragma unroll
                        for (int s = 0; s < 6; s++) {
                            const int v4 = r + s * Z;
                            const float4 x0 = reinterpret_cast<const float4*>(llr)[v4];
                            const float4 x1 = two ? reinterpret_cast<const float4*>(llr + N)[v4]
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
                            reinterpret_cast<uint4*>(P)[v4] = make_uint4(h2_stage(x0.x, x1.x), h2_stage(x0.y, x1.y),
                                                                         h2_stage(x0.z, x1.z), h2_stage(x0.w, x1.w));
                        }
                        bits = (two ? 3u : 1u) << (2 * g);
                    } else {
                        bits = 1u << 31;
                    }
                }
            }
            act = unit.vote(bits);
            if (act >> 31) {
                aborted = true;
                break;
            }
            if (act == 0) break;
            if (leader) stage(atomicAdd(&s_ticket, 1));
            /* initial syndrome: layer 0's rows first */
            unsigned fm = unit.vote(bits & bits_of(rows_fail(L0{}, L1{})));
            if (act & ~fm) fm |= unit.vote((bits & ~fm) ? bits & ~fm & bits_of(rows_fail(L1{}, LE{})) : 0u);
            const unsigned done = act & ~fm;
            if (owner && ((done >> (2 * g)) & 3u)) write((done >> (2 * g)) & 3u, 0, 0u);
            act &= fm;
            t = 0;
            if (done) unit.sync();   /* the outputs are read before a layer, or the next pairs, change P */
            if (act == 0) continue;
            unit_clear_messages<R>(M, tm);
        }
        const bool busy = owner && ((act >> (2 * g)) & 3u);
        /* the shuffle makes the row uniform: 1.5% faster here, unlike in LearnedRow */
        const uint2* const w = a.wab[__shfl_sync(0xffffffffu, t < a.wrows ? t : a.wrows - 1, 0)];
        uint32_t last_par = 0;
        static_for<MB>([&](auto I) {
            constexpr int i = decltype(I)::value;
            constexpr int d = layer_degree(R, i);
            constexpr int b0 = block_index(R, i, 0);
            constexpr bool LAST = i == MB - 1;
            constexpr int ni = (i + 1) % MB;
            uint32_t L[d], A[d], mu[d], m[d];
            uint32_t* ptr[d];
            uint32_t sgn = 0;
            static_for<d>([&](auto E) {
                ptr[E] = at(I, E);
                L[E] = *ptr[E];
            });
            tm_wait_ld<d>(M);
            if constexpr (i == 0 || LAST) tm_wait_st();
            static_for<d>([&](auto E) {
                L[E] = h2_sub(L[E], M[E]);
                A[E] = h2_abs(L[E]);
                sgn ^= L[E];
            });
            tm_ld<layer_degree(R, ni)>(M, tm + block_index(R, ni, 0));
            min_others<MinH2, d, true>(A, mu, kH2Clamp);
            /* the sign as a factor +-1 (exact): the FMA pipe has room, the ALU pipe,
             * 68% busy with the sign ORed in, has not (262,144 r1/2 z=96 frames 3.02 ->
             * 2.96 ms); the posterior as one fma, L + msg exactly */
            const uint32_t one = ((sgn ^ ((d & 1) ? kH2Sign : 0u)) & kH2Sign) | 0x3c003c00u;
            static_for<d>([&](auto E) {
                const uint2 ab = w[b0 + E];
                const uint32_t mag = h2_fma_relu(ab.x, mu[E], ab.y);
                const uint32_t sign = (L[E] & kH2Sign) ^ one;
                m[E] = h2_mul(mag, sign);
                const uint32_t pn = h2_fma(mag, sign, L[E]);
                if ((FULL && G == 1) || busy) *ptr[E] = pn;
                if constexpr (LAST) last_par ^= pn;
            });
            if constexpr (LAST && (d & 1)) last_par ^= kH2Sign;
            tm_st<d>(m, tm + b0);
            if constexpr (!LAST) unit.sync();
        });
        t++;
        const unsigned mine = owner ? act & (3u << (2 * g)) : 0u;
        unsigned fm = unit.vote(mine & bits_of(last_par));
        if (act & ~fm) fm |= unit.vote((mine & ~fm) ? mine & ~fm & bits_of(rows_fail(L0{}, LH{})) : 0u);
        if (act & ~fm) fm |= unit.vote((mine & ~fm) ? mine & ~fm & bits_of(rows_fail(LH{}, LM{})) : 0u);
        const unsigned done = t >= a.iters ? act : act & ~fm;
        if (done) {
            if (owner && ((done >> (2 * g)) & 3u)) write((done >> (2 * g)) & 3u, t, fm >> (2 * g));
            act &= ~done;
            unit.sync();   /* the outputs are read before the next layer, or the next pairs, change P */
        }
    }
    tm_wait_ld<layer_degree(R, 0)>(M);
    tm_wait_st();
    if (aborted && leader) {
        atomicOr(a.err, kErrWaitTimeout);
        if (pend) mbar_wait_bounded(&s_bar[slot], phase, kWaitLimitUs);
    }
    tm_fence_before_sync();
    __syncthreads();
    tm_fence_after_sync();
    if (warp == 0) tm_dealloc<512>(tm0);
}

/* ------------------------------------------------------------- launches */

/* what the dispatch tables hold for a code; nothing where the unit kernel is never the faster */
template <int R, int Z, class Row>
constexpr UnitLaunch<typename Row::Args> unit_launch()
{
    constexpr long long from = unit_min_frames(Row::kKind, R, Z);
    if constexpr (from < 0) {
        return {};
    } else {
        using S = UnitShape<R, Z, !Row::kLockstep>;
        return {&unit_decode_kernel<R, Z, Row>, S::THREADS, S::SMEM, 1, from};
    }
}
template <int R, int Z>
constexpr UnitLaunch<Lms16Args> unit_launch16()
{
    constexpr long long from = unit_min_frames(kUnitLearned16, R, Z);
    if constexpr (from < 0) {
        return {};
    } else {
        using S = UnitShape<R, Z, false>;
        return {&unit_decode16_kernel<R, Z>, S::THREADS, S::SMEM16, 2, from};
    }
}

}  // namespace wldpc

#endif
