/*
 * Learned (neural) normalized/offset min-sum: decoder, training forward /
 * backward, and Adam, for sm_100a.
 *
 * The model generalises the reference's two min-sum flavours (reference
 * lib/ldpc_decoder.cc:17-21,220-231: message = s * min * 0.815, or
 * s * max(min - 0.10, 0)) to one scale a and one offset b per (iteration t,
 * layer i, base column c):
 *
 *   L_e   = P[v_e] - m_e                       (float)
 *   mu_e  = min over the other edges of |L|
 *   m'_e  = s_e * max(a[t,i,c_e] * mu_e - b[t,i,c_e], 0)      (fmaf)
 *   P[v_e] = L_e + m'_e
 *
 * with s_e the sign the other edges imply (sign bit = signbit; positive LLR =
 * bit 1, so an odd-degree row flips the product of the other signs) applied
 * as a product with +-1.0 (the reference's MS form s * min; it flips the
 * sign bit of the magnitude exactly, signed zeros included), the
 * same layered schedule as the plain decoder, T <= 8 trained iterations
 * (a decoder may run past T with the weights of iteration T-1), and
 * the reference's stopping rule (slice x >= 0, stop at a zero syndrome).
 * Weights a = 0.815, b = 0 give a float normalized min-sum.
 * A NaN L (from inf - inf, or in the input) is no minimum of another edge and
 * counts as positive; an edge whose others are all NaN gets the message 0. The
 * hard bit of a NaN is 0, though the stopping rule counts it as 1 (not x < 0).
 *
 * Messages: the decoder keeps every edge's message in a register of the
 * thread that owns the edge's row (one per non-zero block: 76 to 88), so
 * pass 1 reads the old message without a load and without recomputing it
 * from compressed state and the previous iteration's weights; shared memory
 * holds only the posteriors. The weights are read from the kernel
 * parameters as (a, b) pairs (staging them in shared memory measured 21%
 * slower). The sign
 * parity is an XOR of the L words; the minima over the other edges come from
 * min_others(), without the compare and select per edge that tracking the two
 * smallest needed (r1/2 z=96, 65,536 frames: 1.55 -> 1.32 ms; r5/6 z=96: 0.98
 * -> 0.89 ms). All arithmetic is fp32.
 *
 * Training (one frame at a time per CTA): the forward pass runs all T
 * iterations and stores the posterior and the messages at the iteration
 * boundaries (checkpoints); the loss is the BCE mean over iterations, bits and
 * frames (positive LLR = bit 1: loss = softplus(sg * P), sg = +1 for bit 0,
 * -1 for bit 1). The backward pass walks the iterations in reverse: it
 * restores iteration t's inputs from the checkpoints, recomputes its forward
 * keeping every edge's L, and back-propagates through its layers in reverse.
 * Subgradients: sign() and the argmin choice are constant, d|x|/dx = sign(x),
 * relu'(0) = 0; edge e != i1 takes its magnitude from i1 (the first edge with
 * |L| == min1), edge i1 from i2 (the first other edge with |L| == min2).
 * An infinite minimum (known bits) counts as the largest finite number.
 * A CTA adds up the weight gradients of its frames; a second kernel adds the
 * CTAs' in a fixed order (deterministic) and applies Adam.
 */
#ifndef WLDPC_LMS_CUH
#define WLDPC_LMS_CUH

#include <cfloat>
#include <cstdint>
#include "codes.h"
#include "device_util.cuh"
#include "min_others.cuh"
#include "nms_decode.cuh"

namespace wldpc {

constexpr int kLmsMaxIter = 8;
constexpr int kLmsMaxBlocks = 96;

/* Weights per (iteration, non-zero block): blocks in row-major base-matrix
 * order, so block b of layer i has column layer_col(rate, i, e). */
struct LmsWeights {
    float a[kLmsMaxIter][kLmsMaxBlocks];
    float b[kLmsMaxIter][kLmsMaxBlocks];
};

struct LmsArgs {
    const float* llr;       /* frames x n, 16-byte aligned */
    int8_t* hard;           /* frames x n, 4-byte aligned */
    float* post;            /* frames x n or null */
    int32_t* status;        /* frames or null: iterations | synfail << 16 */
    unsigned* err;
    long long frames;
    int iters;              /* iteration cap */
    int wrows;              /* trained iterations T <= kLmsMaxIter; iteration t >= T uses row T-1 */
    unsigned wait_limit_us = kWaitLimitUs;   /* bound of the staging wait (the drain wait after a timeout is full) */
    float2 wab[kLmsMaxIter][kLmsMaxBlocks];   /* (a, b) per (iteration, block): one 8-byte load per edge */
};

/* Frames (or frame pairs) per CTA for the learned decoders: 32/gcd(z, 32)
 * of them make the CTA a whole number of warps; while that would exceed 384
 * threads (the register file must hold a few such CTAs at ~128 registers per
 * thread) or 100 KB of posteriors, halve it (the last warp is then partial). */
constexpr int lms_group(int z, int frame_bytes)
{
    int g = 32 / gcd_c(z, 32);
    while (g > 1 && (g * z > 384 || g * frame_bytes > 100 * 1024)) g /= 2;
    return g;
}

template <int R, int Z>
struct LmsShape {
    static constexpr int MB = kMb[R];
    static constexpr int NBLK = num_blocks(R);
    static constexpr int N = kNB * Z;
    static constexpr int E = NBLK * Z;
    static constexpr int G = lms_group(Z, N * 4);   /* frames per CTA */
    static constexpr int THREADS = G * Z;
    static constexpr int SMEM = G * N * 4;
};

/* ------------------------------------------------------------ inference */

/* Edge addressing of the fp32 decoder: the index col*z + (r + s) mod z
 * (edge_var_c) where that measured faster on a B200 (by 1-18%; all 114 codes
 * timed, outputs identical), else a pointer chosen by one compare and select
 * (edge_ptr), which was up to 8% faster on the others. */
constexpr bool lms_index_addressing(int R, int Z)
{
    switch (R) {
    case 0: return Z == 68;
    case 1: return Z == 40 || Z == 96;
    case 2: return Z == 80;
    case 3: return Z == 64 || Z == 96;
    case 4: return Z == 64 || Z == 96;
    default: return Z == 80 || Z == 96;
    }
}

/* Codes whose schedule came out slower than with two tracked minima (4 to 15%
 * for batches of 8 to 400 frames; all 114 timed), and what the compiler does
 * better with there: the minima in two-input form (to the tracked form's time
 * 0.94-1.00, rate 3/4B z = 32 0.73-0.79), or the layer's weights loaded ahead of
 * the minima (0.73-0.92). Elsewhere the one or the other is slower by up to 20%. */
constexpr bool lms_plain_minima(int R, int Z)
{
    return (R == 0 && Z == 28) || (R == 3 && Z == 32) || (R == 4 && (Z == 32 || Z == 40));
}
constexpr bool lms_early_weights(int R, int Z) { return Z == 64 && (R == 0 || R == 3 || R == 4); }

template <int R, int Z, int I, int E>
__device__ __forceinline__ float* lms_edge(float* P, float* Pr, float* Prz, int r)
{
    if constexpr (lms_index_addressing(R, Z))
        return P + edge_var_c<R, Z, I, E>(r);
    else
        return edge_ptr<R, Z, I, E>(Pr, Prz, r);
}

template <int R, int Z>
__global__ void __launch_bounds__(LmsShape<R, Z>::THREADS)
lms_decode_kernel(const __grid_constant__ LmsArgs a)
{
    using S = LmsShape<R, Z>;
    constexpr int MB = S::MB, N = S::N, G = S::G;
    extern __shared__ __align__(128) float smem_lms[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ unsigned s_fail[2], s_last[2], s_half[2];

    const int tid = threadIdx.x;
    const int g = G == 1 ? 0 : tid / Z;
    const int r = tid - g * Z;
    const long long f0 = (long long)blockIdx.x * G;
    const long long left = a.frames - f0;
    const int nf = left < G ? (int)left : G;
    float* P = smem_lms + g * N;                 /* posteriors of frame g */
    float* const Pr = P + r;                     /* lms_edge bases */
    float* const Prz = Pr - Z;

    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        s_fail[0] = 0;
        s_fail[1] = 0;
        s_last[0] = 0;
        s_last[1] = 0;
        s_half[0] = 0;
        s_half[1] = 0;
        const uint32_t bytes = (uint32_t)(nf * N * 4);
        mbar_arrive_expect_tx(&bar, bytes);
        bulk_g2s(smem_lms, a.llr + f0 * N, bytes, &bar);
    }
    __syncthreads();
    const bool ok = mbar_wait_bounded(&bar, 0, a.wait_limit_us);
    if (__syncthreads_or(!ok)) {
        if (tid == 0) {
            atomicOr(a.err, kErrWaitTimeout);
            mbar_wait_bounded(&bar, 0, kWaitLimitUs);   /* let an in-flight copy land before exit */
        }
        return;
    }

    /* syndrome of the thread's rows in layers FIRST .. END-1: 1 if any fails */
    auto rows_fail = [&](auto FIRST, auto END) -> unsigned {
        unsigned fail = 0;
        static_for<decltype(END)::value - decltype(FIRST)::value>([&](auto I_) {
            using I = std::integral_constant<int, decltype(FIRST)::value + decltype(I_)::value>;
            constexpr int d = layer_degree(R, I::value);
            bool odd = (d & 1) != 0;   /* parity of the hard bits: d minus the negatives */
            static_for<d>([&](auto E_) {
                odd = odd != (*lms_edge<R, Z, I::value, E_>(P, Pr, Prz, r) < 0.0f);
            });
            fail |= odd ? 1u : 0u;
        });
        return fail;
    };
    /* per-frame OR over the CTA (bit g: frame g); one barrier */
    auto frame_fail = [&](unsigned fail, unsigned* slot) -> unsigned {
        if constexpr (G == 1) {
            return __syncthreads_or((int)fail) ? 1u : 0u;
        } else {
            if (fail) atomicOr(slot, 1u << g);
            __syncthreads();
            return *slot;
        }
    };

    /* this thread's check-to-variable messages, one per block (its row of every
     * layer), in registers: every index is a compile-time constant */
    float Mr[S::NBLK];
#pragma unroll
    for (int q = 0; q < S::NBLK; q++) Mr[q] = 0.0f;

    /* initial syndrome (reference lib/ldpc_decoder.cc:127-139): layer 0's
     * rows first; only frames that pass there check the other layers */
    using L0 = std::integral_constant<int, 0>;
    using L1 = std::integral_constant<int, 1>;
    using LM = std::integral_constant<int, MB - 1>;
    using LH = std::integral_constant<int, (MB - 1) / 2>;
    using LE = std::integral_constant<int, MB>;
    const bool live = g < nf;
    const unsigned lives = (1u << nf) - 1u;
    unsigned fmask = frame_fail(live ? rows_fail(L0{}, L1{}) : 0u, &s_last[0]);
    if (lives & ~fmask)
        fmask |= frame_fail(live && !((fmask >> g) & 1u) ? rows_fail(L1{}, LE{}) : 0u, &s_fail[0]);
    bool active = live && ((fmask >> g) & 1u);
    int iters = 0;

    for (int t = 0; t < a.iters && fmask != 0u; ++t) {
        const int slot = (t + 1) & 1;   /* read last two iterations ago, before many barriers */
        if constexpr (G > 1) {
            if (tid == 0) {
                s_fail[slot] = 0;
                s_last[slot] = 0;
                s_half[slot] = 0;
            }
        }
        /* parity of the last layer's row from the posteriors it writes: no
         * later layer changes them in this iteration, so they are final */
        bool last_odd = false;
        /* this iteration's (a, b) pairs: the same address in every thread */
        const float2* const wab = a.wab[t < a.wrows ? t : a.wrows - 1];
        static_for<MB>([&](auto I) {
            constexpr int d = layer_degree(R, I);
            constexpr int b0 = block_index(R, I, 0);
            constexpr bool LAST = decltype(I)::value == MB - 1;
            if (active) {
                float L[d], A[d], mu[d];
                uint32_t sgn = 0;
                static_for<d>([&](auto E_) {
                    constexpr int e = decltype(E_)::value;
                    const float x = *lms_edge<R, Z, I, e>(P, Pr, Prz, r);
                    const float l = __fsub_rn(x, Mr[b0 + e]);
                    L[e] = l;
                    A[e] = fabsf(l);
                    sgn ^= __float_as_uint(l);   /* bit 31: parity of the negative L */
                });
                constexpr bool EARLY = lms_early_weights(R, Z);
                float2 w[d];
                if constexpr (EARLY) static_for<d>([&](auto E_) { w[E_] = wab[b0 + E_]; });
                min_others<typename std::conditional<lms_plain_minima(R, Z), MinF32Plain, MinF32>::type, d>(A, mu);
                /* positive LLR = bit 1: the extrinsic sign flips on odd-degree rows */
                const uint32_t fb = (sgn ^ ((uint32_t)(d & 1) << 31)) & 0x80000000u;
                const uint32_t fbo = fb | 0x3f800000u;   /* with sign(L_e): +-1.0 */
                static_for<d>([&](auto E_) {
                    constexpr int e = decltype(E_)::value;
                    const float l = L[e];
                    if constexpr (!EARLY) w[e] = wab[b0 + e];
                    const float2 ab = w[e];
                    const float mag = fmaxf(__fmaf_rn(ab.x, mu[e], -ab.y), 0.0f);
                    const float msg = __fmul_rn(mag, __uint_as_float((__float_as_uint(l) & 0x80000000u) ^ fbo));
                    Mr[b0 + e] = msg;
                    const float pn = __fadd_rn(l, msg);
                    *lms_edge<R, Z, I, e>(P, Pr, Prz, r) = pn;
                    if constexpr (LAST) last_odd = last_odd != (pn < 0.0f);
                });
                if constexpr (LAST) last_odd = last_odd != ((d & 1) != 0);
            }
            if constexpr (!LAST) __syncthreads();
        });
        /* stopping rule (zero syndrome over every row): a frame with a failing
         * row in the last layer fails; the other active frames check the
         * remaining layers in two halves, with a vote after each (a frame that
         * fails in the first half skips the second). The first vote is the last
         * layer's barrier. */
        const unsigned lmask = frame_fail(active && last_odd ? 1u : 0u, &s_last[slot]);
        unsigned fm = lmask;
        if (fmask & ~fm)
            fm |= frame_fail(active && !((fm >> g) & 1u) ? rows_fail(L0{}, LH{}) : 0u, &s_fail[slot]);
        if (fmask & ~fm)
            fm |= frame_fail(active && !((fm >> g) & 1u) ? rows_fail(LH{}, LM{}) : 0u, &s_half[slot]);
        fmask = fm;
        if (active) {
            iters = t + 1;
            active = (fmask >> g) & 1u;
        }
    }

    const int total = nf * N;
    int8_t* hard = a.hard + f0 * N;
    for (int v = tid * 4; v < total; v += S::THREADS * 4) {
        const float4 p = *reinterpret_cast<const float4*>(smem_lms + v);
        const uint32_t wv = (p.x >= 0.0f ? 1u : 0u) | (p.y >= 0.0f ? 1u << 8 : 0u) |
                            (p.z >= 0.0f ? 1u << 16 : 0u) | (p.w >= 0.0f ? 1u << 24 : 0u);
        *reinterpret_cast<uint32_t*>(hard + v) = wv;
        if (a.post) *reinterpret_cast<float4*>(a.post + f0 * N + v) = p;
    }
    if (a.status && live && r == 0) a.status[f0 + g] = iters | ((active ? 1 : 0) << 16);
}

/* ------------------------------------------------------------- training */

struct LmsTrainArgs {
    const float* llr;       /* frames x n */
    const uint8_t* cw;      /* frames x n transmitted bits (0/1) */
    float* ck_post;         /* per CTA T x n: posteriors after iteration t */
    float* ck_msg;          /* per CTA T x E: messages after iteration t */
    float* gpart;           /* per CTA 2 x T x NBLK: weight gradient over its frames */
    double* loss_part;      /* per CTA: loss over its frames */
    const float* wa;        /* T x NBLK scales (device) */
    const float* wb;        /* T x NBLK offsets (device) */
    long long frames;
    int iters;              /* T */
    float inv_norm;         /* 1 / (T * n * frames) */
};

__device__ __forceinline__ float softplus_f(float x) { return x > 0.0f ? x + log1pf(__expf(-x)) : log1pf(__expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + __expf(-x)); }

/* One frame at a time per CTA of whole warps. Lanes past z idle along on another
 * lane's row: what they read, maybe while it is written, reaches no sum. */
template <int R, int Z>
struct LmsTrainShape {
    static constexpr int MB = kMb[R];
    static constexpr int NBLK = num_blocks(R);
    static constexpr int N = kNB * Z;
    static constexpr int E = NBLK * Z;
    static constexpr int W = (Z + 31) / 32;
    static constexpr int THREADS = 32 * W;
    /* P, gP, gM, the CTA's weight gradient, the iteration's (a, b) pairs and
     * its gradient per warp */
    static constexpr int SMEM = (2 * N + E + 2 * kLmsMaxIter * NBLK + 2 * NBLK + W * 2 * NBLK) * 4;
    /* 12 warps on an SM, as many as the shared memory allows at z = 96: up to
     * 168 registers, one per message and the layer in work */
    static constexpr int MIN_CTAS = 12 / W;
};

/* one iteration of the thread's rows on P; m: the messages, replaced by the
 * new ones, or (RECORD) by the L they were turned into */
template <int R, int Z, bool RECORD, int NBLK>
__device__ __forceinline__ void lms_train_iteration(float* Pr, float* Prz, int r, bool owner, const float2* wab,
                                                    float (&m)[NBLK])
{
    static_for<kMb[R]>([&](auto I) {
        constexpr int d = layer_degree(R, I);
        constexpr int b0 = block_index(R, I, 0);
        float L[d], A[d], mu[d];
        uint32_t sgn = 0;
        static_for<d>([&](auto E_) {
            constexpr int e = decltype(E_)::value;
            const float l = __fsub_rn(*edge_ptr<R, Z, I, e>(Pr, Prz, r), m[b0 + e]);
            L[e] = l;
            A[e] = fabsf(l);
            sgn ^= __float_as_uint(l);
        });
        min_others<MinF32, d>(A, mu);
        const uint32_t fbo = ((sgn ^ ((uint32_t)(d & 1) << 31)) & 0x80000000u) | 0x3f800000u;
        static_for<d>([&](auto E_) {
            constexpr int e = decltype(E_)::value;
            const float l = L[e];
            const float2 ab = wab[b0 + e];
            const float mag = fmaxf(__fmaf_rn(ab.x, mu[e], -ab.y), 0.0f);
            const float msg = __fmul_rn(mag, __uint_as_float((__float_as_uint(l) & 0x80000000u) ^ fbo));
            m[b0 + e] = RECORD ? l : msg;
            if (owner) *edge_ptr<R, Z, I, e>(Pr, Prz, r) = __fadd_rn(l, msg);
        });
        __syncthreads();
    });
}

/* K (a power of two, up to 32) sums over the warp at once: each step halves
 * the values a lane holds and doubles the lanes they cover, K - 1 shuffles
 * instead of 5 K. Lane l ends with value l / (32 / K). */
template <int K>
__device__ __forceinline__ float warp_sums(float (&v)[K], int lane)
{
    int bit = 16;
#pragma unroll
    for (int s = K / 2; s >= 1; s /= 2) {
        const bool up = (lane & bit) != 0;
#pragma unroll
        for (int i = 0; i < s; i++) {
            const float send = up ? v[i] : v[i + s], keep = up ? v[i + s] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
        bit >>= 1;
    }
#pragma unroll
    for (int o = 16 / K; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

/* Loss and weight gradient. CTA c takes frames c, c + gridDim.x, ... What
 * bounded the first form (one frame per launch of z threads, messages, their
 * L and their gradient in shared memory: 6 warps on an SM; ten shuffles and
 * two atomic additions per edge, per-thread atomics where z is no multiple of
 * 32) was latency: 950 cycles per warp, edge and iteration. Here a thread's
 * messages are registers, which the recomputed forward turns into the L that
 * the backward pass reads, only the message gradients stay in shared memory,
 * the rows' weight gradients are summed over a warp 16 or 32 at a time, and a
 * CTA adds its frames' gradients up (fixed order) instead of writing each:
 * a step of 4096 r1/2 z=96 frames 6.07 -> 1.83 ms.
 * The last iteration is run once: its L are recorded on the way forward. */
template <int R, int Z>
__global__ void __launch_bounds__(LmsTrainShape<R, Z>::THREADS, LmsTrainShape<R, Z>::MIN_CTAS)
lms_train_kernel(const __grid_constant__ LmsTrainArgs a)
{
    using S = LmsTrainShape<R, Z>;
    constexpr int MB = S::MB, N = S::N, E = S::E, NBLK = S::NBLK, TH = S::THREADS, W = S::W;
    extern __shared__ __align__(128) float smem_tr[];
    float* const P = smem_tr;
    float* const gP = P + N;
    float* const gM = gP + N;
    float* const gW = gM + E;                                       /* [2][T][NBLK] */
    float2* const wab = reinterpret_cast<float2*>(gW + 2 * kLmsMaxIter * NBLK);
    float* const part = reinterpret_cast<float*>(wab + NBLK);       /* [warp][2][NBLK] */
    __shared__ double s_loss[W];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool owner = Z % 32 == 0 || tid < Z;
    const int r = owner ? tid : tid % Z;
    const int T = a.iters;
    float* const Pr = P + r;
    float* const Prz = Pr - Z;
    float* const Gr = gP + r;
    float* const Grz = Gr - Z;
    float* const ckp = a.ck_post + blockIdx.x * (long long)T * N;
    float* const ckm = a.ck_msg + blockIdx.x * (long long)T * E;
    for (int q = tid; q < 2 * T * NBLK; q += TH) gW[q] = 0.0f;
    double loss = 0.0;

    for (long long f = blockIdx.x; f < a.frames; f += gridDim.x) {
        const float* const llr = a.llr + f * N;
        const uint8_t* const cw = a.cw + f * N;
        float m[NBLK];
        __syncthreads();   /* the frame before is done with P, gP and gM */
        for (int q = tid; q < N; q += TH) {
            P[q] = llr[q];
            gP[q] = 0.0f;
        }
        for (int q = tid; q < E; q += TH) gM[q] = 0.0f;
#pragma unroll
        for (int q = 0; q < NBLK; q++) m[q] = 0.0f;
        auto weights = [&](int t) {   /* between two barriers */
            for (int q = tid; q < NBLK; q += TH) {
                const float2 ab = make_float2(a.wa[t * NBLK + q], a.wb[t * NBLK + q]);
                /* a scale of 0 makes no message of an infinite minimum, whatever the offset: a
                 * hair below 0, which no finite minimum feels, says so of the largest one too */
                wab[q] = make_float2(ab.x == 0.0f ? -1e-30f : ab.x, ab.y);
            }
        };

        /* forward, keeping what each iteration ends with except the last two:
         * the last but one leads straight into the last */
        for (int t = 0; t < T - 1; t++) {
            weights(t);
            __syncthreads();
            lms_train_iteration<R, Z, false>(Pr, Prz, r, owner, wab, m);
            if (t < T - 2) {
                for (int q = tid; q < N; q += TH) ckp[(long long)t * N + q] = P[q];
                if (owner) {
#pragma unroll
                    for (int q = 0; q < NBLK; q++) ckm[(long long)t * E + q * Z + r] = m[q];
                }
            }
        }

        /* backward; P and m hold iteration t's inputs, from the checkpoint
         * after iteration t - 1 except for the last */
        float floss = 0.0f;
        for (int t = T - 1; t >= 0; t--) {
            if (t < T - 1) {
                const float* const pin = t == 0 ? llr : ckp + (long long)(t - 1) * N;
                for (int q = tid; q < N; q += TH) P[q] = pin[q];
#pragma unroll
                for (int q = 0; q < NBLK; q++) m[q] = t == 0 ? 0.0f : ckm[(long long)(t - 1) * E + q * Z + r];
            }
            weights(t);
            __syncthreads();
            lms_train_iteration<R, Z, true>(Pr, Prz, r, owner, wab, m);   /* m: L from here */
            /* loss of iteration t and its gradient */
            for (int q = tid; q < N; q += TH) {
                const float p = P[q];
                const float sg = cw[q] ? -1.0f : 1.0f;
                floss += softplus_f(sg * p);
                gP[q] += sg * sigmoid_f(sg * p) * a.inv_norm;
            }
            __syncthreads();
            static_for<MB>([&](auto IR) {
                constexpr int I = MB - 1 - decltype(IR)::value;
                constexpr int d = layer_degree(R, I);
                constexpr int b0 = block_index(R, I, 0);
                float L[d], gL[d];
                uint32_t negpar = (uint32_t)(d & 1) << 31;   /* odd-degree rows flip the extrinsic sign */
                static_for<d>([&](auto E_) {
                    constexpr int e = decltype(E_)::value;
                    L[e] = m[b0 + e];
                    gL[e] = *edge_ptr<R, Z, I, e>(Gr, Grz, r);
                    negpar ^= __float_as_uint(L[e]);
                });
                float m1, m2;
                two_min_abs<0, d>(L, m1, m2);
                /* i1: the first edge with |L| == m1, i2: the first other one with |L| == m2 */
                int i1 = 0, i2 = 0;
                static_for<d>([&](auto E_) {
                    constexpr int e = d - 1 - decltype(E_)::value;
                    i1 = fabsf(L[e]) == m1 ? e : i1;
                });
                static_for<d>([&](auto E_) {
                    constexpr int e = d - 1 - decltype(E_)::value;
                    i2 = fabsf(L[e]) == m2 && e != i1 ? e : i2;
                });
                /* an infinite minimum (known bits) as the largest finite one: times zero it
                 * is NaN, but what relu cut off, and an idle lane, adds nothing. (Cleared
                 * edge by edge instead, by selects or behind a branch that few rows take:
                 * 4% slower at r1/2 z=96, 4-20% at the other rates.) */
                m1 = fminf(m1, FLT_MAX);
                m2 = fminf(m2, FLT_MAX);
                constexpr int K = 2 * d <= 16 ? 16 : 32;
                constexpr int H = (2 * d + K - 1) / K;    /* groups of K sums (2 for d = 20) */
                float v[H][K];
#pragma unroll
                for (int h = 0; h < H; h++)
#pragma unroll
                    for (int q = 0; q < K; q++) v[h][q] = 0.0f;
                float g_to_i1 = 0.0f, g_to_i2 = 0.0f;
                static_for<d>([&](auto E_) {
                    constexpr int e = decltype(E_)::value;
                    const float mu = (fabsf(L[e]) == m1) ? m2 : m1;
                    const float2 ab = wab[b0 + e];
                    const float pre = __fmaf_rn(ab.x, mu, -ab.y);
                    const float G = owner ? gL[e] + gM[(b0 + e) * Z + r] : 0.0f;
                    /* gradient of the magnitude, zero where relu cut it off */
                    const float gs = pre > 0.0f ? __uint_as_float(__float_as_uint(G) ^ ((negpar ^ __float_as_uint(L[e])) &
                                                                                       0x80000000u))
                                                : 0.0f;
                    v[e / K][e % K] = gs * mu;
                    v[(d + e) / K][(d + e) % K] = -gs;
                    const float gmu = gs * ab.x;
                    if (e == i1) g_to_i2 += gmu;
                    else g_to_i1 += gmu;
                });
                static_for<d>([&](auto E_) {
                    constexpr int e = decltype(E_)::value;
                    const float sgn_l = __uint_as_float((__float_as_uint(L[e]) & 0x80000000u) | 0x3f800000u);
                    float g = gL[e];
                    if (e == i1) g += g_to_i1 * sgn_l;
                    if (e == i2) g += g_to_i2 * sgn_l;
                    if (owner) {
                        *edge_ptr<R, Z, I, e>(Gr, Grz, r) = g;
                        gM[(b0 + e) * Z + r] = -g;
                    }
                });
#pragma unroll
                for (int h = 0; h < H; h++) {
                    const float sum = warp_sums<K>(v[h], lane);
                    const int k = h * K + lane / (32 / K);
                    if (lane % (32 / K) == 0 && k < 2 * d)
                        part[warp * 2 * NBLK + (k < d ? b0 + k : NBLK + b0 + k - d)] = sum;
                }
                __syncthreads();
            });
            for (int q = tid; q < 2 * NBLK; q += TH) {
                float g = part[q];
                for (int w = 1; w < W; w++) g += part[w * 2 * NBLK + q];
                gW[q < NBLK ? t * NBLK + q : (T + t) * NBLK + q - NBLK] += g;
            }
        }
        loss += (double)floss;
    }
    /* the CTA's loss and gradient */
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) s_loss[warp] = loss;
    __syncthreads();
    if (tid == 0) {
        double sum = 0.0;
        for (int w = 0; w < W; w++) sum += s_loss[w];
        a.loss_part[blockIdx.x] = sum * (double)a.inv_norm;
    }
    for (int q = tid; q < 2 * T * NBLK; q += TH) a.gpart[(long long)blockIdx.x * 2 * T * NBLK + q] = gW[q];
}

/* Column sums of the CTAs' gradients in a fixed order, then Adam; w holds a
 * then b, [T][NBLK] each. */
struct AdamArgs {
    const float* gpart;      /* rows x nw */
    const double* loss_part; /* rows */
    float* grad;             /* nw, written (the reduced gradient) */
    float* w;                /* nw parameters */
    float* m;                /* nw first moments */
    float* v;                /* nw second moments */
    float* loss_out;         /* one float: the batch loss, or null */
    int rows;                /* CTAs of the training launch, or 1 */
    int nw;
    int step;                /* 1-based Adam step */
    float lr, beta1, beta2, eps;
    int apply;               /* 0: only reduce the gradient */
};

}  // namespace wldpc

#endif
