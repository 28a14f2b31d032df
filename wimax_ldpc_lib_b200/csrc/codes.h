/*
 * WiMAX 802.16e QC-LDPC code description, shared by host and device code.
 *
 * kBase holds the standard's prototype circulant shifts p(i, j) at z0 = 96 for
 * the six code rates, in the reference's enum order (reference
 * include/enums.h:4-12); -1 is an all-zero block, rows past kMb[rate] are
 * padding. The reference ships the same matrices pre-expanded for all 19
 * expansion factors (reference lib/matrices/wimax_N_RATE.cc, selected in
 * reference lib/ldpc.cc:69-1206); they are expanded here by rule instead:
 *
 *   shift(p, z) = p              if p <= 0
 *               = p mod z        for rate 2/3A
 *               = floor(p*z/96)  otherwise        (also applied to D)
 *
 * Expanded check row r (0 <= r < z) of base row i connects variable
 * j*z + (r + shift) mod z for every block column j with p(i, j) >= 0; the
 * reference lists them in increasing j (reference lib/matrices/wimax_576_0_5.cc:8-10).
 *
 * Everything is constexpr so that kernels specialised on (rate, z) resolve
 * columns, shifts and degrees at compile time.
 */
#ifndef WLDPC_CODES_H
#define WLDPC_CODES_H

#ifdef __CUDACC__
#define WLDPC_HD __host__ __device__
#else
#define WLDPC_HD
#endif

namespace wldpc {

/* Host-buffer batch calls pipeline copy-in, decode and copy-out over
 * kHostStages streams in chunks; with three stages chunk k+2 is copied in while
 * chunk k is copied out, so both copy directions stay busy. A chunk is an
 * eighth of the batch, between 1024 and 8192 frames: the last chunk's decode
 * and copy out overlap with nothing (16,384 frames of rate 1/2 z = 96, hard
 * bits back: 3.43 ms in chunks of 8192, 3.03 in chunks of 2048; the copy in
 * alone takes 2.96), while large batches want long copies (262,144 frames,
 * posterior back: 64.3 ms with 8192-frame chunks, 65.8-66.2 with 16384, 64.7
 * with 4096; a fourth stage did not help). */
constexpr int kHostStages = 3;
constexpr unsigned long host_chunk(unsigned long frames)
{
    const unsigned long eighth = (frames + 7) / 8;
    const unsigned long chunk = eighth < 1024 ? 1024 : eighth > 8192 ? 8192 : eighth;
    return chunk < frames ? chunk : frames;
}



constexpr int kNB = 24;        /* base block columns */
constexpr int kMaxMb = 12;     /* base rows of rate 1/2 */
constexpr int kRates = 6;
constexpr int kZMin = 24, kZMax = 96, kZStep = 4, kNumZ = 19;
constexpr int kMaxDeg = 20;    /* rate 5/6 */
constexpr int kMaxN = kNB * kZMax;

enum Rate { HALFRATE = 0, TWOTHIRDSA = 1, TWOTHIRDSB = 2, THREEQUARTERSA = 3,
            THREEQUARTERSB = 4, FIVESIXTHS = 5 };

constexpr int kMb[kRates] = {12, 8, 8, 6, 6, 4};
constexpr int kD96[kRates] = {7, 1, 95, 48, 80, 80};
constexpr int kX[kRates] = {5, 4, 6, 3, 2, 1};

constexpr signed char kBase[kRates][kMaxMb][kNB] = {
    /* rate 1/2: mb=12, D(96)=7, X=5 */
    {
        { -1, 94, 73, -1, -1, -1, -1, -1, 55, 83, -1, -1,  7,  0, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, 27, -1, -1, -1, 22, 79,  9, -1, -1, -1, 12, -1,  0,  0, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, 24, 22, 81, -1, 33, -1, -1, -1,  0, -1, -1,  0,  0, -1, -1, -1, -1, -1, -1, -1, -1},
        { 61, -1, 47, -1, -1, -1, -1, -1, 65, 25, -1, -1, -1, -1, -1,  0,  0, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, 39, -1, -1, -1, 84, -1, -1, 41, 72, -1, -1, -1, -1, -1,  0,  0, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, 46, 40, -1, 82, -1, -1, -1, 79,  0, -1, -1, -1, -1,  0,  0, -1, -1, -1, -1, -1},
        { -1, -1, 95, 53, -1, -1, -1, -1, -1, 14, 18, -1, -1, -1, -1, -1, -1, -1,  0,  0, -1, -1, -1, -1},
        { -1, 11, 73, -1, -1, -1,  2, -1, -1, 47, -1, -1, -1, -1, -1, -1, -1, -1, -1,  0,  0, -1, -1, -1},
        { 12, -1, -1, -1, 83, 24, -1, 43, -1, -1, -1, 51, -1, -1, -1, -1, -1, -1, -1, -1,  0,  0, -1, -1},
        { -1, -1, -1, -1, -1, 94, -1, 59, -1, -1, 70, 72, -1, -1, -1, -1, -1, -1, -1, -1, -1,  0,  0, -1},
        { -1, -1,  7, 65, -1, -1, -1, -1, 39, 49, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1,  0,  0},
        { 43, -1, -1, -1, -1, 66, -1, 41, -1, -1, -1, 26,  7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1,  0},
    },
    /* rate 2/3A: mb=8, D(96)=1, X=4 */
    {
        {  3,  0, -1, -1,  2,  0, -1,  3,  7, -1,  1,  1, -1, -1, -1, -1,  1,  0, -1, -1, -1, -1, -1, -1},
        { -1, -1,  1, -1, 36, -1, -1, 34, 10, -1, -1, 18,  2, -1,  3,  0, -1,  0,  0, -1, -1, -1, -1, -1},
        { -1, -1, 12,  2, -1, 15, -1, 40, -1,  3, -1, 15, -1,  2, 13, -1, -1, -1,  0,  0, -1, -1, -1, -1},
        { -1, -1, 19, 24, -1,  3,  0, -1,  6, -1, 17, -1, -1, -1,  8, 39, -1, -1, -1,  0,  0, -1, -1, -1},
        { 20, -1,  6, -1, -1, 10, 29, -1, -1, 28, -1, 14, -1, 38, -1, -1,  0, -1, -1, -1,  0,  0, -1, -1},
        { -1, -1, 10, -1, 28, 20, -1, -1,  8, -1, 36, -1,  9, -1, 21, 45, -1, -1, -1, -1, -1,  0,  0, -1},
        { 35, 25, -1, 37, -1, 21, -1, -1,  5, -1, -1,  0, -1,  4, 20, -1, -1, -1, -1, -1, -1, -1,  0,  0},
        { -1,  6,  6, -1, -1, -1,  4, -1, 14, 30, -1,  3, 36, -1, 14, -1,  1, -1, -1, -1, -1, -1, -1,  0},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    },
    /* rate 2/3B: mb=8, D(96)=95, X=6 */
    {
        {  2, -1, 19, -1, 47, -1, 48, -1, 36, -1, 82, -1, 47, -1, 15, -1, 95,  0, -1, -1, -1, -1, -1, -1},
        { -1, 69, -1, 88, -1, 33, -1,  3, -1, 16, -1, 37, -1, 40, -1, 48, -1,  0,  0, -1, -1, -1, -1, -1},
        { 10, -1, 86, -1, 62, -1, 28, -1, 85, -1, 16, -1, 34, -1, 73, -1, -1, -1,  0,  0, -1, -1, -1, -1},
        { -1, 28, -1, 32, -1, 81, -1, 27, -1, 88, -1,  5, -1, 56, -1, 37, -1, -1, -1,  0,  0, -1, -1, -1},
        { 23, -1, 29, -1, 15, -1, 30, -1, 66, -1, 24, -1, 50, -1, 62, -1, -1, -1, -1, -1,  0,  0, -1, -1},
        { -1, 30, -1, 65, -1, 54, -1, 14, -1,  0, -1, 30, -1, 74, -1,  0, -1, -1, -1, -1, -1,  0,  0, -1},
        { 32, -1,  0, -1, 15, -1, 56, -1, 85, -1,  5, -1,  6, -1, 52, -1,  0, -1, -1, -1, -1, -1,  0,  0},
        { -1,  0, -1, 47, -1, 13, -1, 61, -1, 84, -1, 55, -1, 78, -1, 41, 95, -1, -1, -1, -1, -1, -1,  0},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    },
    /* rate 3/4A: mb=6, D(96)=48, X=3 */
    {
        {  6, 38,  3, 93, -1, -1, -1, 30, 70, -1, 86, -1, 37, 38,  4, 11, -1, 46, 48,  0, -1, -1, -1, -1},
        { 62, 94, 19, 84, -1, 92, 78, -1, 15, -1, -1, 92, -1, 45, 24, 32, 30, -1, -1,  0,  0, -1, -1, -1},
        { 71, -1, 55, -1, 12, 66, 45, 79, -1, 78, -1, -1, 10, -1, 22, 55, 70, 82, -1, -1,  0,  0, -1, -1},
        { 38, 61, -1, 66,  9, 73, 47, 64, -1, 39, 61, 43, -1, -1, -1, -1, 95, 32,  0, -1, -1,  0,  0, -1},
        { -1, -1, -1, -1, 32, 52, 55, 80, 95, 22,  6, 51, 24, 90, 44, 20, -1, -1, -1, -1, -1, -1,  0,  0},
        { -1, 63, 31, 88, 20, -1, -1, -1,  6, 40, 56, 16, 71, 53, -1, -1, 27, 26, 48, -1, -1, -1, -1,  0},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    },
    /* rate 3/4B: mb=6, D(96)=80, X=2 */
    {
        { -1, 81, -1, 28, -1, -1, 14, 25, 17, -1, -1, 85, 29, 52, 78, 95, 22, 92,  0,  0, -1, -1, -1, -1},
        { 42, -1, 14, 68, 32, -1, -1, -1, -1, 70, 43, 11, 36, 40, 33, 57, 38, 24, -1,  0,  0, -1, -1, -1},
        { -1, -1, 20, -1, -1, 63, 39, -1, 70, 67, -1, 38,  4, 72, 47, 29, 60,  5, 80, -1,  0,  0, -1, -1},
        { 64,  2, -1, -1, 63, -1, -1,  3, 51, -1, 81, 15, 94,  9, 85, 36, 14, 19, -1, -1, -1,  0,  0, -1},
        { -1, 53, 60, 80, -1, 26, 75, -1, -1, -1, -1, 86, 77,  1,  3, 72, 60, 25, -1, -1, -1, -1,  0,  0},
        { 77, -1, -1, -1, 15, 28, -1, 35, -1, 72, 30, 68, 85, 84, 26, 64, 11, 89,  0, -1, -1, -1, -1,  0},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    },
    /* rate 5/6: mb=4, D(96)=80, X=1 */
    {
        {  1, 25, 55, -1, 47,  4, -1, 91, 84,  8, 86, 52, 82, 33,  5,  0, 36, 20,  4, 77, 80,  0, -1, -1},
        { -1,  6, -1, 36, 40, 47, 12, 79, 47, -1, 41, 21, 12, 71, 14, 72,  0, 44, 49,  0,  0,  0,  0, -1},
        { 51, 81, 83,  4, 67, -1, 21, -1, 31, 24, 91, 61, 81,  9, 86, 78, 60, 88, 67, 15, -1, -1,  0,  0},
        { 50, -1, 50, 15, -1, 36, 13, 10, 11, 20, 53, 90, 29, 92, 57, 30, 84, 92, 11, 66, 80, -1, -1,  0},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        { -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    },
};

constexpr bool valid_z(int z) { return z >= kZMin && z <= kZMax && (z % kZStep) == 0; }
constexpr bool valid_rate(int r) { return r >= 0 && r < kRates; }
constexpr int z_index(int z) { return (z - kZMin) / kZStep; }

constexpr int shift_rule(int rate, int p, int z)
{
    return p <= 0 ? p : (rate == TWOTHIRDSA ? p % z : (p * z) / 96);
}
constexpr int mb_of(int rate) { return kMb[rate]; }
constexpr int kb_of(int rate) { return kNB - kMb[rate]; }
constexpr int n_of(int z) { return kNB * z; }
constexpr int k_of(int rate, int z) { return (kNB - kMb[rate]) * z; }
constexpr int D_of(int rate, int z) { return shift_rule(rate, kD96[rate], z); }

/* number of non-zero blocks in base row i */
constexpr int layer_degree(int rate, int i)
{
    int d = 0;
    for (int j = 0; j < kNB; j++) d += kBase[rate][i][j] >= 0 ? 1 : 0;
    return d;
}
/* block column of the e-th non-zero block of base row i */
constexpr int layer_col(int rate, int i, int e)
{
    for (int j = 0; j < kNB; j++)
        if (kBase[rate][i][j] >= 0) {
            if (e == 0) return j;
            --e;
        }
    return -1;
}
constexpr int layer_shift(int rate, int z, int i, int e)
{
    return shift_rule(rate, kBase[rate][i][layer_col(rate, i, e)], z);
}
/* number of info blocks (column < kb) in base row i */
constexpr int layer_info_degree(int rate, int i)
{
    int d = 0;
    for (int j = 0; j < kb_of(rate); j++) d += kBase[rate][i][j] >= 0 ? 1 : 0;
    return d;
}
constexpr int num_blocks(int rate)
{
    int b = 0;
    for (int i = 0; i < kMb[rate]; i++) b += layer_degree(rate, i);
    return b;
}
constexpr int max_degree(int rate)
{
    int d = 0;
    for (int i = 0; i < kMb[rate]; i++) d = layer_degree(rate, i) > d ? layer_degree(rate, i) : d;
    return d;
}

}  // namespace wldpc

#endif
