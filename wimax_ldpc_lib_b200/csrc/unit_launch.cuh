/* Launching the persistent unit decoders (unit_decode.cuh). */
#ifndef WLDPC_UNIT_LAUNCH_CUH
#define WLDPC_UNIT_LAUNCH_CUH

#include <cuda_runtime.h>

namespace wldpc {

enum UnitKind : int { kUnitPlain = 0, kUnitLearned = 1, kUnitLearned16 = 2 };

/* The smallest batch that goes to the unit kernel, per decoder, rate and z
 * (24 to 96 in steps of 4). A persistent CTA holds 4 to 32 frames or pairs (8 at
 * r1/2 z = 96, 24 at z = 32), so a small batch leaves most of it idle while
 * each frame's layers take longer than in a CTA of its own; a large batch gains
 * by 16 to 24 warps per SM instead of 9 to 15 and by not waiting for a CTA's
 * slowest frame. All 114 codes were timed with both kernels at 64, 250, 600, 1200,
 * 2500, 5000 and 30,000 frames (outputs identical); a code's line is the first
 * of those sizes from which on the unit kernel was never more than 1% slower.
 * Digits: 1: 64 frames, 2: 600, 3: 2500, 4: 5000, 5: 20,000, 0: never.
 * At 30,000 frames the unit kernel took, where it is used, 0.64-0.99 of the
 * other's time for plain, 0.55-0.99 for learned fp32 and 0.47-0.99
 * for binary16; least where z is no multiple of 16. */
constexpr const char* kUnitMin[3][6] = {
    {
        "5153435111212141113",
        "5133535111014141113",
        "5155335111511141114",
        "5153030131014141113",
        "5155440131013131110",
        "5355510131314101115",
    },
    {
        "3151315111111151115",
        "4153510111013351113",
        "1113315311421331115",
        "1113530111112331215",
        "2111440111132231110",
        "1253415112031241110",
    },
    {
        "1153415111511151114",
        "1143335111533331113",
        "1154315331533343115",
        "3154440333011343314",
        "2153310131033331113",
        "3153315111431341114",
    },
};
constexpr long long unit_min_frames(UnitKind kind, int rate, int z)
{
    constexpr long long lines[6] = {-1, 64, 600, 2500, 5000, 20000};
    return lines[kUnitMin[kind][rate][(z - 24) / 4] - '0'];
}

template <typename Args>
struct UnitLaunch {
    void (*kernel)(const Args) = nullptr;   /* null: the code keeps its one-frame-per-CTA kernel */
    int threads = 0, smem = 0;
    int frames = 1;                         /* frames per ticket */
    long long min_frames = 0;
};

/* whether a batch goes to the unit kernel: it holds frame numbers in 32 bits */
template <typename Args>
inline bool unit_takes(const UnitLaunch<Args>& k, long long frames)
{
    return k.kernel && frames >= k.min_frames && frames <= 0x7ffffffeLL;
}

template <typename Args>
inline cudaError_t launch_unit(const UnitLaunch<Args>& k, const Args& a, cudaStream_t st)
{
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem);
    if (e != cudaSuccess) return e;
    const long long tickets = (a.frames + k.frames - 1) / k.frames;
    k.kernel<<<(unsigned)(tickets < sms ? tickets : sms), k.threads, k.smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace wldpc

#endif
