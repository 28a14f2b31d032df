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
 * slowest frame. All 114 codes were timed with both kernels at eleven sizes
 * from 64 to 30,000 frames, each at three Eb/N0, launches back to back (outputs
 * identical); from a code's line on, one of the six below, the unit kernel was
 * faster on the mean of the three, and at none of them more than 3.5% slower (two
 * runs differ by 2 to 4% at the small sizes). A change of either kernel wants
 * them timed again.
 * Digits: 1: 64 frames, 2: 400, 3: 1800, 4: 6000, 5: 15,000, 6: 30,000, 0:
 * never. At 30,000 frames the unit kernel took, where it is used, 0.64-0.99 of
 * the other's time for plain, 0.55-1.00 for learned fp32 and 0.47-0.99 for
 * binary16; least where z is no multiple of 16. */
constexpr const char* kUnitMin[3][6] = {
    {
        "6164436131413141114",
        "5154535111033141114",
        "5164535111514141114",
        "6165040141014341314",
        "6155540131034341110",
        "6365610131445301115",
    },
    {
        "5103516113031161115",
        "5163530322033361135",
        "5113536311533343315",
        "5123430111033443335",
        "4153440112033343330",
        "5144556131033463110",
    },
    {
        "2144445131533351114",
        "1154445333634331114",
        "4254445232633333335",
        "6365450433013344445",
        "6254440333033433316",
        "5254346221543441115",
    },
};
constexpr long long unit_min_frames(UnitKind kind, int rate, int z)
{
    constexpr long long lines[7] = {-1, 64, 400, 1800, 6000, 15000, 30000};
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
