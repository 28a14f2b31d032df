/*
 * How host-buffer batches are cut: copy-in, decode and copy-out of their chunks
 * are pipelined over kHostStages streams; with three stages chunk k+2 is copied
 * in while chunk k is copied out, so both copy directions stay busy. (A fourth
 * stage did not help.)
 */
#ifndef WLDPC_HOST_BATCH_H
#define WLDPC_HOST_BATCH_H

#include <cuda_runtime_api.h>

namespace wldpc {

constexpr int kHostStages = 3;

/* Frames of n values per chunk.
 * Pinned buffers: an eighth of the batch, between 1024 and 8192 frames: the
 * last chunk's decode and copy out overlap with nothing (16,384 frames of rate
 * 1/2 z = 96, hard bits back: 3.43 ms in chunks of 8192, 3.03 in chunks of 2048;
 * the copy in alone takes 2.96), while large batches want long copies (262,144
 * frames, posterior back: 64.3 ms with 8192-frame chunks, 65.8-66.2 with 16384,
 * 64.7 with 4096). A chunk costs some 12 us by itself, so short frames take
 * fewer: at least 7 MB where only hard bits come back (12,000 rate-1/2 z = 24
 * frames, binary16: 594 us with 8192-frame chunks, 628 in eighths, 600 so; 8192
 * frames 490, 480 and 440), and one chunk below 6 MB (1500 frames, posterior
 * back: 3% slower in two).
 * Pageable buffers: chunks of 8192, since their copies wait for one another
 * and for the decode, and nothing overlaps whatever the chunk; shorter ones only
 * add launches and fill the GPU less (rate 1/2 z = 24, hard bits back: 8192
 * frames 1.45 ms whole, 2.0 in eighths; z = 96: 8.3 and 9.0). */
constexpr unsigned long host_chunk(unsigned long frames, unsigned long n, bool pinned, bool posterior)
{
    const unsigned long frame_bytes = 4 * n, eighth = (frames + 7) / 8;
    const bool whole = !pinned || frames * frame_bytes < 6000000;
    const unsigned long fill = posterior ? 0 : 7000000 / frame_bytes, least = fill > 1024 ? fill : 1024;
    const unsigned long chunk = whole || eighth > 8192 ? 8192 : eighth < least ? least : eighth;
    return chunk < frames ? chunk : frames;
}

/* whether the driver copies from and to p without staging (null: nothing to copy) */
inline bool host_pinned(const void* p)
{
    if (!p) return true;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

}  // namespace wldpc

#endif
