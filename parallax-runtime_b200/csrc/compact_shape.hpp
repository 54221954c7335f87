// Tile shapes of the compaction kernels (kernels/compact.cu) and the padding of a flags array that
// follows from them. Plain C++: the host side sizes the array with it.
#pragma once

#include <stddef.h>

namespace pxb {

// One CTA per tile. Shape chosen by measurement (112 KiB tiles, 2 CTAs/SM); can be overridden at
// build time (PXB_COMPACT_BLOCK / _VPT / _SUB / _CTAS) to sweep it; SUB x (BLOCK / 32) must be 32.
#ifndef PXB_COMPACT_BLOCK
#define PXB_COMPACT_BLOCK 512
#endif
#ifndef PXB_COMPACT_VPT
#define PXB_COMPACT_VPT 7
#endif
#ifndef PXB_COMPACT_SUB
#define PXB_COMPACT_SUB 2
#endif
#ifndef PXB_COMPACT_CTAS
#define PXB_COMPACT_CTAS 2
#endif
// The pipeline: 15 parts of 3.5 KiB, four tiles and their flags fit an SM.
constexpr int kCompactPipeWorkers = 15;
constexpr int kCompactPipeVpt = 7;  // odd number of 16-byte words: conflict-free rows

// Elements of a tile, for elements of `elem` bytes.
constexpr size_t compact_tile(size_t elem) {
    return (size_t)PXB_COMPACT_SUB * PXB_COMPACT_BLOCK * PXB_COMPACT_VPT * (16 / elem);
}
constexpr size_t compact_pipe_tile(size_t elem) {
    return (size_t)kCompactPipeWorkers * 32 * kCompactPipeVpt * (16 / elem);
}

// Bytes of a flags array of n elements: the kernels read the flags of whole tiles (bytes past n are
// masked), so it reaches to the end of the last tile of every shape. The shapes do not nest.
constexpr size_t compact_flags_padding(size_t n) {
    const size_t tiles[] = {compact_tile(4), compact_tile(8), compact_pipe_tile(4), compact_pipe_tile(8)};
    size_t end = 0;
    for (size_t t : tiles) {
        const size_t e = (n + t - 1) / t * t;
        if (e > end) end = e;
    }
    return end + 16;
}

}  // namespace pxb
