// Ascending sort of large arrays: one-sweep LSD radix sort with 8-bit digits.
//
// Reference: a global bitonic network, one dispatch + fence wait per (k, j) stage
// (src/kernel/kernel_launcher.cpp:1568-1606, shaders/bitonic.comp:15-29).
//
// Keys are ordered as unsigned integers after the order-preserving transform of
// sortkey.cuh, exactly as the merge sort in sort.cu orders them. A sort under a total order
// of the key bits has one result, so both paths return the same bytes.
//
// Method: D. Adinets and D. Merrill, "Onesweep: A Faster Least Significant Digit Radix Sort
// for GPUs" (2022). One upfront kernel counts the histogram of every digit position in a
// single read of the keys. Then each digit pass, lowest digit first, reads and writes the
// keys once:
//   1. a persistent CTA claims the next tile (atomic counter, so every tile it waits on
//      belongs to a CTA that is already running or done) and loads its keys, warp-striped,
//      while the tile before it is looked back and written;
//   2. ranks them stably by the current digit, warp by warp: each warp walks its keys in
//      index order and, per 32 keys, groups lanes with equal digits (eight ballots and
//      shared lane masks in turn), so a key's rank is the warp's running count of its digit
//      plus its lower peers;
//   3. publishes the tile's 256 digit counts at once (state AGG), then finds each digit's
//      global offset by decoupled look-back over the per-(tile, digit) words of earlier
//      tiles (one thread per digit) and publishes the inclusive count (state INC); tile 0
//      starts every chain from the exclusive scan of the upfront histogram;
//   4. places the keys in digit order in shared memory and writes each digit's run to
//      its global offset, so a warp's stores cover consecutive addresses.
// Look-back words are 64-bit: [63:42] pass epoch, [41:40] state, [39:0] count. Words of
// earlier passes carry older epochs and read as "not ready", so nothing is cleared between
// passes. Waits are bounded like the other look-backs (lookback.cuh: kSpinLimit).
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "../pdl.cuh"
#include "../runtime.hpp"
#include "../segplan.cuh"
#include "../sortkey.cuh"
#include "../tiles.cuh"

namespace pxb {
namespace {

constexpr int kBins = 256;
constexpr int kValBits = 40;
constexpr uint64_t kValMask = (uint64_t(1) << kValBits) - 1;
constexpr uint64_t kStAgg = uint64_t(1) << kValBits;
constexpr uint64_t kStInc = uint64_t(2) << kValBits;
constexpr int kEpochShift = 42;
constexpr int kLookWindow = 4;  // predecessor words a look-back step loads at once

// Keys per thread ("rows" of 32 keys per warp) of the largest tile, at two 256-thread CTAs per
// SM. What bounds a pass is not HBM (a quarter busy) but the shared-memory pipe (random digits, 79 %
// busy) and the ALU (ballots, 54 %) together, plus a cost per tile (counts,
// digit scan, look-back) of some 4,000 cycles: large tiles of few warps win until the keys and
// their ranks no longer fit the 128 registers. Digit pass measured on B200, 2^26 uint32 keys /
// 2^25 int64 keys: 512 threads x 24 / 16 rows, one tile per CTA (as it was) 306 / 215 us; 256 x
// 48 / 32 226 / 169; 256 x 56 / 36 223 / 166; 64 rows 222 / -, 40 rows - / 184 (spills). Three
// CTAs per SM of 256 x 36 / 24 242 / 190.
template <typename K> struct RadixShape;
template <> struct RadixShape<uint32_t> {
    static constexpr int BLOCK = 256, ITEMS = 56, CTAS = 2;
};
template <> struct RadixShape<uint64_t> {
    static constexpr int BLOCK = 256, ITEMS = 36, CTAS = 2;
};

// Rows per warp of a tile of `keys` keys: a tile is spread over all warps in whole steps of
// kRowStep rows (the end is padded with the largest key). Steps of four keep the row loop's
// bounds checks off every row (239 against 252 us per pass with a check per row).
constexpr int kRowStep = 4;
template <int BLOCK>
__host__ __device__ __forceinline__ uint32_t rows_of(uint32_t keys) {
    return (keys + BLOCK * kRowStep - 1) / (BLOCK * kRowStep) * kRowStep;
}

// One tile of keys and two [warps][256] tables (counts, lane masks).
template <typename K>
constexpr size_t radix_smem() {
    return (size_t)RadixShape<K>::BLOCK * RadixShape<K>::ITEMS * sizeof(K) +
           (size_t)(RadixShape<K>::BLOCK / 32) * kBins * sizeof(uint32_t) * 2;
}

template <typename K>
__device__ __forceinline__ uint32_t digit_of(K k, int shift) {
    if constexpr (sizeof(K) == 8)  // shift is a multiple of 8 and the same for all threads
        return __byte_perm((uint32_t)(k >> (shift & 32)), 0u, 0x4440u | ((uint32_t)shift >> 3 & 3u));
    else
        return __byte_perm((uint32_t)k, 0u, 0x4440u | ((uint32_t)shift >> 3));
}

__device__ __forceinline__ uint64_t ld_relaxed_u64(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Lanes whose 8-bit digit equals this lane's: eight ballots, each inverted where the lane's
// own bit is clear (a test that sets a predicate, the vote, a predicated NOT and half an AND
// per bit).
__device__ __forceinline__ uint32_t ballot_peers(uint32_t d) {
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        uint32_t m;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "and.b32 %0, %1, %2;\n\t"
            "setp.ne.u32 p, %0, 0;\n\t"
            "vote.sync.ballot.b32 %0, p, 0xffffffff;\n\t"
            "@!p not.b32 %0, %0;\n\t}"
            : "=r"(m) : "r"(d), "r"(1u << b));
        peers &= m;
    }
    return peers;
}
__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---- upfront histogram ----------------------------------------------------------------------
// Counts, for every digit position p, how many keys have each digit value, in one read of
// the keys. Shared-memory atomics are the limit here, and what they cost is bank conflicts:
// each lane counts into its own copy of the histograms, laid out [p][digit][copy] with
// copy = lane % COPIES, so with 32 copies lane l always hits bank l (conflict-free) and
// with 16 copies at most two lanes share a bank. The host sizes the grid so that every
// per-CTA count stays below 2^32.
template <typename K> struct HistShape;
template <> struct HistShape<uint32_t> { static constexpr int COPIES = 32, U = 16; };
template <> struct HistShape<uint64_t> { static constexpr int COPIES = 16, U = 8; };
constexpr int kHistBlock = 1024;

template <typename K>
constexpr size_t hist_smem() {
    return (size_t)sizeof(K) * kBins * HistShape<K>::COPIES * sizeof(uint32_t);
}

template <typename K, int XF>
__global__ void __launch_bounds__(kHistBlock)
    k_radix_hist(const K* __restrict__ in, uint64_t n, unsigned long long* __restrict__ hist) {
    constexpr int P = sizeof(K);
    constexpr int COPIES = HistShape<K>::COPIES, U = HistShape<K>::U;
    extern __shared__ __align__(16) uint32_t sh[];  // [P][kBins][COPIES]
    for (int i = threadIdx.x; i < P * kBins * COPIES; i += kHistBlock) sh[i] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    uint32_t* const mine = sh + (lane % COPIES);
    const uint64_t stride = (uint64_t)gridDim.x * kHistBlock;
    uint64_t i = (uint64_t)blockIdx.x * kHistBlock + threadIdx.x;
    for (; i + (U - 1) * stride < n; i += U * stride) {
        K k[U];
#pragma unroll
        for (int u = 0; u < U; ++u) k[u] = to_key<K, XF>(__ldcs(in + i + u * stride));
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int p = 0; p < P; ++p)
                atomicAdd(mine + (p * kBins + digit_of(k[u], 8 * p)) * COPIES, 1u);
    }
    for (; i < n; i += stride) {
        const K k = to_key<K, XF>(in[i]);
#pragma unroll
        for (int p = 0; p < P; ++p) atomicAdd(mine + (p * kBins + digit_of(k, 8 * p)) * COPIES, 1u);
    }
    __syncthreads();
    // one (position, digit) row per thread; copies read in a lane-rotated order so a warp's
    // 32 rows hit 32 different banks
    for (int j = threadIdx.x; j < P * kBins; j += kHistBlock) {
        uint32_t v = 0;
#pragma unroll 8
        for (int c = 0; c < COPIES; ++c) v += sh[j * COPIES + ((c + lane) % COPIES)];
        if (v) atomicAdd(&hist[j], (unsigned long long)v);
    }
}

// Exclusive scan over the 256 digits held by threads 0..255 (one value each); every thread
// of the CTA calls it (threads 256.. pass zero). `part` is shared scratch of 8 elements.
template <typename T, int BLOCK>
__device__ __forceinline__ T digit_exclusive_scan(T v, T* part) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const T inc = warp_inclusive_scan(v, OpSum());
    if (warp < kBins / 32 && lane == 31) part[warp] = inc;
    __syncthreads();
    T before = T(0);
    if (warp < kBins / 32)
        for (int w = 0; w < warp; ++w) before += part[w];
    __syncthreads();  // part may be reused by the caller's next scan
    return before + inc - v;
}

// Segmented mode of a digit pass (many segments, each sorted on its own, in one launch): the
// claimed tile is work item `tile` of the planner's list (segplan.cuh), i.e. tile k of one
// segment; offsets are segment-local, the look-back stops at the segment's first tile, and
// that tile starts every digit's chain from the segment's own histogram.
struct SegRadix {
    SegSrc src;                   // segments: data at in_addr, temporary at aux_addr
    const uint32_t* item_start;   // S + 1: first work item of every segment
    const uint32_t* item_seg;     // work item -> segment
    const uint32_t* seg_hist;     // [S][npos][256] digit counts of every segment
    const uint32_t* epoch_base;   // this call's first pass epoch (device side)
    uint64_t S;
    uint32_t npos, pos;           // digit positions counted, this pass's position among them
    uint32_t parity;              // 0: data -> temporary, 1: temporary -> data
};

// ---- one digit pass --------------------------------------------------------------------------
// XF_IN transforms keys as they are read (the first pass reads the caller's values),
// XF_OUT restores them as they are written (the last pass writes the caller's values).
template <typename K, int XF_IN, int XF_OUT, bool SEG = false>
__global__ void __launch_bounds__(RadixShape<K>::BLOCK, RadixShape<K>::CTAS)
    k_radix_pass(const K* in_, K* out_, uint64_t n_, int shift, const unsigned long long* hist, uint64_t* status, uint32_t epoch_,
                 uint32_t tiles_, uint32_t tile_rows, uint32_t* counters, volatile int32_t* err,
                 SegRadix sr) {
    constexpr int BLOCK = RadixShape<K>::BLOCK, ITEMS = RadixShape<K>::ITEMS;
    constexpr int TILE = BLOCK * ITEMS, WARPS = BLOCK / 32;
    constexpr int G = kRowStep;
    static_assert(BLOCK == kBins, "one thread per digit");
    static_assert(ITEMS % G == 0 && 32 * ITEMS <= 0xffff, "whole steps, two 16-bit ranks per register");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K* const s_keys = reinterpret_cast<K*>(smem_raw);
    // [WARPS][kBins]: each warp's running count of every digit, then its offset in the tile
    uint32_t* const s_wh = reinterpret_cast<uint32_t*>(smem_raw + (size_t)TILE * sizeof(K));
    __shared__ uint64_t s_goff[kBins];
    __shared__ uint32_t s_goff32[kBins];
    __shared__ uint64_t s_part64[kBins / 32];
    __shared__ uint32_t s_part32[kBins / 32];
    __shared__ uint32_t s_tile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = lanemask_lt();
    const uint32_t self = 1u << lane;
    uint32_t* const wh = s_wh + warp * kBins;
    uint32_t* const wm = s_wh + (WARPS + warp) * kBins;
    for (int i = lane; i < kBins; i += 32) wh[i] = wm[i] = 0u;
    dependent_prologue();
    if (tid == 0) s_tile = atomicAdd(&counters[0], 1u);
    const uint32_t tiles = SEG ? sr.item_start[sr.S] : tiles_;
    const uint32_t epoch = SEG ? *sr.epoch_base + sr.pos : epoch_;
    const uint32_t tile_keys = BLOCK * tile_rows;
    __syncthreads();

    // plain: tile `tile` of the array; segmented: work item `tile` is tile tk of a segment
    struct Tile {
        const K* in;
        K* out;
        uint64_t n;
        uint32_t tk, seg, valid;
    };
    auto locate = [&](uint32_t tile) {
        Tile t;
        t.in = in_;
        t.out = out_;
        t.n = n_;
        t.tk = tile;
        t.seg = 0;
        if constexpr (SEG) {
            t.seg = sr.item_seg[tile];
            t.tk = tile - sr.item_start[t.seg];
            t.n = sr.src.len(t.seg);
            const uint64_t a = sr.src.in_addr(t.seg), b = sr.src.aux_addr(t.seg);
            t.in = reinterpret_cast<const K*>(sr.parity ? b : a);
            t.out = reinterpret_cast<K*>(sr.parity ? a : b);
            // shorter than two: sorted already, and may come without a temporary
            if (t.n < 2) t.n = 0;
        }
        const uint64_t base = (uint64_t)t.tk * tile_keys;
        const uint64_t rem = t.n > base ? t.n - base : 0;
        t.valid = rem < (uint64_t)tile_keys ? (uint32_t)rem : tile_keys;
        t.in += base;
        return t;
    };
    K k[ITEMS];
    // keys of warp w: tile positions [w * 32 * rows, (w + 1) * 32 * rows), row j of lane l at
    // w * 32 * rows + 32 j + l, so rows walked in order visit keys in index order
    auto load = [&](const Tile& t) {
        const uint32_t rows = rows_of<BLOCK>(t.valid);
        const uint32_t w0 = (uint32_t)warp * 32 * rows + lane;
        if (t.valid == (uint32_t)TILE) {
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) k[j] = __ldcs(t.in + w0 + 32 * j);
        } else if (t.valid != 0) {  // padding re-reads the last key; it is replaced later
#pragma unroll
            for (int j0 = 0; j0 < ITEMS; j0 += G) {
                if (j0 >= (int)rows) break;
#pragma unroll
                for (int j = j0; j < j0 + G; ++j) k[j] = __ldcs(t.in + min(w0 + 32 * j, t.valid - 1));
            }
        }
    };

    uint32_t tile = s_tile;
    Tile t;
    if (tile < tiles) {
        t = locate(tile);
        load(t);
    }
    while (tile < tiles) {
        const int rows = (int)rows_of<BLOCK>(t.valid);
        const uint32_t w0 = (uint32_t)warp * 32 * rows + lane;
        // padding at the tile's end: the largest key, digit 255 after all others
        if (t.valid == (uint32_t)rows * BLOCK) {
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) k[j] = to_key<K, XF_IN>(k[j]);
        } else {
#pragma unroll
            for (int j = 0; j < ITEMS; ++j)
                k[j] = w0 + 32 * j < t.valid ? to_key<K, XF_IN>(k[j]) : ~K(0);
        }

        // 1. stable ranks of the warp's rows by the current digit: wh[d] is the warp's count
        // of digit d so far; a key's rank is that count plus its lower peers in its row. Even
        // rows find their peers with ballots (ALU), odd rows through a table of lane masks
        // (shared-memory atomic OR, read back, cleared by the group's highest lane): the two
        // pipes share the work. Digit pass of 2^26 keys, all else equal: masks on every fourth
        // row 239 us, every third 231, every second 226 (tiles of 48 rows); every second 223,
        // two of three 227 (56 rows).
        uint32_t rank2[ITEMS / 2];  // 16-bit ranks, two per register
#pragma unroll
        for (int j0 = 0; j0 < ITEMS; j0 += G) {
            if (j0 >= rows) break;
#pragma unroll
            for (int j = j0; j < j0 + G; ++j) {
                const uint32_t d = digit_of(k[j], shift);
                uint32_t peers;
                if (j & 1) {
                    atomicOr(&wm[d], self);
                    __syncwarp();
                    peers = wm[d];
                } else {
                    peers = ballot_peers(d);
                }
                const uint32_t c = wh[d] + __popc(peers & lt);
                __syncwarp();
                if (peers >> lane == 1u) {  // the highest peer
                    wh[d] = c + 1;
                    if (j & 1) wm[d] = 0u;
                }
                __syncwarp();
                rank2[j / 2] = (j & 1) ? rank2[j / 2] | (c << 16) : c;
            }
        }
        __syncthreads();

        // 2. per digit: counts of the warps -> exclusive over warps (in key order); tile
        // count; publish AGG. Then the digit's start in the tile is added to every warp's
        // offset, so the placement finds a key's slot with one table read.
        uint32_t cnt = 0;
        uint32_t wex[WARPS];
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            wex[w] = cnt;
            cnt += s_wh[w * kBins + tid];
        }
        if (t.tk != 0)
            st_relaxed_u64(&status[(uint64_t)tile * kBins + tid],
                           ((uint64_t)epoch << kEpochShift) | kStAgg | cnt);
        uint32_t claim = 0;
        if (tid == 0) claim = atomicAdd(&counters[0], 1u);
        const uint32_t loc = digit_exclusive_scan<uint32_t, BLOCK>(cnt, s_part32);
        uint64_t start = 0;  // first tile: the digit's first output position
        if (t.tk == 0) {
            uint64_t h;
            if constexpr (SEG) h = sr.seg_hist[((uint64_t)t.seg * sr.npos + sr.pos) * kBins + tid];
            else h = hist[tid];
            start = digit_exclusive_scan<uint64_t, BLOCK>(h, s_part64);
        }
#pragma unroll
        for (int w = 0; w < WARPS; ++w) s_wh[w * kBins + tid] = wex[w] + loc;
        if (tid == 0) s_tile = claim;
        __syncthreads();

        // 3. keys in digit order in shared memory. (The empty asm keeps the compiler from
        // holding every key's digit in a register since the ranking.)
#pragma unroll
        for (int j0 = 0; j0 < ITEMS; j0 += G) {
            if (j0 >= rows) break;
            uint32_t slot[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int j = j0 + g;
                K key = k[j];
                if constexpr (sizeof(K) == 8) asm volatile("" : "+l"(key));
                else asm volatile("" : "+r"(key));
                const uint32_t r = (j & 1) ? rank2[j / 2] >> 16 : rank2[j / 2] & 0xffffu;
                slot[g] = wh[digit_of(key, shift)] + r;
            }
#pragma unroll
            for (int g = 0; g < G; ++g) s_keys[slot[g]] = k[j0 + g];
        }
        __syncwarp();
#pragma unroll
        for (int i = lane; i < kBins; i += 32) wh[i] = 0u;

        // the next tile's keys are on their way while this one looks back and is written
        const uint32_t next = s_tile;
        Tile tn = t;
        if (next < tiles) {
            tn = locate(next);
            load(tn);
        }

        // 4. look-back, one thread per digit. The words of the kLookWindow nearest unvisited
        // predecessors are loaded together, so one round trip to L2 covers several tiles; they
        // are then consumed in order until an inclusive count ends the walk.
        uint64_t excl = start;
        if (t.tk != 0) {  // (segmented: the walk ends at the segment's first tile, always INC)
            bool done = false;
            for (int64_t j = (int64_t)tile - 1; !done && j >= 0; j -= kLookWindow) {
                uint64_t w[kLookWindow];
#pragma unroll
                for (int q = 0; q < kLookWindow; ++q)
                    w[q] = j - q >= 0 ? ld_relaxed_u64(&status[(uint64_t)(j - q) * kBins + tid]) : 0;
#pragma unroll
                for (int q = 0; q < kLookWindow; ++q) {
                    if (done || j - q < 0) break;
                    uint64_t v = w[q];
                    uint32_t spins = 0;
                    while (!((uint32_t)(v >> kEpochShift) == epoch && (v & (kStAgg | kStInc)))) {
                        if (++spins > kSpinLimit) {
                            *err = 1;
                            done = true;
                            break;
                        }
                        if (spins > 8) nanosleep_ns(32);
                        v = ld_relaxed_u64(&status[(uint64_t)(j - q) * kBins + tid]);
                    }
                    if (done) break;
                    excl += v & kValMask;
                    if (v & kStInc) done = true;
                }
            }
        }
        st_relaxed_u64(&status[(uint64_t)tile * kBins + tid],
                       ((uint64_t)epoch << kEpochShift) | kStInc | ((excl + cnt) & kValMask));
        // output position of tile-sorted index x: goff[d] + x (excl >= loc always)
        s_goff[tid] = excl - loc;
        s_goff32[tid] = (uint32_t)(excl - loc);
        __syncthreads();

        // 5. each digit's run to its global offset
        bool bad = false;  // an output position outside the array: skipped and reported
        if (t.n <= 0xffffffffull && t.valid == (uint32_t)TILE) {  // whole tile, 32-bit offsets
            const uint32_t n32 = (uint32_t)t.n;
#pragma unroll
            for (int j0 = 0; j0 < ITEMS; j0 += G) {
                K key[G];
                uint32_t pos[G];
#pragma unroll
                for (int g = 0; g < G; ++g) key[g] = s_keys[(uint32_t)(j0 + g) * BLOCK + tid];
#pragma unroll
                for (int g = 0; g < G; ++g)
                    pos[g] = s_goff32[digit_of(key[g], shift)] + (uint32_t)(j0 + g) * BLOCK + tid;
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    if (pos[g] < n32) t.out[pos[g]] = from_key<K, XF_OUT>(key[g]);
                    else bad = true;
                }
            }
        } else {
#pragma unroll 4
            for (uint32_t x = tid; x < t.valid; x += BLOCK) {
                const K key = s_keys[x];
                const uint64_t pos = s_goff[digit_of(key, shift)] + x;
                if (pos < t.n) t.out[pos] = from_key<K, XF_OUT>(key);
                else bad = true;
            }
        }
        if (bad) *err = kErrRadixRange;
        tile = next;
        t = tn;
    }
    if (tid == 0) persistent_exit(counters);
}

// CTAs of a digit pass that can be resident at once: its grid.
template <typename K>
uint64_t radix_resident() {
    return (uint64_t)RadixShape<K>::CTAS * device_info().sm_count;
}

// Rows per warp of a tile (BLOCK x rows keys): the largest tile, cut so that the tiles fill
// whole waves of the resident CTAs (2^22 uint32 keys: 106 us against 122 with full tiles, the
// last wave nearly empty). An array that fits one tile per SM gets smaller tiles, one on every
// SM: two per SM make the look-back longer than the ranking they save (2^20 uint32 keys 60 us
// at two tiles per SM, 56 at one; 300,001 int64 keys 92 and 82).
template <typename K>
uint32_t radix_rows(uint64_t n) {
    constexpr uint64_t BLOCK = RadixShape<K>::BLOCK, ITEMS = RadixShape<K>::ITEMS;
    const uint64_t sms = device_info().sm_count;
    const uint64_t res = n <= BLOCK * ITEMS * sms ? sms : radix_resident<K>();
    const uint64_t waves = (n + BLOCK * ITEMS * res - 1) / (BLOCK * ITEMS * res);
    uint64_t rows = (n + BLOCK * res * waves - 1) / (BLOCK * res * waves);
    rows = (rows + kRowStep - 1) / kRowStep * kRowStep;
    return (uint32_t)(rows < ITEMS ? rows : ITEMS);
}

template <typename K, int XF_IN, int XF_OUT>
bool launch_pass(const K* in, K* out, uint64_t n, int shift, const unsigned long long* hist,
                 uint64_t* status, uint32_t epoch, uint32_t* counters, volatile int32_t* err,
                 uint64_t tiles, uint32_t rows, cudaStream_t s) {
    constexpr size_t smem = radix_smem<K>();
    if (!smem_opt_in<k_radix_pass<K, XF_IN, XF_OUT>>(smem))
        return cuda_ok(cudaGetLastError(), "k_radix_pass shared-memory opt-in");
    const uint64_t res = radix_resident<K>();
    return launch_dependent(k_radix_pass<K, XF_IN, XF_OUT>, (unsigned)(tiles < res ? tiles : res),
                            RadixShape<K>::BLOCK, smem, s, "k_radix_pass launch", in, out, n, shift,
                            hist, status, epoch, (uint32_t)tiles, rows, counters, err, SegRadix{});
}

// ---- segmented radix sort -------------------------------------------------------------------
// Digit counts of every segment for digit positions p0 .. P-1. A CTA takes `per_cta`
// consecutive work items (tiles; consecutive items are mostly of one segment), loads each
// tile's keys into registers before counting them in shared memory (one memory round trip
// per tile), and adds its counts to the segment's histogram with one global atomic per
// nonzero (position, digit) when the segment changes and at its end: a long segment costs
// one flush per `per_cta` tiles instead of one per tile. seg_hist must be zero on entry.
// Bank conflicts of the random digits bound it (122 M records: 262 us, 3.7 TB/s); eight copies
// of the counts, one per lane residue, measured 307 us.
constexpr int kSegHistBlock = 512;

// Work items per CTA: eight where that still leaves four CTAs for every SM; a short work list
// gets a CTA per item (five 8-byte items on one CTA: 45 us, on five 9 us).
inline uint32_t seg_hist_items(uint64_t items) {
    const uint64_t per = items / (4ull * device_info().sm_count);
    return per < 1 ? 1u : per > 8 ? 8u : (uint32_t)per;
}

template <typename K, int XF>
__global__ void __launch_bounds__(kSegHistBlock)
    k_seg_radix_hist(SegRadix sr, int p0, uint32_t per_cta, uint32_t tile, uint32_t* seg_hist) {
    dependent_prologue();
    constexpr int P = sizeof(K);
    constexpr int TILE = RadixShape<K>::BLOCK * RadixShape<K>::ITEMS;
    constexpr int PER = (TILE + kSegHistBlock - 1) / kSegHistBlock;
    __shared__ uint32_t h[P][kBins];
    const uint32_t total = sr.item_start[sr.S];
    const uint32_t i0 = blockIdx.x * per_cta;
    if (i0 >= total) return;
    const uint32_t i1 = total - i0 < per_cta ? total : i0 + per_cta;
    const int tid = threadIdx.x;
    const int npos = P - p0;
    for (int i = tid; i < P * kBins; i += kSegHistBlock) (&h[0][0])[i] = 0u;
    __syncthreads();
    auto flush = [&](uint64_t seg) {  // called by the whole CTA (segment ids are uniform)
        __syncthreads();
        for (int i = tid; i < npos * kBins; i += kSegHistBlock) {
            uint32_t& c = h[p0 + i / kBins][i % kBins];
            if (c) atomicAdd(&seg_hist[seg * npos * kBins + i], c);
            c = 0u;
        }
        __syncthreads();
    };
    uint64_t cur = sr.item_seg[i0];
    for (uint32_t item = i0; item < i1; ++item) {
        const uint64_t seg = sr.item_seg[item];
        if (seg != cur) {
            flush(cur);
            cur = seg;
        }
        const uint64_t len = sr.src.len(seg);
        if (len < 2) continue;  // not sorted (see k_radix_pass)
        const uint64_t k = item - sr.item_start[seg];
        const K* in = reinterpret_cast<const K*>(sr.src.in_addr(seg)) + k * tile;
        const uint64_t rem = len - k * tile;
        const uint32_t cnt = rem < (uint64_t)tile ? (uint32_t)rem : tile;
        K key[PER];
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const uint32_t i = (uint32_t)(tid + j * kSegHistBlock);
            key[j] = i < cnt ? to_key<K, XF>(__ldcs(in + i)) : K(0);
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if ((uint32_t)(tid + j * kSegHistBlock) >= cnt) break;
            for (int p = p0; p < P; ++p) atomicAdd(&h[p][digit_of(key[j], 8 * p)], 1u);
        }
    }
    flush(cur);
}

// Advances the device-side epoch of the segmented radix words by `npass` (so every replay
// of a captured call uses new epochs) and records this call's first epoch in counters[3].
// When the 22-bit epoch would wrap, the look-back words are cleared first.
__global__ void __launch_bounds__(256)
    k_seg_radix_epoch(uint32_t* counters, uint32_t npass, uint64_t* status, uint64_t words) {
    __shared__ uint32_t s_base;
    __shared__ bool s_wrap;
    dependent_prologue();
    if (threadIdx.x == 0) {
        uint32_t e = counters[2];
        if (e == 0) e = 1;  // a zeroed buffer: words of epoch 0 never match
        s_wrap = e + npass >= (1u << (64 - kEpochShift));
        s_base = s_wrap ? 1u : e;
    }
    __syncthreads();
    if (s_wrap)
        for (uint64_t i = threadIdx.x; i < words; i += 256) status[i] = 0ull;
    __syncthreads();
    if (threadIdx.x == 0) {
        counters[2] = s_base + npass;
        counters[3] = s_base;
    }
}

template <typename K, int XF_IN, int XF_OUT>
bool launch_seg_pass(const SegRadix& sr, int shift, uint64_t* status, uint32_t* counters,
                     volatile int32_t* err, uint64_t items_cap, uint32_t rows, cudaStream_t s) {
    constexpr size_t smem = radix_smem<K>();
    if (!smem_opt_in<k_radix_pass<K, XF_IN, XF_OUT, true>>(smem))
        return cuda_ok(cudaGetLastError(), "k_radix_pass shared-memory opt-in");
    const uint64_t res = radix_resident<K>();
    return launch_dependent(k_radix_pass<K, XF_IN, XF_OUT, true>,
                            (unsigned)(items_cap < res ? items_cap : res), RadixShape<K>::BLOCK,
                            smem, s, "segmented k_radix_pass launch", nullptr, nullptr, 0, shift,
                            nullptr, status, 0, 0, rows, counters, err, sr);
}

// S segments (CSR offsets or descriptors, segplan.cuh), each sorted in place by digit
// positions p0 .. P-1 (p0 = 4 on 8-byte records: stably by the high 32 bits). Launches: the
// planner (+ item map), a histogram clear, the segment histograms, the epoch step and one
// launch per digit pass; all capturable in a CUDA graph (device-side epochs).
template <typename K, int XF>
bool seg_radix_sort_keys(Workspace& ws, SegSrc src, uint64_t count, uint64_t S, int p0,
                         bool graph) {
    constexpr int P = sizeof(K);
    // a batch of little work gets smaller tiles, as a small array does
    const uint32_t rows = radix_rows<K>(count);
    const uint32_t tile = RadixShape<K>::BLOCK * rows;
    const uint64_t items_cap = S + count / tile + 1;
    const uint32_t npos = (uint32_t)(P - p0);
    if (items_cap >= 0x7fffffffull || (npos % 2) != 0) {
        set_error(PARALLAX_ERR_INVALID_ARGUMENT, "segmented sort: too many tiles");
        return false;
    }
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    const bool csr_tmp = src.offsets != nullptr;
    const size_t tmp_bytes = csr_tmp ? up(count * sizeof(K)) : 0;
    const size_t hist_bytes = up(S * npos * kBins * sizeof(uint32_t));
    char* t = static_cast<char*>(ws.temp(tmp_bytes + hist_bytes));
    char* sb = static_cast<char*>(ws.seg(256 + up((S + 1) * 4) + up(items_cap * 4)));
    StatusEntry* st = static_cast<StatusEntry*>(ws.seg_status(1));
    const uint64_t words = items_cap * kBins;
    char* rb = static_cast<char*>(ws.seg_radix(256 + words * 8));
    if (!t || !sb || !st || !rb) return false;
    if (csr_tmp) src.aux = reinterpret_cast<uint64_t>(t);
    src.aux_stride = 0;
    src.elem = sizeof(K);
    uint32_t* plan_counters = reinterpret_cast<uint32_t*>(sb);
    uint32_t* item_start = reinterpret_cast<uint32_t*>(sb + 256);
    uint32_t* item_seg = reinterpret_cast<uint32_t*>(sb + 256 + up((S + 1) * 4));
    uint32_t* seg_hist = reinterpret_cast<uint32_t*>(t + tmp_bytes);
    uint32_t* counters = reinterpret_cast<uint32_t*>(rb);
    uint64_t* status = reinterpret_cast<uint64_t*>(rb + 256);
    volatile int32_t* err = &ws.d_slot->spin_error;
    cudaStream_t s = ws.stream();

    SegRadix sr{};
    sr.src = src;
    sr.item_start = item_start;
    sr.item_seg = item_seg;
    sr.seg_hist = seg_hist;
    sr.epoch_base = counters + 3;
    sr.S = S;
    sr.npos = npos;
    ProfScope prof(ws, "segmented_radix_sort", 2 * count * sizeof(K));
    count_launch(4 + npos);
    auto enqueue = [&]() -> bool {
        if (!cuda_ok(cudaMemsetAsync(seg_hist, 0, hist_bytes, s), "segment histogram clear") ||
            !launch_dependent(k_seg_plan<kPlanBlock>, 1, kPlanBlock, 0, s, "segment plan launch", src, S, count, tile,
                              item_start, plan_counters, SegEmpty::NONE, nullptr, st,
                              ws.seg_status_cap, err, items_cap <= kInlineItems ? item_seg : nullptr))
            return false;
        if (items_cap > kInlineItems &&
            !launch_dependent(k_seg_map<256>, seg_map_grid(S), 256, 0, s, "segment map launch",
                              item_start, S, item_seg))
            return false;
        const uint32_t per = seg_hist_items(items_cap);
        if (!launch_dependent(k_seg_radix_hist<K, XF>, (unsigned)((items_cap + per - 1) / per),
                              kSegHistBlock, 0, s, "segment histogram launch", sr, p0, per, tile,
                              seg_hist) ||
            !launch_dependent(k_seg_radix_epoch, 1, 256, 0, s, "segment epoch launch", counters, npos,
                              status, words))
            return false;
        for (int p = p0; p < P; ++p) {
            SegRadix q = sr;
            q.pos = (uint32_t)(p - p0);
            q.parity = (uint32_t)((p - p0) & 1);
            bool ok;
            if (p == p0 && p == P - 1)
                ok = launch_seg_pass<K, XF, XF>(q, 8 * p, status, counters, err, items_cap, rows, s);
            else if (p == p0)
                ok = launch_seg_pass<K, XF, 0>(q, 8 * p, status, counters, err, items_cap, rows, s);
            else if (p == P - 1)
                ok = launch_seg_pass<K, 0, XF>(q, 8 * p, status, counters, err, items_cap, rows, s);
            else
                ok = launch_seg_pass<K, 0, 0>(q, 8 * p, status, counters, err, items_cap, rows, s);
            if (!ok) return false;
        }
        return cuda_ok(cudaGetLastError(), "segmented radix sort launch");
    };
    if (!graph) return enqueue();
    char key[256];
    snprintf(key, sizeof key, "segradix/%d/%d/%d/%p/%p/%llu/%llu", (int)sizeof(K), XF, p0,
             (const void*)src.in, (const void*)src.offsets, (unsigned long long)S,
             (unsigned long long)count);
    return graph_launch(ws, key, enqueue);
}

// The radix buffer: [0, 256) tile claim / exit counters, then a histogram per digit position, then
// the per-(tile, digit) look-back words.
constexpr size_t kRadixHistOff = 256;
template <typename K>
constexpr size_t kRadixStatusOff = kRadixHistOff + sizeof(K) * kBins * 8;

template <typename K>
size_t radix_bytes(uint64_t n) {
    const uint64_t tile = (uint64_t)RadixShape<K>::BLOCK * radix_rows<K>(n);
    return kRadixStatusOff<K> + (n + tile - 1) / tile * kBins * 8;
}

// Digit passes p0 .. P-1: p0 = 0 sorts by the whole key; p0 = 4 on 8-byte records sorts
// them stably by their high 32 bits alone (LSD passes are stable), the (key << 32 | value)
// records of a sort_kv handle.
template <typename K, int XF>
bool radix_sort_keys(Workspace& ws, void* d_data, uint64_t n, int p0 = 0) {
    constexpr int P = sizeof(K);
    const uint32_t rows = radix_rows<K>(n);
    const uint64_t tile = (uint64_t)RadixShape<K>::BLOCK * rows;
    const uint64_t tiles = (n + tile - 1) / tile;
    if (tiles > 0x7fffffffull || n > kValMask) {
        set_error(PARALLAX_ERR_INVALID_ARGUMENT, "sort: too many elements");
        return false;
    }
    K* data = static_cast<K*>(d_data);
    K* tmp = static_cast<K*>(ws.temp(n * sizeof(K)));
    if (!tmp) return false;
    char* rb = static_cast<char*>(ws.radix(radix_bytes<K>(n)));
    if (!rb) return false;
    const uint32_t ep0 = ws.next_radix_epochs(P);
    uint32_t* counters = reinterpret_cast<uint32_t*>(rb);
    auto* hist = reinterpret_cast<unsigned long long*>(rb + kRadixHistOff);
    auto* status = reinterpret_cast<uint64_t*>(rb + kRadixStatusOff<K>);
    volatile int32_t* err = &ws.d_slot->spin_error;
    cudaStream_t s = ws.stream();
    if (!cuda_ok(cudaMemsetAsync(hist, 0, (size_t)P * kBins * 8, s), "radix histogram clear"))
        return false;
    {
        // grid: one CTA per SM (the copies fill most of its shared memory), more when needed
        // to keep per-CTA counts below 2^31
        uint64_t grid = (uint64_t)device_info().sm_count;
        const uint64_t need = (n + kHistBlock - 1) / kHistBlock;
        if (grid > need) grid = need;
        const uint64_t min_grid = (n >> 31) + 1;
        if (grid < min_grid) grid = min_grid;
        constexpr size_t hsmem = hist_smem<K>();
        if (!smem_opt_in<k_radix_hist<K, XF>>(hsmem))
            return cuda_ok(cudaGetLastError(), "k_radix_hist shared-memory opt-in");
        ProfScope prof(ws, "k_radix_hist", n * sizeof(K));
        k_radix_hist<K, XF><<<(unsigned)grid, kHistBlock, hsmem, s>>>(data, n, hist);
    }
    count_launch();
    static_assert(P % 2 == 0, "an even number of passes ends in the caller's array");
    for (int p = p0; p < P; ++p) {  // P - p0 is even, so the last pass ends in `data`
        const K* src = ((p - p0) % 2 == 0) ? data : tmp;
        K* dst = ((p - p0) % 2 == 0) ? tmp : data;
        const unsigned long long* hp = hist + (size_t)p * kBins;
        bool ok;
        {
            ProfScope prof(ws, "k_radix_pass", 2 * n * sizeof(K));
            if (p == p0)
                ok = launch_pass<K, XF, 0>(src, dst, n, 8 * p, hp, status, ep0 + p, counters, err,
                                           tiles, rows, s);
            else if (p == P - 1)
                ok = launch_pass<K, 0, XF>(src, dst, n, 8 * p, hp, status, ep0 + p, counters, err,
                                           tiles, rows, s);
            else
                ok = launch_pass<K, 0, 0>(src, dst, n, 8 * p, hp, status, ep0 + p, counters, err,
                                          tiles, rows, s);
        }
        if (!ok) return false;
        count_launch();
    }
    return cuda_ok(cudaGetLastError(), "radix sort launch");
}

}  // namespace

bool launch_segmented_radix_sort(Workspace& ws, DType t, const SegSrc& src, uint64_t count,
                                 uint64_t S, bool by_key, bool graph) {
    if (by_key) {
        if (t != DType::U64) {
            set_error(PARALLAX_ERR_INVALID_ARGUMENT, "segmented sort: by-key sorts 8-byte records");
            return false;
        }
        return seg_radix_sort_keys<uint64_t, 0>(ws, src, count, S, 4, graph);
    }
    switch (t) {
        case DType::U32: return seg_radix_sort_keys<uint32_t, 0>(ws, src, count, S, 0, graph);
        case DType::I32: return seg_radix_sort_keys<uint32_t, 1>(ws, src, count, S, 0, graph);
        case DType::F32: return seg_radix_sort_keys<uint32_t, 2>(ws, src, count, S, 0, graph);
        case DType::U64: return seg_radix_sort_keys<uint64_t, 0>(ws, src, count, S, 0, graph);
        case DType::I64: return seg_radix_sort_keys<uint64_t, 1>(ws, src, count, S, 0, graph);
        case DType::F64: return seg_radix_sort_keys<uint64_t, 2>(ws, src, count, S, 0, graph);
        default: break;
    }
    set_error(PARALLAX_ERR_INVALID_ARGUMENT, "segmented sort: unsupported element type");
    return false;
}

uint64_t segmented_radix_tile(DType t) {
    return dtype_size(t) == 4 ? (uint64_t)RadixShape<uint32_t>::BLOCK * RadixShape<uint32_t>::ITEMS
                              : (uint64_t)RadixShape<uint64_t>::BLOCK * RadixShape<uint64_t>::ITEMS;
}

size_t radix_buffer_bytes(DType t, size_t n) {
    return dtype_size(t) == 4 ? radix_bytes<uint32_t>(n) : radix_bytes<uint64_t>(n);
}

bool launch_radix_sort(Workspace& ws, DType t, void* d_data, size_t n, bool by_key) {
    if (by_key) {
        if (t != DType::U64) {
            set_error(PARALLAX_ERR_INVALID_ARGUMENT, "sort: by-key sorts 8-byte records");
            return false;
        }
        return radix_sort_keys<uint64_t, 0>(ws, d_data, n, 4);
    }
    switch (t) {
        case DType::U32: return radix_sort_keys<uint32_t, 0>(ws, d_data, n);
        case DType::I32: return radix_sort_keys<uint32_t, 1>(ws, d_data, n);
        case DType::F32: return radix_sort_keys<uint32_t, 2>(ws, d_data, n);
        case DType::U64: return radix_sort_keys<uint64_t, 0>(ws, d_data, n);
        case DType::I64: return radix_sort_keys<uint64_t, 1>(ws, d_data, n);
        case DType::F64: return radix_sort_keys<uint64_t, 2>(ws, d_data, n);
        default: break;
    }
    set_error(PARALLAX_ERR_INVALID_ARGUMENT, "sort: unsupported element type");
    return false;
}

}  // namespace pxb
