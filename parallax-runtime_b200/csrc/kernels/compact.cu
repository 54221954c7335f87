// Stable single-pass compaction: copy_if / remove_if / unique, and stable partition.
//
// Reference: four or more dispatches with fence waits - a flags kernel writing 1.0/0.0
// in the ELEMENT type, a multi-pass scan of those flags, a host read of the last
// position, then a scatter kernel (src/kernel/kernel_launcher.cpp:1701-1791,
// shaders/flags.comp:14-18, shaders/scatter.comp:15-22). Element-typed positions make
// fp32 counts inexact beyond 2^24; here counts are 32-bit within a tile and 64-bit
// across tiles.
//
// Here: arrays of more than a wave go through a persistent warp-specialised pipeline
// (k_compact_pipe); smaller ones and unaligned inputs take one 512-thread CTA per 112 or 56 KiB
// tile, in blockIdx order, staged as bulk-copied sub-tiles (tiles.cuh). Phase 1 evaluates the
// predicate (or the adjacent-difference test for unique) on 28 / 14 consecutive elements per thread
// as each sub-tile lands, keeps the flags as bit masks, and ranks the kept elements with one shuffle
// scan per sub-tile and one 32-lane scan over the (sub-tile, warp) counts; the tile's output offset
// comes from a decoupled look-back on kept counts. Phase 2 packs the kept elements at the front of
// the staged tile, sub-tile by sub-tile (a packed element never lands beyond the sub-tile
// being packed), and writes them with coalesced stores. Traffic: n*s read + k*s written.
// Partition writes every element: kept ones to [0, k), the rest in order to [k, n). The
// rejected elements' offsets need k, so partition runs a count pass first (one read of
// the input); each sub-tile is then permuted in shared memory (kept run, rejected run)
// and both runs are written with coalesced stores.
#include <stdint.h>

#include <type_traits>

#include "../compact_shape.hpp"
#include "../lookback.cuh"
#include "../pdl.cuh"
#include "../pred.cuh"
#include "../runtime.hpp"
#include "../tiles.cuh"
#include "../tma.cuh"

namespace pxb {
namespace {

constexpr int kBlock = PXB_COMPACT_BLOCK;
constexpr int kVpt = PXB_COMPACT_VPT;
constexpr int kSub = PXB_COMPACT_SUB;
constexpr int kCtasPerSm = PXB_COMPACT_CTAS;

template <typename T>
struct Shape {
    static constexpr int V = 16 / sizeof(T);
    static constexpr int ITEMS = kVpt * V;
    static constexpr int SUB = kBlock * ITEMS;
    static constexpr int TILE = kSub * SUB;
    static constexpr size_t SMEM = TILE * sizeof(T);
    static_assert(TILE == compact_tile(sizeof(T)), "flags arrays are padded to it");
};

// Shared state of one CTA's tile processing.
struct CompactSmem {
    uint32_t cnt[32];               // (sub-tile, warp) kept counts
    uint64_t red[kBlock / 32 + 1];  // look-back scratch
    int first[kBlock / 32];
};

// One staged tile: flags, ranks, look-back, then packed (select / unique) or scattered
// (partition) output. MODE: 0 select (copy_if / remove_if), 1 unique, 2 partition.
// `prev_of_tile` is the element before the tile (unique only). Ends with a barrier after
// which the tile buffer may be refilled.
template <typename T, int MODE, bool BULK, int NSUB>
__device__ __forceinline__ void compact_tile(T* buf, uint64_t* bars, uint32_t parity,
                                             CompactSmem& sm, uint64_t tile, uint64_t base,
                                             uint32_t cnt, T prev_of_tile, T* out, uint64_t n,
                                             const PredDev<T>& pred,
                                             const TileStatus<uint64_t>& ts,
                                             const unsigned long long* num_true,
                                             unsigned long long* count_out, bool last_tile) {
    constexpr int V = Shape<T>::V;
    constexpr int ITEMS = Shape<T>::ITEMS;
    constexpr int SUB = Shape<T>::SUB;
    constexpr int WARPS = kBlock / 32;
    static_assert(NSUB * WARPS <= 32, "one lane per (sub-tile, warp)");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t row0 = (uint32_t)tid * ITEMS;

    // ---- phase 1: flags and ranks ----
    uint32_t fl[NSUB];   // bit j: element j of this thread's row in sub-tile s is kept
    uint32_t tex[NSUB];  // kept elements before this row within its warp
#pragma unroll
    for (int s = 0; s < NSUB; ++s) {
        if constexpr (BULK) wait_bar(&bars[s], parity, ts.err);
        const uint32_t e0 = (uint32_t)s * SUB + row0;  // tile index of the row's first element
        T x[ITEMS];
        load_row<T, ITEMS, V>(buf + e0, x);
        uint32_t f = 0;
        if constexpr (MODE == 1) {
            const T prev = e0 > 0 ? buf[e0 - 1] : prev_of_tile;
            const bool first_global = base == 0 && e0 == 0;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const bool keep = (j == 0 && first_global) || !(x[j] == (j ? x[j - 1] : prev));
                if (e0 + j < cnt && keep) f |= 1u << j;
            }
        } else {
            f = pred.template flags<ITEMS>(x, base + e0);
            if (e0 + ITEMS > cnt) f &= e0 >= cnt ? 0u : (1u << (cnt - e0)) - 1u;
        }
        fl[s] = f;
        const uint32_t incl = warp_inclusive_scan((uint32_t)__popc(f), OpSum());
        const uint32_t ex = shfl_up(incl, 1);
        tex[s] = lane == 0 ? 0u : ex;
        if (lane == 31) sm.cnt[s * WARPS + warp] = incl;
    }
    __syncthreads();
    // Every warp scans the 32 (sub-tile, warp) counts itself, then the whole CTA runs the
    // look-back on kept counts.
    uint32_t woff[NSUB];  // kept elements before this warp's rows within the tile
    uint32_t tile_kept;
    {
        const uint32_t v = lane < NSUB * WARPS ? sm.cnt[lane] : 0u;
        const uint32_t vi = warp_inclusive_scan(v, OpSum());
        tile_kept = shfl_idx(vi, 31);
        uint32_t vex = shfl_up(vi, 1);
        if (lane == 0) vex = 0;
#pragma unroll
        for (int s = 0; s < NSUB; ++s) woff[s] = shfl_idx(vex, s * WARPS + warp);
    }
    const uint64_t prefix =
        lookback_cta<uint64_t, kBlock, true>(ts, tile, (uint64_t)tile_kept, sm.red, sm.first);
    if (MODE != 2 && last_tile && tid == 0) *count_out = prefix + tile_kept;

    if constexpr (MODE == 2) {
        // ---- partition: per sub-tile, kept elements are packed at its front and the
        // rejected ones after them (an in-place permutation of the sub-tile, done from
        // registers after a barrier), then both runs are stored with coalesced writes:
        // kept to [prefix + kept before the sub-tile, ...), rejected to
        // [num_true + rejected before the sub-tile, ...).
        const uint64_t nt = *num_true;
        const uint64_t rej_base = nt + (base - prefix);
        uint32_t sub_before[NSUB + 1];  // kept elements of the tile before each sub-tile
        {
            const uint32_t v = lane < NSUB * WARPS ? sm.cnt[lane] : 0u;
            const uint32_t vi = warp_inclusive_scan(v, OpSum());
            uint32_t vex = shfl_up(vi, 1);
            if (lane == 0) vex = 0;
#pragma unroll
            for (int s = 0; s < NSUB; ++s) sub_before[s] = shfl_idx(vex, s * WARPS);
            sub_before[NSUB] = tile_kept;
        }
#pragma unroll
        for (int s = 0; s < NSUB; ++s) {
            const uint32_t s0 = (uint32_t)s * SUB;
            const uint32_t ks = sub_before[s + 1] - sub_before[s];      // kept in sub-tile
            const uint32_t valid = cnt > s0 ? (cnt - s0 < (uint32_t)SUB ? cnt - s0 : (uint32_t)SUB) : 0u;
            T* sb = buf + s0;
            T x[ITEMS];
            load_row<T, ITEMS, V>(sb + row0, x);
            __syncthreads();  // every row of sub-tile s is in registers before permuting
            uint32_t rk = woff[s] + tex[s] - sub_before[s];  // kept before this row (sub-tile)
            uint32_t rr = row0 - rk;                          // rejected before this row
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                if (row0 + j >= valid) break;
                if (fl[s] >> j & 1u) sb[rk++] = x[j];
                else sb[ks + rr++] = x[j];
            }
            __syncthreads();
            const uint64_t kdst = prefix + sub_before[s];
            const uint64_t rdst = rej_base + (s0 - sub_before[s]);
            for (uint32_t i = tid; i < valid; i += kBlock) {
                const uint64_t dst = i < ks ? kdst + i : rdst + (i - ks);
                if (dst < n) out[dst] = sb[i];
                else *ts.err = 3;  // only reachable after a failed wait: never write out of range
            }
        }
        if (tid == 0 && last_tile) *count_out = nt;
    } else {
        // ---- pack kept elements at the front of the tile, then store them ----
#pragma unroll
        for (int s = 0; s < NSUB; ++s) {
            T x[ITEMS];
            load_row<T, ITEMS, V>(buf + (uint32_t)s * SUB + row0, x);
            __syncthreads();  // every row of sub-tile s is in registers before packing
            uint32_t r = woff[s] + tex[s];
#pragma unroll
            for (int j = 0; j < ITEMS; ++j)
                if (fl[s] >> j & 1u) buf[r++] = x[j];
        }
        __syncthreads();
        for (uint32_t i = tid; i < tile_kept; i += kBlock) {
            if (prefix + i < n) out[prefix + i] = buf[i];
            else *ts.err = 3;
        }
    }
    __syncthreads();  // buffer and shared state free for the next tile
}

// One CTA per tile of NSUB sub-tiles (arrays of at most a wave, unaligned inputs), in blockIdx order
// (see k_scan).
template <typename T, int MODE, bool BULK, int NSUB>
__global__ void __launch_bounds__(kBlock, kCtasPerSm)
k_compact(const T* in, T* out, uint64_t n, PredDev<T> pred, TileStatus<uint64_t> ts,
          const unsigned long long* num_true,
          unsigned long long* count_out) {
    constexpr int SUB = Shape<T>::SUB;
    constexpr int TILE = NSUB * SUB;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* buf = reinterpret_cast<T*>(smem_raw);
    __shared__ __align__(8) uint64_t bars[NSUB];
    __shared__ CompactSmem sm;
    dependent_prologue();
    const uint64_t tile = blockIdx.x;
    const uint64_t base = tile * (uint64_t)TILE;
    const uint64_t rem = n - base;
    const uint32_t cnt = rem < (uint64_t)TILE ? (uint32_t)rem : (uint32_t)TILE;
    stage_tile<T, SUB, NSUB, kBlock, BULK>(buf, bars, in, base, cnt);
    const T prev = (MODE == 1 && base > 0) ? in[base - 1] : T(0);
    __syncthreads();
    compact_tile<T, MODE, BULK, NSUB>(buf, bars, 0, sm, tile, base, cnt, prev, out, n, pred, ts,
                                num_true, count_out, tile == gridDim.x - 1);
}

// Persistent pipeline without CTA-wide barriers, one CTA per SM (compare k_scan_pipe, scan.cu).
// Input 16-byte aligned.
//   mover      claims a tile, bulk-loads it (and, for unique, the 16 bytes before it) into a free
//              buffer
//   workers    every warp owns a part of each tile, a row of ITEMS elements per lane. It evaluates
//              the flags of the next tile as soon as that has landed, else packs the oldest tile
//              whose offset is known: kept elements to the front of its part, then stored as one
//              run. Counting comes first, so a tile's count never waits for a look-back.
//   publisher  the tile's count
//   look-back  the tile's output offset
// What bounds it is the workers' latency chain per tile (flags 1,000 to 1,800 cycles, packing 1,200,
// storing 900 of a 4,600-cycle period) behind HBM at 0.7 to 0.85 of the copy rate. 2^28 int32 x % 3
// == 0 / fp32 x > 0.5 / unique, us: one CTA per 112 KiB tile 397 / 399 / 354, the same with a line per
// look-back entry 350 / 358 / 309, this pipeline 299 / 297 / 266. Before a part was totalled with one
// redux instead of five shuffles 313 / 301 / 270; then also 20 workers with rows of 80 bytes 315 / 311 /
// 281, 24 with 48 bytes and five buffers 426 / 381 / 350, 20 with 112 bytes and three buffers 313 / 342
// / 297, counting and packing on separate warps 395 / 422 / 342; now also 12 workers and five buffers
// 326 / 315 / 295, two groups of 14 workers on alternate tiles 344 / 348 / 310, two or three look-back
// warps or a walk that starts before the count is known 301 / 299 / 268.
constexpr int kPipeWorkers = kCompactPipeWorkers;
constexpr int kPipeStages = 4;
constexpr int kPipeBlock = (kPipeWorkers + 3) * 32;

template <typename T>
struct PipeShape {
    static constexpr int V = 16 / sizeof(T);
    static constexpr int ITEMS = kCompactPipeVpt * V;
    static constexpr int PART = 32 * ITEMS;
    static constexpr int TILE = kPipeWorkers * PART;  // 52.5 KiB
    static constexpr size_t SMEM = (size_t)kPipeStages * TILE * sizeof(T);
    static_assert(TILE == compact_pipe_tile(sizeof(T)), "flags arrays are padded to it");
};

template <typename T, int MODE>
__global__ void __launch_bounds__(kPipeBlock, 1)
k_compact_pipe(const T* in, T* out, uint64_t n, uint32_t num_tiles, PredDev<T> pred,
               TileStatus<uint64_t> ts, const unsigned long long* num_true,
               unsigned long long* count_out, uint32_t* counters) {
    using Sh = PipeShape<T>;
    constexpr int V = Sh::V, ITEMS = Sh::ITEMS, PART = Sh::PART, TILE = Sh::TILE;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* const bufs = reinterpret_cast<T*>(smem_raw);
    __shared__ __align__(16) T s_head[kPipeStages][V];            // the 16 bytes before the tile
    __shared__ __align__(8) uint64_t full[kPipeStages], counted[kPipeStages], published[kPipeStages],
        ready[kPipeStages], packed[kPipeStages];
    __shared__ uint32_t s_flags[kPipeStages][kPipeWorkers * 32];  // kept elements of every row
    __shared__ uint32_t s_tot[kPipeStages][kPipeWorkers];         // kept of a part
    __shared__ uint32_t s_before[kPipeStages][kPipeWorkers];      // kept of the tile before it
    __shared__ uint64_t s_prefix[kPipeStages];                    // kept before the tile
    __shared__ uint32_t s_kept[kPipeStages];
    __shared__ uint32_t s_tile[kPipeStages];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < kPipeStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&counted[s], kPipeWorkers);
            mbar_init(&published[s], 1);
            mbar_init(&ready[s], 1);
            mbar_init(&packed[s], kPipeWorkers);
        }
        fence_mbar_init();
    }
    __syncthreads();
    dependent_prologue();
    auto count_of = [&](uint32_t t) {
        const uint64_t rem = n - (uint64_t)t * TILE;
        return rem < (uint64_t)TILE ? (uint32_t)rem : (uint32_t)TILE;
    };
    auto phase = [](uint32_t it) { return (it / kPipeStages) & 1u; };
    // Warp-uniform test of a barrier: lanes may see it complete at different polls, and the phase
    // cannot move on before this warp has arrived, so every lane then waits for what one lane saw.
    auto landed = [&](uint64_t* bar, uint32_t parity) {
        if (!__any_sync(0xffffffffu, mbar_test_wait(bar, parity))) return false;
        wait_bar(bar, parity, ts.err);
        return true;
    };

    if (warp < kPipeWorkers) {
        const uint32_t w0 = (uint32_t)warp * PART, row0 = (uint32_t)tid * ITEMS;
        const uint64_t nt = MODE == 2 ? *num_true : 0;
        uint32_t ci = 0, pi = 0;  // tiles counted and packed by this warp so far
        bool more = true;         // the claim counter has not run out
        uint32_t spins = 0;
        while (more || pi < ci) {
            const bool may_count = more && ci - pi < kPipeStages;
            if (may_count && landed(&full[ci % kPipeStages], phase(ci))) {
                spins = 0;
                const uint32_t b = ci % kPipeStages, t = s_tile[b];
                if (t >= num_tiles) {
                    more = false;
                    continue;
                }
                const T* const buf = bufs + b * TILE;
                const uint64_t base = (uint64_t)t * TILE;
                const uint32_t cnt = count_of(t);
                T x[ITEMS];
                load_row<T, ITEMS, V>(buf + row0, x);
                uint32_t f = 0;
                if constexpr (MODE == 1) {
                    const T prev = tid > 0 ? buf[row0 - (tid > 0)] : s_head[b][V - 1];
#pragma unroll
                    for (int j = 0; j < ITEMS; ++j)
                        f |= (uint32_t)!(x[j] == (j ? x[j > 0 ? j - 1 : 0] : prev)) << j;
                    if (t == 0 && tid == 0) f |= 1u;
                } else {
                    f = pred.template flags<ITEMS>(x, base + row0);
                }
                if (row0 + ITEMS > cnt) f &= row0 >= cnt ? 0u : (1u << (cnt - row0)) - 1u;
                s_flags[b][tid] = f;
                const uint32_t tot = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(f));
                if (lane == 0) {
                    s_tot[b][warp] = tot;
                    mbar_arrive(&counted[b]);
                }
                ++ci;
                continue;
            }
            if (pi < ci && landed(&ready[pi % kPipeStages], phase(pi))) {
                spins = 0;
                const uint32_t b = pi % kPipeStages, t = s_tile[b];
                T* const part = bufs + b * TILE + w0;
                const uint32_t f = s_flags[b][tid];
                T x[ITEMS];
                load_row<T, ITEMS, V>(bufs + b * TILE + row0, x);
                const uint32_t c = __popc(f);
                const uint32_t incl = warp_inclusive_scan(c, OpSum());
                const uint32_t kept = shfl_idx(incl, 31);
                const uint32_t before = s_before[b][warp];
                const uint64_t kdst = s_prefix[b] + before;
                uint32_t valid = 0;
                __syncwarp();  // every row is in registers before the part is overwritten
                uint32_t r = incl - c;
                if constexpr (MODE == 2) {
                    const uint32_t cnt = count_of(t);
                    valid = cnt > w0 ? min(cnt - w0, (uint32_t)PART) : 0u;
                    const uint32_t e0 = lane * ITEMS;
                    uint32_t q = kept + e0 - r;  // rejected ones after the kept run
#pragma unroll
                    for (int j = 0; j < ITEMS; ++j) {
                        const bool keep = f >> j & 1u;
                        if (e0 + j < valid) part[keep ? r : q] = x[j];
                        r += keep;
                        q += !keep;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < ITEMS; ++j)
                        if (f >> j & 1u) part[r++] = x[j];
                }
                __syncwarp();
                // a run of the part to the output, in steps of whole 128-byte lines
                auto store = [&](uint64_t dst, const T* src, uint32_t len) {
                    constexpr int L = 128 / sizeof(T);
                    if (len == 0) return;
                    if (dst + len > n) {  // only after a failed wait: never out of range
                        *ts.err = 3;
                        return;
                    }
                    T* const o = out + dst;
                    const int skew = (int)((reinterpret_cast<uintptr_t>(o) / sizeof(T)) % L);
                    int i = lane - skew;
                    if (i >= 0 && i < (int)len) o[i] = src[i];
#pragma unroll 4
                    for (i += 32; i < (int)len; i += 32) if (i >= 0) o[i] = src[i];
                };
                store(kdst, part, kept);
                if constexpr (MODE == 2)
                    store(nt + ((uint64_t)t * TILE + w0 - kdst), part + kept, valid - kept);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&packed[b]);
                ++pi;
                continue;
            }
            if (++spins > kSpinLimit) {
                *ts.err = 2;
                break;
            }
            nanosleep_ns(32);
        }
    } else if (warp == kPipeWorkers) {  // publisher
        for (uint32_t it = 0;; ++it) {
            const uint32_t b = it % kPipeStages;
            wait_bar(&full[b], phase(it), ts.err);
            const uint32_t t = s_tile[b];
            if (t >= num_tiles) break;
            wait_bar(&counted[b], phase(it), ts.err);
            const uint32_t v = lane < kPipeWorkers ? s_tot[b][lane] : 0u;
            const uint32_t vi = warp_inclusive_scan(v, OpSum());
            if (lane < kPipeWorkers) s_before[b][lane] = vi - v;
            if (lane == 31) {
                publish_aggregate<uint64_t>(ts, t, vi);
                s_kept[b] = vi;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&published[b]);
        }
    } else if (warp == kPipeWorkers + 1) {  // look-back
        for (uint32_t it = 0;; ++it) {
            const uint32_t b = it % kPipeStages;
            wait_bar(&full[b], phase(it), ts.err);
            const uint32_t t = s_tile[b];
            if (t >= num_tiles) break;
            wait_bar(&published[b], phase(it), ts.err);
            const uint64_t kept = s_kept[b];
            const uint64_t prefix = lookback_warp<uint64_t>(ts, t, kept);
            __syncwarp();  // every lane has read the slot (the first tile's walk has no step)
            if (lane == 0) {
                s_prefix[b] = prefix;
                if (t == num_tiles - 1) *count_out = MODE == 2 ? *num_true : prefix + kept;
                mbar_arrive(&ready[b]);
            }
        }
    } else if (lane == 0) {  // mover
        auto load = [&](uint32_t b, uint32_t t) {
            s_tile[b] = t;
            if (t >= num_tiles) {
                mbar_arrive(&full[b]);
                return;
            }
            const uint64_t base = (uint64_t)t * TILE;
            const uint32_t cnt = count_of(t), bulk = bulk_elems<T>(cnt);
            const bool head = MODE == 1 && t != 0;
            T* const buf = bufs + b * TILE;
            for (uint32_t e = bulk; e < cnt; ++e) buf[e] = in[base + e];
            mbar_arrive_expect_tx(&full[b], bulk * (uint32_t)sizeof(T) + (head ? 16u : 0u));
            if (bulk) bulk_load(buf, in + base, bulk * (uint32_t)sizeof(T), &full[b]);
            if (head) bulk_load(s_head[b], in + base - V, 16, &full[b]);
        };
        // one claim at a time, so the CTAs' first tiles interleave (see k_scan_pipe)
        for (uint32_t b = 0; b < kPipeStages; ++b) {
            if (b) wait_bar(&full[b - 1], 0, ts.err);
            load(b, atomicAdd(&counters[0], 1u));
        }
        for (uint32_t it = 0;; ++it) {
            const uint32_t b = it % kPipeStages;
            if (s_tile[b] >= num_tiles) break;
            const uint32_t next = atomicAdd(&counters[0], 1u);
            wait_bar(&packed[b], phase(it), ts.err);
            load(b, next);
        }
        persistent_exit(counters);
    }
}

template <typename T, int MODE, bool BULK, int NSUB>
bool launch_tiles(uint64_t n, cudaStream_t s, const T* in, T* out, PredDev<T> p,
                  TileStatus<uint64_t> ts, const unsigned long long* nt,
                  unsigned long long* count_out) {
    constexpr size_t smem = (size_t)NSUB * Shape<T>::SUB * sizeof(T);
    constexpr uint64_t tile = (uint64_t)NSUB * Shape<T>::SUB;
    if (!smem_opt_in<k_compact<T, MODE, BULK, NSUB>>(smem))
        return cuda_ok(cudaGetLastError(), "k_compact shared-memory opt-in");
    return launch_dependent(k_compact<T, MODE, BULK, NSUB>, (unsigned)((n + tile - 1) / tile), kBlock, smem,
                            s, "k_compact launch", in, out, n, p, ts, nt, count_out);
}

// Picks the kernel by size (in 112 KiB tiles), as the scans do: up to half a tile per SM single 56
// KiB sub-tiles on twice the SMs, up to one wave 112 KiB tiles, beyond it the pipeline.
template <typename T, int MODE>
bool launch_mode(uint64_t tiles, cudaStream_t s, bool bulk, const T* in, T* out, uint64_t n,
                 PredDev<T> p, TileStatus<uint64_t> ts, const unsigned long long* nt,
                 unsigned long long* count_out, uint32_t* counters) {
    const uint64_t sms = device_info().sm_count;
    if (!bulk) return launch_tiles<T, MODE, false, kSub>(n, s, in, out, p, ts, nt, count_out);
    if (tiles <= sms / 2)
        return launch_tiles<T, MODE, true, 1>(n, s, in, out, p, ts, nt, count_out);
    if (tiles <= 2 * sms)
        return launch_tiles<T, MODE, true, kSub>(n, s, in, out, p, ts, nt, count_out);
    constexpr size_t smem = PipeShape<T>::SMEM;
    if (!smem_opt_in<k_compact_pipe<T, MODE>>(smem))
        return cuda_ok(cudaGetLastError(), "k_compact_pipe shared-memory opt-in");
    const uint64_t pipe_tiles = (n + PipeShape<T>::TILE - 1) / PipeShape<T>::TILE;
    return launch_dependent(k_compact_pipe<T, MODE>, (unsigned)(pipe_tiles < sms ? pipe_tiles : sms),
                            kPipeBlock, smem, s, "k_compact_pipe launch", in, out, n,
                            (uint32_t)pipe_tiles, p, ts, nt, count_out, counters);
}

template <typename T>
bool compact_typed(Workspace& ws, CompactMode mode, const Pred& pr, const void* d_in,
                   void* d_out, uint64_t n, uint64_t* d_count) {
    constexpr int TILE = Shape<T>::TILE;
    const uint64_t tiles = (n + TILE - 1) / TILE;
    // both kernels' tiles: the smaller ones decide the size of the status array
    const uint64_t status_tiles = (n + PipeShape<T>::TILE - 1) / PipeShape<T>::TILE;
    static_assert(PipeShape<T>::TILE <= TILE, "status entries for either kernel");
    if (status_tiles > 0x7fffffffull) {
        set_error(PARALLAX_ERR_INVALID_ARGUMENT, "compaction: too many elements");
        return false;
    }
    char* scratch = ws.scratch(status_tiles);
    if (!scratch) return false;
    auto* nt = reinterpret_cast<unsigned long long*>(scratch + ScratchOff::num_true);
    if (pr.kind == PredKind::FLAGS && (!pr.flags || reinterpret_cast<uintptr_t>(pr.flags) % 4)) {
        set_error(PARALLAX_ERR_INVALID_ARGUMENT, "compaction: flags array missing or unaligned");
        return false;
    }
    if (mode == CompactMode::PARTITION) {
        // count pass: k = |{i : pred(in[i])}| into device scratch
        const bool ok = pr.kind == PredKind::FLAGS
            ? launch_count_flags(ws, pr.flags, n, reinterpret_cast<uint64_t*>(nt))
            : launch_count_if(ws, dtype_of<T>(), pr, d_in, n, reinterpret_cast<uint64_t*>(nt));
        if (!ok) return false;
    }
    auto ts = tile_status_at<uint64_t>(scratch, ws.next_epoch(), &ws.d_slot->spin_error, status_tiles);
    // bulk copies only from HBM; the page-locked host mirror (small coherent operands,
    // whole-heap capture) takes plain loads
    const bool bulk = reinterpret_cast<uintptr_t>(d_in) % 16 == 0 && !arena_contains(d_in);
    const T* in = static_cast<const T*>(d_in);
    T* out = static_cast<T*>(d_out);
    auto* cnt_out = reinterpret_cast<unsigned long long*>(d_count);
    PredDev<T> p = make_pred<T>(pr);
    uint32_t* counters = reinterpret_cast<uint32_t*>(scratch + ScratchOff::counters);
    cudaStream_t s = ws.stream();
    // profile bytes: input read (+ the kept elements written, known only on the device)
    ProfScope prof(ws, mode == CompactMode::PARTITION ? "k_partition"
                       : mode == CompactMode::UNIQUE ? "k_unique" : "k_copy_if",
                   (mode == CompactMode::PARTITION ? 2 : 1) * n * sizeof(T));
    bool ok = false;
    switch (mode) {
        case CompactMode::SELECT:
            ok = launch_mode<T, 0>(tiles, s, bulk, in, out, n, p, ts, nt, cnt_out, counters);
            break;
        case CompactMode::UNIQUE:
            ok = launch_mode<T, 1>(tiles, s, bulk, in, out, n, p, ts, nt, cnt_out, counters);
            break;
        case CompactMode::PARTITION:
            ok = launch_mode<T, 2>(tiles, s, bulk, in, out, n, p, ts, nt, cnt_out, counters);
            break;
    }
    if (!ok) return false;
    count_launch();
    return cuda_ok(cudaGetLastError(), "k_compact launch");
}

}  // namespace

bool launch_compact(Workspace& ws, DType t, CompactMode mode, const Pred& p, const void* d_in,
                    void* d_out, size_t n, uint64_t* d_count) {
    switch (t) {
        case DType::F32: return compact_typed<float>(ws, mode, p, d_in, d_out, n, d_count);
        case DType::F64: return compact_typed<double>(ws, mode, p, d_in, d_out, n, d_count);
        case DType::I32: return compact_typed<int32_t>(ws, mode, p, d_in, d_out, n, d_count);
        case DType::I64: return compact_typed<int64_t>(ws, mode, p, d_in, d_out, n, d_count);
        case DType::U32: return compact_typed<uint32_t>(ws, mode, p, d_in, d_out, n, d_count);
        case DType::U64: return compact_typed<uint64_t>(ws, mode, p, d_in, d_out, n, d_count);
        default: break;
    }
    set_error(PARALLAX_ERR_INVALID_ARGUMENT, "compaction: unsupported element type");
    return false;
}

}  // namespace pxb
