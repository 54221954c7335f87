// Single-pass inclusive / exclusive '+' scan.
//
// Reference: block Hillis-Steele scan (8 rounds, 2 barriers each) + recursive scan of the
// block sums + an add-offsets pass, each a separate dispatch with a fence wait
// (src/kernel/kernel_launcher.cpp:1280-1342, shaders/scan.comp:16-35,
// shaders/scan_add.comp:14-19); exclusive adds a shift pass writing
// out[i] = init + incl[i-1] (kernel_launcher.cpp:1346-1475).
//
// Here: one launch. 16-byte-aligned device operands of more than a wave of tiles go through a
// persistent pipeline, one warp-specialised CTA per SM (k_scan_pipe): tiles are bulk-loaded
// (cp.async.bulk) into a ring of buffers, summed and published as they land, looked back
// (lookback.cuh) while later tiles load, scanned in place and bulk-stored. Smaller ones, operands
// that are not aligned or lie in the host mirror, scans whose copies overlap their tiles, and the
// allocation-free entry point take one 512-thread CTA per 112 KiB (smallest arrays: 56 KiB) tile
// (two per SM), in blockIdx order (k_scan): stage, sum, look back, rescan, store.
// Rows are 28 (4-byte) or 14 (8-byte) consecutive elements per thread (112 bytes, an odd number
// of 16-byte words: conflict-free 128-bit shared loads).
// HBM traffic is the algorithmic minimum: n*s read + n*s written.
// Accumulation: fp32 data is scanned per thread in fp32 (28 terms per sub-tile) and carried
// across threads, warps and tiles in fp64; integers wrap around in their unsigned type.
#include <stdint.h>
#include <string.h>

#include <mutex>

#include "../lookback.cuh"
#include "../pdl.cuh"
#include "../runtime.hpp"
#include "../tiles.cuh"
#include "../tma.cuh"

namespace pxb {
namespace {

// Tile shape, chosen by measurement on B200 (2^28 elements): 112 KiB tiles at two CTAs per
// SM beat 48 KiB tiles at four per SM by 8-10 % (the look-back's fixed latency is paid per
// tile), and 16 KiB or 80 KiB tiles were slower still.
// The shape can be overridden at build time (PXB_SCAN_BLOCK / _VPT / _SUB / _CTAS) to sweep
// it; kSub x (kBlock / 32) must be 32.
#ifndef PXB_SCAN_BLOCK
#define PXB_SCAN_BLOCK 512
#endif
#ifndef PXB_SCAN_VPT
#define PXB_SCAN_VPT 7
#endif
#ifndef PXB_SCAN_SUB
#define PXB_SCAN_SUB 2
#endif
#ifndef PXB_SCAN_CTAS
#define PXB_SCAN_CTAS 2
#endif
constexpr int kBlock = PXB_SCAN_BLOCK;
constexpr int kVpt = PXB_SCAN_VPT;  // 16-byte vectors per thread; odd => conflict-free row reads
constexpr int kCtasPerSm = PXB_SCAN_CTAS;

template <typename T> struct ScanTypes;
template <> struct ScanTypes<float> { using L = float; using A = double; };
template <> struct ScanTypes<double> { using L = double; using A = double; };
template <> struct ScanTypes<int32_t> { using L = uint32_t; using A = uint32_t; };
template <> struct ScanTypes<uint32_t> { using L = uint32_t; using A = uint32_t; };
template <> struct ScanTypes<int64_t> { using L = uint64_t; using A = uint64_t; };
template <> struct ScanTypes<uint64_t> { using L = uint64_t; using A = uint64_t; };

constexpr int kSub = PXB_SCAN_SUB;  // sub-tiles per look-back tile; kSub x warps = 32 lanes

template <typename T>
struct ScanShape {
    static constexpr int V = 16 / sizeof(T);
    static constexpr int ITEMS = kVpt * V;          // elements per thread per sub-tile
    static constexpr int SUB = kBlock * ITEMS;      // 56 KiB sub-tile
    static constexpr int TILE = kSub * SUB;         // 112 KiB look-back tile
    static constexpr size_t SMEM = TILE * sizeof(T);
};

// Phase 1 sums each thread's 112-byte row of every sub-tile as soon as that sub-tile lands;
// one 32-lane scan over the (sub-tile, warp) totals - in element order - gives every
// warp's offset and the tile aggregate; warp 0 runs the look-back. Phase 2 re-reads each
// row from shared memory, scans it and writes the results in place. The caller has
// staged the tile (bulk part arriving on bars[] with `parity`, ragged part filled) and
// stores it afterwards.
template <typename T, bool EXCL, bool BULK, int NSUB>
__device__ __forceinline__ void scan_tile(T* buf, uint64_t* bars, uint32_t parity,
                                          typename ScanTypes<T>::A* s_tot, uint64_t tile,
                                          typename ScanTypes<T>::A init,
                                          const TileStatus<typename ScanTypes<T>::A>& ts,
                                          typename ScanTypes<T>::A* red, int* first,
                                          T* sub_out = nullptr, uint32_t bulk = 0) {
    using L = typename ScanTypes<T>::L;
    using A = typename ScanTypes<T>::A;
    constexpr int V = ScanShape<T>::V;
    constexpr int ITEMS = ScanShape<T>::ITEMS;
    constexpr int SUB = ScanShape<T>::SUB;
    constexpr int WARPS = kBlock / 32;
    static_assert(NSUB * WARPS <= 32, "one lane per (sub-tile, warp)");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // ---- phase 1: row totals of every sub-tile ----
    A tex[NSUB];  // exclusive prefix of this thread's row within its warp, per sub-tile
#pragma unroll
    for (int s = 0; s < NSUB; ++s) {
        if constexpr (BULK) wait_bar(&bars[s], parity, ts.err);
        const uint4* row = reinterpret_cast<const uint4*>(buf + s * SUB + tid * ITEMS);
        L sum = L(0);
#pragma unroll
        for (int v = 0; v < kVpt; ++v) {
            const uint4 r = row[v];
            const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
            for (int k = 0; k < V; ++k) sum = sum + (L)e[k];
        }
        const A incl = warp_inclusive_scan((A)sum, OpSum());
        const A ex = shfl_up(incl, 1);
        tex[s] = lane == 0 ? A(0) : ex;
        if (lane == 31) s_tot[s * WARPS + warp] = incl;
    }
    __syncthreads();
    // Every warp scans the 32 (sub-tile, warp) totals itself (identical shuffle sequence,
    // identical result), then the whole CTA runs the look-back.
    A woff[NSUB];  // offset of this warp's rows within the tile, per sub-tile
    A agg;
    {
        const A v = lane < NSUB * WARPS ? s_tot[lane] : A(0);
        const A vi = warp_inclusive_scan(v, OpSum());
        agg = shfl_idx(vi, 31);
        A vex = shfl_up(vi, 1);
        if (lane == 0) vex = A(0);
#pragma unroll
        for (int s = 0; s < NSUB; ++s) woff[s] = shfl_idx(vex, s * WARPS + warp);
    }
    const A prefix = lookback_cta<A, kBlock, true>(ts, tile, agg, red, first);

    // ---- phase 2: scan each row and write the results in place ----
#pragma unroll
    for (int s = 0; s < NSUB; ++s) {
        A tb = (prefix + woff[s]) + tex[s];
        if constexpr (EXCL) tb = init + tb;
        uint4* row = reinterpret_cast<uint4*>(buf + s * SUB + tid * ITEMS);
        L x[ITEMS];
#pragma unroll
        for (int v = 0; v < kVpt; ++v) {
            const uint4 r = row[v];
            const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
            for (int k = 0; k < V; ++k) x[v * V + k] = (L)e[k];
        }
#pragma unroll
        for (int j = 1; j < ITEMS; ++j) x[j] = x[j - 1] + x[j];
#pragma unroll
        for (int v = 0; v < kVpt; ++v) {
            uint4 r;
            T* e = reinterpret_cast<T*>(&r);
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const int j = v * V + k;
                if constexpr (EXCL) e[k] = (T)(j == 0 ? tb : tb + (A)x[j - 1]);
                else e[k] = (T)(tb + (A)x[j]);
            }
            row[v] = r;
        }
        if constexpr (BULK) {
            // with sub_out: each sub-tile's bulk store leaves as soon as the sub-tile is
            // written, so its shared-memory read overlaps the next sub-tile's rescan
            if (sub_out && s + 1 < NSUB) {
                fence_proxy_async_smem();
                __syncthreads();
                const uint32_t lo = (uint32_t)s * SUB, hi = bulk < lo + SUB ? bulk : lo + SUB;
                if (tid == 0 && hi > lo) {
                    bulk_store(sub_out + lo, buf + lo, (hi - lo) * (uint32_t)sizeof(T));
                    bulk_commit();
                }
            }
        }
    }
    if constexpr (BULK) fence_proxy_async_smem();
    __syncthreads();
    if constexpr (BULK) {
        if (sub_out) {
            const uint32_t lo = (uint32_t)(NSUB - 1) * SUB;
            if (tid == 0 && bulk > lo) {
                bulk_store(sub_out + lo, buf + lo, (bulk - lo) * (uint32_t)sizeof(T));
                bulk_commit();
            }
        }
    }
}

// One CTA per tile of NSUB 56 KiB sub-tiles, in blockIdx order: arrays of less than a wave,
// unaligned operands (BULK = false), scans that overlap their copies and the allocation-free entry
// point.
// `tile0` is the first tile of this launch: a scan launched in chunks (so its copies can
// overlap its tiles) passes each chunk's first tile, and every chunk shares one look-back
// epoch, so the first tile of a chunk looks back into the chunks before it.
// The look-back relies on in-order dispatch of the blocks; a wait that nonetheless never ends gives
// up after its poll limit with PARALLAX_ERR_DEVICE_SPIN. (A claim counter instead of blockIdx
// measured 5-8 % slower.)
template <typename T, bool EXCL, bool BULK, int NSUB>
__global__ void __launch_bounds__(kBlock, kCtasPerSm)
k_scan(const T* in, T* out, uint64_t n,  // in == out allowed (in-place ABI scan)
       typename ScanTypes<T>::A init, TileStatus<typename ScanTypes<T>::A> ts, uint64_t tile0) {
    using A = typename ScanTypes<T>::A;
    constexpr int SUB = ScanShape<T>::SUB;
    constexpr int TILE = NSUB * SUB;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* buf = reinterpret_cast<T*>(smem_raw);
    __shared__ __align__(8) uint64_t bars[NSUB];
    __shared__ A s_tot[32];
    __shared__ A s_red[kBlock / 32 + 1];
    __shared__ int s_first[kBlock / 32];
    const int tid = threadIdx.x;
    dependent_prologue();
    const uint64_t tile = tile0 + blockIdx.x;
    const uint64_t base = tile * (uint64_t)TILE;
    const uint64_t rem = n - base;
    const uint32_t cnt = rem < (uint64_t)TILE ? (uint32_t)rem : (uint32_t)TILE;
    const uint32_t bulk = stage_tile<T, SUB, NSUB, kBlock, BULK>(buf, bars, in, base, cnt);
    __syncthreads();
    scan_tile<T, EXCL, BULK, NSUB>(buf, bars, 0, s_tot, tile, init, ts, s_red, s_first,
                             BULK ? out + base : nullptr, bulk);
    for (uint32_t e = bulk + tid; e < cnt; e += kBlock) out[base + e] = buf[e];
    if constexpr (BULK) {
        if (tid == 0 && bulk) bulk_wait_read_all();
    }
}

// Persistent pipeline without CTA-wide barriers. Operands 16-byte aligned.
//   mover      claims a tile, bulk-loads it into a free buffer, bulk-stores it when every
//              scanning warp has written it, and reuses the buffer
//   sum warps  totals of the scanning warps' parts of a tile as soon as it lands; its aggregate
//              is published at once, whatever the CTA's earlier tiles still wait for
//   look-back  the tile's prefix: walk over earlier tiles, offset of every scanning warp
//   scan warps results, written in place
// What bounds it is HBM: at 2^28 fp32 / int32 elements 338 / 328 us (6.35 / 6.56 TB/s, 0.97 /
// 1.00 of a plain copy) against 422 / 407 for one CTA per 112 KiB tile, whose load, look-back and
// store follow one another. Its look-back is a chain through L2, so what matters is that a tile's
// aggregate never waits for anything but its own load (sums in the scan warps, behind the tile
// before: 3,500 us, each CTA in turn waiting for the others' queues) and that few polls meet at
// one L2 line (TileStatus). Measured on the fp32 scan, us: four 56 KiB buffers on one CTA 338,
// three 461, four 28 KiB buffers on two CTAs 348; sum warps 8 / 4 338 / 348; look-back warps 1 / 2
// 338 / 350; entries per lane and round of the walk 1 / 2 / 4 338 / 371 / 372.
constexpr int kPipeWarps = 16;   // scan warps
constexpr int kPipeStages = 4;   // tile buffers
constexpr int kSumWarps = 8;
constexpr int kPipeBlock = (kPipeWarps + kSumWarps + 2) * 32;

template <typename T>
struct PipeShape {
    static constexpr int V = 16 / sizeof(T);
    static constexpr int ITEMS = kVpt * V;
    static constexpr int TILE = kPipeWarps * 32 * ITEMS;
    static constexpr size_t SMEM = (size_t)kPipeStages * TILE * sizeof(T);
};

template <typename T, bool EXCL>
__global__ void __launch_bounds__(kPipeBlock, 1)
k_scan_pipe(const T* in, T* out, uint64_t n, uint32_t num_tiles,
            typename ScanTypes<T>::A init, TileStatus<typename ScanTypes<T>::A> ts,
            uint32_t* counters) {
    using L = typename ScanTypes<T>::L;
    using A = typename ScanTypes<T>::A;
    constexpr int V = PipeShape<T>::V, ITEMS = PipeShape<T>::ITEMS, TILE = PipeShape<T>::TILE;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* const bufs = reinterpret_cast<T*>(smem_raw);
    __shared__ __align__(8) uint64_t full[kPipeStages], added[kPipeStages], summed[kPipeStages],
        ready[kPipeStages], written[kPipeStages];
    __shared__ A s_tot[kPipeStages][kPipeWarps], s_off[kPipeStages][kPipeWarps], s_agg[kPipeStages];
    __shared__ uint32_t s_tile[kPipeStages];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < kPipeStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&added[s], kSumWarps);
            mbar_init(&summed[s], 1);
            mbar_init(&ready[s], 1);
            mbar_init(&written[s], kPipeWarps);
        }
        fence_mbar_init();
    }
    __syncthreads();
    dependent_prologue();
    auto count_of = [&](uint32_t t) {
        const uint64_t rem = n - (uint64_t)t * TILE;
        return rem < (uint64_t)TILE ? (uint32_t)rem : (uint32_t)TILE;
    };

    if (warp < kPipeWarps) {
        const uint32_t row0 = (uint32_t)tid * ITEMS;
        for (uint32_t it = 0;; ++it) {
            const uint32_t b = it % kPipeStages, ph = (it / kPipeStages) & 1u;
            wait_bar(&full[b], ph, ts.err);
            if (s_tile[b] >= num_tiles) break;
            uint4* row = reinterpret_cast<uint4*>(bufs + b * TILE + row0);
            L x[ITEMS];
#pragma unroll
            for (int v = 0; v < kVpt; ++v) {
                const uint4 r = row[v];
                const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
                for (int k = 0; k < V; ++k) x[v * V + k] = (L)e[k];
            }
#pragma unroll
            for (int j = 1; j < ITEMS; ++j) x[j] = x[j - 1] + x[j];
            A tex = shfl_up(warp_inclusive_scan((A)x[ITEMS - 1], OpSum()), 1);
            if (lane == 0) tex = A(0);
            wait_bar(&ready[b], ph, ts.err);
            A tb = s_off[b][warp] + tex;
            if constexpr (EXCL) tb = init + tb;
#pragma unroll
            for (int v = 0; v < kVpt; ++v) {
                uint4 r;
                T* e = reinterpret_cast<T*>(&r);
#pragma unroll
                for (int k = 0; k < V; ++k) {
                    const int j = v * V + k;
                    if constexpr (EXCL) e[k] = (T)(j == 0 ? tb : tb + (A)x[j - 1]);
                    else e[k] = (T)(tb + (A)x[j]);
                }
                row[v] = r;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&written[b]);
        }
    } else if (warp < kPipeWarps + kSumWarps) {
        const int sw = warp - kPipeWarps;
        for (uint32_t it = 0;; ++it) {
            const uint32_t b = it % kPipeStages, ph = (it / kPipeStages) & 1u;
            wait_bar(&full[b], ph, ts.err);
            const uint32_t t = s_tile[b];
            if (t >= num_tiles) break;
            const uint32_t cnt = count_of(t);
#pragma unroll
            for (int part = sw; part < kPipeWarps; part += kSumWarps) {
                const uint32_t row0 = (uint32_t)(part * 32 + lane) * ITEMS;
                const uint4* row = reinterpret_cast<const uint4*>(bufs + b * TILE + row0);
                L sum = L(0);
                if (cnt == (uint32_t)TILE) {
#pragma unroll
                    for (int v = 0; v < kVpt; ++v) {
                        const uint4 r = row[v];
                        const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
                        for (int k = 0; k < V; ++k) sum = sum + (L)e[k];
                    }
                } else {  // the last tile: what lies beyond the array counts as zero
                    for (int j = 0; j < ITEMS; ++j)
                        if (row0 + j < cnt) sum = sum + (L)bufs[b * TILE + row0 + j];
                }
                const A tot = warp_reduce((A)sum, OpSum());
                if (lane == 0) s_tot[b][part] = tot;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&added[b]);
            if (sw == 0) {
                wait_bar(&added[b], ph, ts.err);
                const A v = lane < kPipeWarps ? s_tot[b][lane] : A(0);
                const A vi = warp_inclusive_scan(v, OpSum());
                const A agg = shfl_idx(vi, 31);
                A vex = shfl_up(vi, 1);
                if (lane == 0) {
                    vex = A(0);
                    publish_aggregate(ts, t, agg);
                    s_agg[b] = agg;
                }
                if (lane < kPipeWarps) s_off[b][lane] = vex;
                __syncwarp();
                if (lane == 0) mbar_arrive(&summed[b]);
            }
        }
    } else if (warp == kPipeWarps + kSumWarps) {
        for (uint32_t it = 0;; ++it) {
            const uint32_t b = it % kPipeStages, ph = (it / kPipeStages) & 1u;
            wait_bar(&full[b], ph, ts.err);
            const uint32_t t = s_tile[b];
            if (t >= num_tiles) break;
            wait_bar(&summed[b], ph, ts.err);
            const A prefix = lookback_warp<A>(ts, t, s_agg[b]);
            if (lane < kPipeWarps) s_off[b][lane] = prefix + s_off[b][lane];
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[b]);
        }
    } else if (lane == 0) {
        auto load = [&](uint32_t b, uint32_t t) {
            s_tile[b] = t;
            if (t >= num_tiles) {
                mbar_arrive(&full[b]);
                return;
            }
            const uint64_t base = (uint64_t)t * TILE;
            const uint32_t cnt = count_of(t), bulk = bulk_elems<T>(cnt);
            T* const buf = bufs + b * TILE;
            for (uint32_t e = bulk; e < cnt; ++e) buf[e] = in[base + e];
            mbar_arrive_expect_tx(&full[b], bulk * (uint32_t)sizeof(T));
            if (bulk) bulk_load(buf, in + base, bulk * (uint32_t)sizeof(T), &full[b]);
        };
        // One claim at a time, so the CTAs' first tiles interleave: tiles claimed in a row would
        // be loaded in a row, and every other CTA's first look-back would wait for the last.
        for (uint32_t b = 0; b < kPipeStages; ++b) {
            if (b) wait_bar(&full[b - 1], 0, ts.err);
            load(b, atomicAdd(&counters[0], 1u));
        }
        for (uint32_t it = 0;; ++it) {
            const uint32_t b = it % kPipeStages;
            const uint32_t t = s_tile[b];
            if (t >= num_tiles) break;
            const uint32_t next = atomicAdd(&counters[0], 1u);
            wait_bar(&written[b], (it / kPipeStages) & 1u, ts.err);
            const uint64_t base = (uint64_t)t * TILE;
            const uint32_t cnt = count_of(t), bulk = bulk_elems<T>(cnt);
            const T* const buf = bufs + b * TILE;
            if (bulk) {
                bulk_store(out + base, buf, bulk * (uint32_t)sizeof(T));
                bulk_commit();
            }
            for (uint32_t e = bulk; e < cnt; ++e) out[base + e] = buf[e];
            bulk_wait_read_all();
            load(b, next);
        }
        persistent_exit(counters);
    }
}

// Launches tiles [tile0, tile0 + count).
template <typename T, bool EXCL, bool BULK, int NSUB = kSub>
bool launch_tiles_single(const T* in, T* out, uint64_t n, typename ScanTypes<T>::A init,
                         TileStatus<typename ScanTypes<T>::A> ts, uint64_t count,
                         cudaStream_t s, uint64_t tile0 = 0) {
    constexpr size_t smem = (size_t)NSUB * ScanShape<T>::SUB * sizeof(T);
    if (!smem_opt_in<k_scan<T, EXCL, BULK, NSUB>>(smem))
        return cuda_ok(cudaGetLastError(), "k_scan shared-memory opt-in");
    return launch_dependent(k_scan<T, EXCL, BULK, NSUB>, (unsigned)count, kBlock, smem, s, "k_scan launch",
                            in, out, n, init, ts, tile0);
}

template <typename T, bool EXCL>
bool launch_pipe(const T* in, T* out, uint64_t n, typename ScanTypes<T>::A init,
                 TileStatus<typename ScanTypes<T>::A> ts, uint32_t* counters, cudaStream_t s) {
    constexpr size_t smem = PipeShape<T>::SMEM;
    if (!smem_opt_in<k_scan_pipe<T, EXCL>>(smem))
        return cuda_ok(cudaGetLastError(), "k_scan_pipe shared-memory opt-in");
    const uint64_t tiles = (n + PipeShape<T>::TILE - 1) / PipeShape<T>::TILE;
    const uint64_t res = device_info().sm_count;
    return launch_dependent(k_scan_pipe<T, EXCL>, (unsigned)(tiles < res ? tiles : res), kPipeBlock, smem,
                            s, "k_scan_pipe launch", in, out, n, (uint32_t)tiles, init, ts, counters);
}

// Picks the kernel of an aligned device scan by its size (in 112 KiB tiles). Up to half a tile per
// SM: single 56 KiB sub-tiles, so twice the SMs share the work (synchronous call, 2^20 int32 / int64
// 16.4 -> 15.0 / 18.1 -> 15.8 us, 1000 fp32 15.1 -> 13.3). Up to one wave (two tiles per SM): all
// tiles are in flight at once anyway and the pipeline's start costs more than it saves (2^20 int32
// 17.4 us, 100,003 fp32 18.0 against 14.6). Beyond it the pipeline (16,000,001 fp32 41.9 -> 38.4).
template <typename T, bool EXCL>
bool launch_scan_tiles(const T* in, T* out, uint64_t n, typename ScanTypes<T>::A init,
                       TileStatus<typename ScanTypes<T>::A> ts, uint64_t tiles, bool bulk,
                       uint32_t* counters, cudaStream_t s) {
    if (!bulk) return launch_tiles_single<T, EXCL, false>(in, out, n, init, ts, tiles, s);
    const uint64_t sms = device_info().sm_count;
    if (tiles <= sms / 2) {
        const uint64_t subs = (n + ScanShape<T>::SUB - 1) / ScanShape<T>::SUB;
        return launch_tiles_single<T, EXCL, true, 1>(in, out, n, init, ts, subs, s);
    }
    if (tiles <= 2 * sms)
        return launch_tiles_single<T, EXCL, true>(in, out, n, init, ts, tiles, s);
    return launch_pipe<T, EXCL>(in, out, n, init, ts, counters, s);
}

template <typename T>
bool scan_typed(Workspace& ws, bool exclusive, const void* d_in, void* d_out, uint64_t n,
                const void* init_host) {
    using A = typename ScanTypes<T>::A;
    constexpr int TILE = ScanShape<T>::TILE;
    const uint64_t tiles = (n + TILE - 1) / TILE;
    if (n / PipeShape<T>::TILE >= 0x7fffffffull) {
        set_error(PARALLAX_ERR_INVALID_ARGUMENT, "scan: %llu elements exceed the grid limit",
                  (unsigned long long)n);
        return false;
    }
    // both kernels' tiles: the smaller ones decide the size of the status array
    const uint64_t status_tiles = (n + PipeShape<T>::TILE - 1) / PipeShape<T>::TILE;
    static_assert(PipeShape<T>::TILE <= TILE, "status entries for either kernel");
    char* scratch = ws.scratch(status_tiles);
    if (!scratch) return false;
    auto ts = tile_status_at<A>(scratch, ws.next_epoch(), &ws.d_slot->spin_error, status_tiles);
    A init = A(0);
    if (exclusive && init_host) {
        T v;
        memcpy(&v, init_host, sizeof(T));
        init = (A)v;
    }
    // bulk copies only between HBM and shared memory; operands in the page-locked host
    // mirror (small coherent operands, whole-heap capture) take the plain-load path
    const bool bulk = (reinterpret_cast<uintptr_t>(d_in) % 16 == 0) &&
                      (reinterpret_cast<uintptr_t>(d_out) % 16 == 0) &&
                      !arena_contains(d_in) && !arena_contains(d_out);
    const T* in = static_cast<const T*>(d_in);
    T* out = static_cast<T*>(d_out);
    cudaStream_t s = ws.stream();
    ProfScope prof(ws, exclusive ? "k_scan_exclusive" : "k_scan_inclusive", 2 * n * sizeof(T));
    uint32_t* counters = reinterpret_cast<uint32_t*>(scratch + ScratchOff::counters);
    const bool ok = exclusive
        ? launch_scan_tiles<T, true>(in, out, n, init, ts, tiles, bulk, counters, s)
        : launch_scan_tiles<T, false>(in, out, n, init, ts, tiles, bulk, counters, s);
    if (!ok) return false;
    count_launch();
    return cuda_ok(cudaGetLastError(), "k_scan launch");
}

// Scan of host arena operands with the copies interleaved with the tiles. The tiles are
// launched in chunks of kCopyChunkTiles on the workspace stream; chunk c's upload runs on
// the workspace's upload stream and chunk c's download on its download stream, ordered by
// events, so while the tiles of chunk c run, chunk c+1 is on its way up and chunk c-1 on its
// way down (the two copy directions run on separate copy engines). All chunks share one
// look-back epoch: the result is the same scan as one launch over every tile.
constexpr uint64_t kCopyChunkTiles = 296;  // two waves of two CTAs per SM: ~33 MB of fp32

template <typename T>
bool scan_copies_typed(Workspace& ws, bool exclusive, const void* h_in, const void* d_in,
                       void* h_out, void* d_out, uint64_t n, const void* init_host) {
    using A = typename ScanTypes<T>::A;
    constexpr int TILE = ScanShape<T>::TILE;
    const uint64_t tiles = (n + TILE - 1) / TILE;
    const bool bulk = (reinterpret_cast<uintptr_t>(d_in) % 16 == 0) &&
                      (reinterpret_cast<uintptr_t>(d_out) % 16 == 0);
    if (tiles > 0x7fffffffull || !bulk || !ws.copy_streams()) {
        cudaGetLastError();
        // one launch, copies before and after it
        cudaStream_t s = ws.stream();
        if (h_in && !arena_copy_async(const_cast<void*>(d_in), h_in, n * sizeof(T), true, s))
            return false;
        if (!scan_typed<T>(ws, exclusive, d_in, d_out, n, init_host)) return false;
        return !h_out || arena_copy_async(h_out, d_out, n * sizeof(T), false, s);
    }
    char* scratch = ws.scratch(tiles);
    if (!scratch) return false;
    auto ts = tile_status_at<A>(scratch, ws.next_epoch(), &ws.d_slot->spin_error, tiles);
    A init = A(0);
    if (exclusive && init_host) {
        T v;
        memcpy(&v, init_host, sizeof(T));
        init = (A)v;
    }
    const T* in = static_cast<const T*>(d_in);
    T* out = static_cast<T*>(d_out);
    cudaStream_t s = ws.stream();
    // On a failure part way, no copy may outlive the call: wait for both copy streams.
    auto fail = [&]() {
        cudaStreamSynchronize(ws.copy_up);
        cudaStreamSynchronize(ws.copy_down);
        cudaGetLastError();
        return false;
    };
    // the copy streams start after everything already queued on the workspace stream
    if (!cuda_ok(cudaEventRecord(ws.ev_copy[0], s), "copy event") ||
        !cuda_ok(cudaStreamWaitEvent(ws.copy_up, ws.ev_copy[0], 0), "copy wait") ||
        !cuda_ok(cudaStreamWaitEvent(ws.copy_down, ws.ev_copy[0], 0), "copy wait"))
        return fail();
    uint64_t chunks = 0;
    for (uint64_t t0 = 0; t0 < tiles; t0 += kCopyChunkTiles, ++chunks) {
        const uint64_t t1 = t0 + kCopyChunkTiles < tiles ? t0 + kCopyChunkTiles : tiles;
        const uint64_t e0 = t0 * TILE, e1 = t1 * TILE < n ? t1 * TILE : n;
        const size_t off = e0 * sizeof(T), bytes = (e1 - e0) * sizeof(T);
        if (h_in) {
            if (!arena_copy_async(const_cast<T*>(in) + e0, static_cast<const char*>(h_in) + off,
                                  bytes, true, ws.copy_up) ||
                !cuda_ok(cudaEventRecord(ws.ev_copy[1], ws.copy_up), "copy event") ||
                !cuda_ok(cudaStreamWaitEvent(s, ws.ev_copy[1], 0), "copy wait"))
                return fail();
        }
        const bool ok =
            exclusive ? launch_tiles_single<T, true, true>(in, out, n, init, ts, t1 - t0, s, t0)
                      : launch_tiles_single<T, false, true>(in, out, n, init, ts, t1 - t0, s, t0);
        if (!ok) return fail();
        if (h_out) {
            if (!cuda_ok(cudaEventRecord(ws.ev_copy[2], s), "copy event") ||
                !cuda_ok(cudaStreamWaitEvent(ws.copy_down, ws.ev_copy[2], 0), "copy wait") ||
                !arena_copy_async(static_cast<char*>(h_out) + off, out + e0, bytes, false,
                                  ws.copy_down))
                return fail();
        }
    }
    count_launch((unsigned)chunks);
    // the workspace stream (what a synchronous call waits on) ends after the last download
    if (!cuda_ok(cudaEventRecord(ws.ev_copy[3], ws.copy_down), "copy event") ||
        !cuda_ok(cudaStreamWaitEvent(s, ws.ev_copy[3], 0), "copy wait"))
        return fail();
    return cuda_ok(cudaGetLastError(), "k_scan launch");
}

}  // namespace

bool launch_scan_copies(Workspace& ws, DType t, bool exclusive, const void* h_in,
                        const void* d_in, void* h_out, void* d_out, size_t n,
                        const void* init_host) {
    switch (t) {
        case DType::F32:
            return scan_copies_typed<float>(ws, exclusive, h_in, d_in, h_out, d_out, n, init_host);
        case DType::F64:
            return scan_copies_typed<double>(ws, exclusive, h_in, d_in, h_out, d_out, n, init_host);
        case DType::I32:
            return scan_copies_typed<int32_t>(ws, exclusive, h_in, d_in, h_out, d_out, n, init_host);
        case DType::I64:
            return scan_copies_typed<int64_t>(ws, exclusive, h_in, d_in, h_out, d_out, n, init_host);
        case DType::U32:
            return scan_copies_typed<uint32_t>(ws, exclusive, h_in, d_in, h_out, d_out, n, init_host);
        case DType::U64:
            return scan_copies_typed<uint64_t>(ws, exclusive, h_in, d_in, h_out, d_out, n, init_host);
        default: break;
    }
    set_error(PARALLAX_ERR_INVALID_ARGUMENT, "scan: unsupported element type");
    return false;
}

bool launch_scan(Workspace& ws, DType t, bool exclusive, const void* d_in, void* d_out, size_t n,
                 const void* init_host) {
    switch (t) {
        case DType::F32: return scan_typed<float>(ws, exclusive, d_in, d_out, n, init_host);
        case DType::F64: return scan_typed<double>(ws, exclusive, d_in, d_out, n, init_host);
        case DType::I32: return scan_typed<int32_t>(ws, exclusive, d_in, d_out, n, init_host);
        case DType::I64: return scan_typed<int64_t>(ws, exclusive, d_in, d_out, n, init_host);
        case DType::U32: return scan_typed<uint32_t>(ws, exclusive, d_in, d_out, n, init_host);
        case DType::U64: return scan_typed<uint64_t>(ws, exclusive, d_in, d_out, n, init_host);
        default: break;
    }
    set_error(PARALLAX_ERR_INVALID_ARGUMENT, "scan: unsupported element type");
    return false;
}

// One scan tile launched as tile 1 of a fresh look-back epoch: tile 0 never publishes in
// that epoch, so the tile's look-back wait can only end by giving up after `polls` polls.
int check_bounded_wait(uint32_t polls) {
    using T = int32_t;
    using A = ScanTypes<T>::A;
    constexpr uint64_t TILE = ScanShape<T>::TILE;
    Workspace* ws = workspace();
    if (!ws) {
        set_error(PARALLAX_ERR_NO_DEVICE, "parallax_check_bounded_wait: no CUDA device");
        return PARALLAX_ERR_NO_DEVICE;
    }
    char* scratch = ws->scratch(2);
    T* buf = static_cast<T*>(ws->temp(2 * TILE * sizeof(T) * 2));
    if (!scratch || !buf) return last_error();
    cudaStream_t s = ws->stream();
    if (!cuda_ok(cudaMemsetAsync(buf, 0, 2 * TILE * sizeof(T), s), "check_bounded_wait: input"))
        return PARALLAX_ERR_CUDA;
    auto ts = tile_status_at<A>(scratch, ws->next_epoch(), &ws->d_slot->spin_error, 2);
    ts.limit = polls;
    if (!launch_tiles_single<T, false, true>(buf, buf + 2 * TILE, 2 * TILE, A(0), ts, 1, s, 1))
        return last_error() ? last_error() : PARALLAX_ERR_CUDA;
    count_launch();
    return sync_stream(*ws);
}

}  // namespace pxb

PXB_EXPORT int parallax_check_bounded_wait(uint32_t polls) {
    pxb::set_ok();
    if (polls == 0 || polls > pxb::kSpinLimit) {
        pxb::set_error(PARALLAX_ERR_INVALID_ARGUMENT,
                       "parallax_check_bounded_wait: polls must be in [1, %u]", pxb::kSpinLimit);
        return PARALLAX_ERR_INVALID_ARGUMENT;
    }
    return pxb::check_bounded_wait(polls);
}

// ---- allocation-free scan -----------------------------------------------------------------
// Some callers cannot allocate device memory at all: code that runs inside an allocation
// hook (a malloc / operator new interposer that routes the heap into the arena would
// re-enter itself if the runtime allocated), or a process whose device memory has been
// handed to its own pool. parallax_scan_noalloc gives them the single-pass scan with no
// allocation by the runtime: the look-back status lives in the fixed static device array
// below (384.25 KiB, held on every GPU that loads this library until the process exits),
// the caller passes device buffers for input and output and a stream, and no workspace,
// stream, event or pinned slot is created.
namespace pxb {
namespace {

constexpr uint64_t kNoAllocTiles = 24576;  // look-back status entries
constexpr size_t kNoAllocBytes = 256 + kNoAllocTiles * sizeof(StatusEntry);
// [0, 4): in-kernel wait-timeout code; [256, ...): look-back status entries. Static device
// memory starts zeroed; later calls find stale entries from older epochs, which read as
// "not ready", so only the timeout code is cleared per call.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kNoAllocMaxDevices = 64;
struct NoAllocDevice {
    bool ready = false;
    char* scratch = nullptr;  // device address of g_noalloc_scratch on that device
    uint32_t epoch = 0;
};
std::mutex g_noalloc_mu;
NoAllocDevice g_noalloc[kNoAllocMaxDevices];

template <typename T>
uint64_t noalloc_max_elements() {
    return kNoAllocTiles * (uint64_t)ScanShape<T>::TILE;
}

template <typename T>
bool noalloc_launch(const void* d_in, void* d_out, uint64_t n, const void* init_host,
                    cudaStream_t s, char* scratch, uint32_t epoch) {
    using A = typename ScanTypes<T>::A;
    constexpr int TILE = ScanShape<T>::TILE;
    const uint64_t tiles = (n + TILE - 1) / TILE;
    TileStatus<A> ts;
    ts.e = reinterpret_cast<StatusEntry*>(scratch + 256);
    ts.epoch = epoch;
    ts.err = reinterpret_cast<int32_t*>(scratch);
    // a line per entry as long as the fixed array holds them
    ts.shift = tiles << kStatusLineShift <= kNoAllocTiles ? kStatusLineShift : 0u;
    A init = A(0);
    if (init_host) {
        T v;
        memcpy(&v, init_host, sizeof(T));
        init = (A)v;
    }
    const bool bulk = (reinterpret_cast<uintptr_t>(d_in) % 16 == 0) &&
                      (reinterpret_cast<uintptr_t>(d_out) % 16 == 0);
    const T* in = static_cast<const T*>(d_in);
    T* out = static_cast<T*>(d_out);
    bool ok;
    if (init_host) {
        ok = bulk ? launch_tiles_single<T, true, true>(in, out, n, init, ts, tiles, s)
                  : launch_tiles_single<T, true, false>(in, out, n, init, ts, tiles, s);
    } else {
        ok = bulk ? launch_tiles_single<T, false, true>(in, out, n, init, ts, tiles, s)
                  : launch_tiles_single<T, false, false>(in, out, n, init, ts, tiles, s);
    }
    if (!ok) return false;
    count_launch();
    return cuda_ok(cudaGetLastError(), "parallax_scan_noalloc launch");
}

}  // namespace
}  // namespace pxb

using namespace pxb;

PXB_EXPORT int parallax_scan_noalloc(parallax_kernel_t scan_kernel, const void* input,
                                     void* output, size_t count, size_t elem_size,
                                     const void* init, void* cuda_stream) {
    set_ok();
    Handle* h = as_handle(scan_kernel);
    if (!h || h->kind != Kind::SCAN) {
        set_error(PARALLAX_ERR_INVALID_HANDLE, "parallax_scan_noalloc: not a scan kernel handle");
        return PARALLAX_ERR_INVALID_HANDLE;
    }
    if (dtype_size(h->dtype) != elem_size || !input || !output) {
        set_error(PARALLAX_ERR_INVALID_ARGUMENT,
                  "parallax_scan_noalloc: null buffer or elem_size %zu does not match the handle",
                  elem_size);
        return PARALLAX_ERR_INVALID_ARGUMENT;
    }
    if (count == 0) return PARALLAX_OK;
    uint64_t max_n = 0;
    switch (h->dtype) {
        case DType::F32: max_n = noalloc_max_elements<float>(); break;
        case DType::F64: max_n = noalloc_max_elements<double>(); break;
        case DType::I32: max_n = noalloc_max_elements<int32_t>(); break;
        case DType::I64: max_n = noalloc_max_elements<int64_t>(); break;
        case DType::U32: max_n = noalloc_max_elements<uint32_t>(); break;
        case DType::U64: max_n = noalloc_max_elements<uint64_t>(); break;
        default: break;
    }
    if (count > max_n) {
        set_error(PARALLAX_ERR_INVALID_ARGUMENT,
                  "parallax_scan_noalloc: %zu elements exceed its maximum of %llu for this "
                  "element type (%llu look-back tiles in a %zu-byte static array); use "
                  "parallax_scan or parallax_exclusive_scan",
                  count, (unsigned long long)max_n, (unsigned long long)kNoAllocTiles,
                  kNoAllocBytes);
        return PARALLAX_ERR_INVALID_ARGUMENT;
    }
    int dev = 0;
    if (!cuda_ok(cudaGetDevice(&dev), "parallax_scan_noalloc: cudaGetDevice"))
        return PARALLAX_ERR_CUDA;
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        set_error(PARALLAX_ERR_UNSUPPORTED, "parallax_scan_noalloc: device %d out of range", dev);
        return PARALLAX_ERR_UNSUPPORTED;
    }
    cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
    char* scratch = nullptr;
    uint32_t epoch = 0;
    {
        std::lock_guard<std::mutex> g(g_noalloc_mu);
        NoAllocDevice& d = g_noalloc[dev];
        if (!d.ready) {
            // Once per device, with that device current. The name of a __device__ array is
            // a host-side stand-in in host code; only this address reaches the kernel.
            void* p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess || !p) {
                cuda_ok(e == cudaSuccess ? cudaErrorInvalidSymbol : e,
                        "parallax_scan_noalloc: cudaGetSymbolAddress");
                return PARALLAX_ERR_CUDA;
            }
            d.scratch = static_cast<char*>(p);
            d.epoch = 0;
            d.ready = true;
        }
        if (++d.epoch >= (1u << 30)) {  // epoch wrap: stale words could alias, clear them
            if (!cuda_ok(cudaMemsetAsync(d.scratch + 256, 0, kNoAllocBytes - 256, s),
                         "parallax_scan_noalloc: clear status"))
                return PARALLAX_ERR_CUDA;
            d.epoch = 1;
        }
        scratch = d.scratch;
        epoch = d.epoch;
    }
    if (!cuda_ok(cudaMemsetAsync(scratch, 0, sizeof(int32_t), s),
                 "parallax_scan_noalloc: clear timeout code"))
        return PARALLAX_ERR_CUDA;
    bool ok = false;
    switch (h->dtype) {
        case DType::F32: ok = noalloc_launch<float>(input, output, count, init, s, scratch, epoch); break;
        case DType::F64: ok = noalloc_launch<double>(input, output, count, init, s, scratch, epoch); break;
        case DType::I32: ok = noalloc_launch<int32_t>(input, output, count, init, s, scratch, epoch); break;
        case DType::I64: ok = noalloc_launch<int64_t>(input, output, count, init, s, scratch, epoch); break;
        case DType::U32: ok = noalloc_launch<uint32_t>(input, output, count, init, s, scratch, epoch); break;
        case DType::U64: ok = noalloc_launch<uint64_t>(input, output, count, init, s, scratch, epoch); break;
        default: break;
    }
    if (!ok) return PARALLAX_ERR_CUDA;
    int32_t code = 0;
    if (!cuda_ok(cudaMemcpyAsync(&code, scratch, sizeof code, cudaMemcpyDeviceToHost, s),
                 "parallax_scan_noalloc: read timeout code") ||
        !cuda_ok(cudaStreamSynchronize(s), "parallax_scan_noalloc: stream synchronize"))
        return PARALLAX_ERR_CUDA;
    if (code) {
        set_error(PARALLAX_ERR_DEVICE_SPIN, "parallax_scan_noalloc: in-kernel wait gave up (%d)",
                  code);
        return PARALLAX_ERR_DEVICE_SPIN;
    }
    return PARALLAX_OK;
}
