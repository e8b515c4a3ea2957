// Depth-sorted alpha path and the radix sort, for sm_100a.
//
//   k_sp_project    sp_project (gps_splat.wgsl:737-777): 24-bit far-to-near key, quad record,
//                   GPS demand probe, plus the screen-tile rectangle of the splat.
//   radix_sort_pairs  stable LSD onesweep sort (replaces gps_sort.wgsl): one histogram pass for
//                   all digits, then one kernel per digit that ranks keys within each warp by
//                   peer groups (each lane ORs its bit into its digit's word of a per-warp row in
//                   shared memory and reads the word back, or ballots), resolves tile offsets by a decoupled
//                   lookback per digit and scatters. Digit width 4, 6 or 8 bits.
//   binning         (bin, splat id) entries in depth order, stably sorted by bin, give every screen bin
//                   its splats in depth order.
//   k_blend         one block per bin, front-to-back f32 blending with early termination
//                   (replaces the rgba16f back-to-front raster of gps_sorted_draw.wgsl:15-38 and the
//                   blend state of sorted.rs:125-138), written to accum = (rgb, 1) like sp_resolve.
//   k_composite     gps_composite.wgsl:41-55 into a headless RGBA8 buffer.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <mutex>

#include "../../include/gpsb200.h"
#include "devmath.cuh"
#include "sorted.h"
#include "pdl.cuh"

namespace gpsb {

typedef unsigned long long ull;

__device__ __forceinline__ uint32_t ld_relaxed32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed32(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ============================================================================ radix sort
constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
// Keys per thread of a onesweep pass, per digit width: 8-bit digits take 27 (6912 keys per tile, 54 KB of
// staging, 3 blocks per SM), whose longer digit runs write out in fuller sectors (2^24 pairs, three passes: 17
// keys 359 us, 23 355, 25 347, 27 343); 4- and 6-bit digits 15 (3840, 4 blocks per SM), where larger
// tiles gained nothing. Sorts of up to kRsSmallMax pairs take 8 (2048): large tiles would leave most SMs
// idle and make the few blocks' chains long (large / small tiles: 50k pairs 51 / 41 us, 400k 57 / 50,
// 560k 55 / 53, 800k 55 / 58, 2M 73 / 96).
#ifndef GPSB_SORT_IPT8
#define GPSB_SORT_IPT8 27
#endif
#ifndef GPSB_SORT_IPT
#define GPSB_SORT_IPT 15
#endif
constexpr int kRsIptSmall = 8;
constexpr uint32_t kRsSmallMax = 600u * 1024u;  // pairs; also bounds the tiles of the no-allocation scratch
template <int BITS>
constexpr int kRsIptLarge = BITS >= 8 ? GPSB_SORT_IPT8 : GPSB_SORT_IPT;
template <int BITS, int IPT>
struct RsShape {
    static constexpr int tile = kRsThreads * IPT;
    static constexpr size_t rows = (size_t)kRsWarps * (1 << BITS) * 8;
    static constexpr size_t stage = (size_t)tile * 8 > rows ? (size_t)tile * 8 : rows;  // dynamic shared memory of one block
    static constexpr int min_blocks = IPT >= 20 ? 3 : 4;
};
constexpr int kMaxPasses = 8;
#ifndef GPSB_SORT_LOOKAHEAD
#define GPSB_SORT_LOOKAHEAD 4
#endif
constexpr int kRsLook = GPSB_SORT_LOOKAHEAD;  // predecessor tiles read per lookback round trip
constexpr uint32_t kStAgg = 1u << 30, kStPre = 2u << 30, kStMask = (1u << 30) - 1u;
template <int BITS>
__global__ void __launch_bounds__(256) k_radix_hist(const uint32_t* __restrict__ keys, uint32_t n, int passes,
                                                    uint32_t* hist) {
    constexpr int BINS = 1 << BITS;
    __shared__ uint32_t s[kMaxPasses * BINS];
    for (int k = threadIdx.x; k < passes * BINS; k += blockDim.x) s[k] = 0;
    __syncthreads();
    grid_dependency_wait();
    launch_dependents();
    auto count = [&](uint32_t k) {
        for (int p = 0; p < passes; ++p) atomicAdd(&s[p * BINS + ((k >> (p * BITS)) & (BINS - 1))], 1u);
    };
    const uint32_t start = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    const uint32_t quads = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0 ? n / 4u : 0u;  // 16-byte loads where aligned
    for (uint32_t i = start; i < quads; i += step) {
        const uint4 k = __ldg(reinterpret_cast<const uint4*>(keys) + i);
        count(k.x);
        count(k.y);
        count(k.z);
        count(k.w);
    }
    for (uint32_t i = 4u * quads + start; i < n; i += step) count(__ldg(&keys[i]));
    __syncthreads();
    for (int k = threadIdx.x; k < passes * BINS; k += blockDim.x)
        if (s[k]) atomicAdd(&hist[k], s[k]);
}

// exclusive scan of every pass's histogram, in place: one block of BINS threads per pass (a single
// thread per pass took 8 us for 256 bins, a chain of dependent loads and stores; this takes 2 us)
template <int BITS>
__global__ void k_radix_hist_scan(uint32_t* hist) {
    grid_dependency_wait();
    launch_dependents();
    constexpr int BINS = 1 << BITS, WARPS = (BINS + 31) / 32;
    __shared__ uint32_t s_sum[WARPS];
    const int tid = threadIdx.x, lane = tid & 31;
    uint32_t* h = hist + blockIdx.x * BINS;
    const uint32_t c = tid < BINS ? h[tid] : 0u;
    uint32_t incl = c;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_sum[tid >> 5] = incl;
    __syncthreads();
    uint32_t base = 0;
    for (int w = 0; w < tid >> 5; ++w) base += s_sum[w];
    if (tid < BINS) h[tid] = base + incl - c;
}

// One digit pass over a tile: rank, scan, scatter into shared memory in digit order, lookback, write-out.
// Bound: shared-memory wavefronts (accesses by digit or by rank fall on the banks at random, 3 to 4 wavefronts
// each), so what counts is how many of them a key takes: the warps' and the tile's digit prefixes are one word,
// and the values follow the keys straight to their rank (their loads come back in one go, before the
// lookback). 2^24 pairs, 24-bit keys, three passes, the histogram and the scan: 335 us; with two prefixes,
// and with the values staged in input order by a bulk copy and fetched through each key's 16-bit
// input index: 388 us. A sort on its own launches its kernels with programmatic stream serialisation, so that
// a pass is resident, its rows cleared, when the one before it ends (50k pairs 42 -> 34 us, 560k 54 -> 47, 4M
// 122 -> 109). The sorts within a frame don't: frames one after another took 0.6 % longer.
// A pass reads what the one before it writes, so the read-only path is open to it only if that one lets it in
// after its last write. Large tiles do so (their dependents start when their blocks exit): plain loads cost them
// 3 to 8 % (2^24 pairs, copies of the input included: 373 us; plain loads and early dependents 398). Small tiles
// let theirs in at once and load plainly, which costs them nothing measurable (400k pairs: 57.5 us both ways).
// All of a thread's keys are loaded before the first is ranked, as no load passes the ranking's barriers.
template <int BITS, int IPT>
__global__ void __launch_bounds__(kRsThreads, RsShape<BITS, IPT>::min_blocks)
    k_onesweep(const uint32_t* kin, const uint32_t* vin, uint32_t* __restrict__ kout,
               uint32_t* __restrict__ vout, uint32_t n, int shift, const uint32_t* gstart, uint32_t* lookback,
               uint32_t* tile_counter, uint32_t* err) {
    constexpr int BINS = 1 << BITS;
    constexpr int kRsTile = RsShape<BITS, IPT>::tile;
    constexpr bool kEarly = IPT == kRsIptSmall;  // dependents start before this pass has written
    auto load = [](const uint32_t* p) { return kEarly ? *p : __ldg(p); };
    __shared__ uint32_t s_wpos[kRsWarps][BINS];  // each warp's digit counts, then the rank in the tile of its first key of a digit
    __shared__ uint32_t s_gbase[BINS];           // global position of the digit's first key of this tile, minus its rank
    // dynamic shared memory (RsShape::stage bytes): keys, then values, in digit order. Until the ranking ends
    // the warps' rows of peer masks lie in it.
    extern __shared__ __align__(16) uint32_t s_stage[];
    uint32_t* s_key = s_stage;
    uint32_t* s_val = s_stage + kRsTile;
    __shared__ uint32_t s_wsum[kRsWarps];
    __shared__ uint32_t s_tile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < kRsWarps * BINS; k += kRsThreads) s_stage[k] = (&s_wpos[0][0])[k] = 0u;
    grid_dependency_wait();
    if (kEarly) launch_dependents();
    if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const uint32_t t = s_tile;
    const uint32_t tile0 = t * kRsTile;
    const uint32_t tile_n = n - tile0 < (uint32_t)kRsTile ? n - tile0 : (uint32_t)kRsTile;
    const bool whole = tile_n == (uint32_t)kRsTile;
    const uint32_t base = tile0 + warp * 32 * IPT + lane;  // this lane's keys lie 32 apart from here
    uint32_t key[IPT], rank[IPT];
    const uint32_t lt = lanemask_lt();
    uint32_t* msk = s_stage + warp * BINS;
    uint32_t* cnts = s_wpos[warp];
    // rank every key within its warp's sub-tile in input order (stable). The lanes that hold one digit find
    // each other (peers) through shared memory (every lane ORs its bit into the digit's mask and reads the
    // word back; the lowest lane clears it) or, every third key, by one ballot per digit bit, which leaves the
    // shared-memory unit free. Then every lane reads its digit's running count of the warp, and the
    // lowest lane of each group adds the group's size (the groups hold distinct digits: no atomics).
    // 2^24 pairs: all OR 343 us, every third by ballots 335, every second 341, all 384.
    auto rank_key = [&](int q, uint32_t d, uint32_t live) {
        const bool mine = (live >> lane) & 1u;
        uint32_t peers;
        const bool vote = q % 3 == 2;
        if (vote) {
            peers = live;
#pragma unroll
            for (int k = 0; k < BITS; ++k) {
                const bool set = (d >> k) & 1u;
                const uint32_t m = __ballot_sync(0xffffffffu, set);
                peers &= set ? m : ~m;
            }
        } else {
            if (mine) atomicOr(&msk[d], 1u << lane);
            __syncwarp();
            peers = msk[d] & live;
        }
        const uint32_t below = __popc(peers & lt), old = cnts[d];
        __syncwarp();
        if (below == 0u && mine) {
            if (!vote) msk[d] = 0u;
            cnts[d] = old + (uint32_t)__popc(peers);
        }
        __syncwarp();  // orders this key's update before the next key's accesses
        rank[q] = old + below;
    };
    if (whole) {
#pragma unroll
        for (int q = 0; q < IPT; ++q) key[q] = load(kin + base + q * 32);
#pragma unroll
        for (int q = 0; q < IPT; ++q) rank_key(q, (key[q] >> shift) & (BINS - 1), 0xffffffffu);
    } else {
#pragma unroll
        for (int q = 0; q < IPT; ++q) key[q] = base + q * 32 < n ? load(kin + base + q * 32) : 0u;
#pragma unroll
        for (int q = 0; q < IPT; ++q) {
            const bool valid = base + q * 32 < n;
            rank_key(q, valid ? ((key[q] >> shift) & (BINS - 1)) : 0u, __ballot_sync(0xffffffffu, valid));
        }
    }
    __syncthreads();
    // per digit: exclusive prefix over warps and the tile count; publish the tile's aggregate early
    uint32_t* lb = lookback + (size_t)t * BINS;
    uint32_t cnt = 0, pre[kRsWarps];
    if (tid < BINS) {
#pragma unroll
        for (int w = 0; w < kRsWarps; ++w) {
            pre[w] = cnt;
            cnt += s_wpos[w][tid];

        }
        st_relaxed32(&lb[tid], (t == 0 ? kStPre : kStAgg) | cnt);
    }
    // exclusive scan of the digit counts over the tile (BINS <= 256 = one value per thread)
    uint32_t incl = tid < BINS ? cnt : 0u;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t a = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += a;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    uint32_t dstart = incl - cnt;
    for (int w = 0; w < warp; ++w) dstart += s_wsum[w];
    if (tid < BINS) {
#pragma unroll
        for (int w = 0; w < kRsWarps; ++w) s_wpos[w][tid] = dstart + pre[w];
    }
    __syncthreads();
    // scatter the keys into shared memory in digit order (stable), then fetch the values, which arrive during
    // the lookback
#pragma unroll
    for (int q = 0; q < IPT; ++q) {
        const uint32_t idx = base + q * 32;
        if (whole || idx < n) {
            rank[q] += cnts[(key[q] >> shift) & (BINS - 1)];
            s_key[rank[q]] = key[q];
            key[q] = load(vin + idx);
        }
    }
#pragma unroll
    for (int q = 0; q < IPT; ++q)
        if (whole || base + q * 32 < n) s_val[rank[q]] = key[q];
    // lookback per digit, kRsLook predecessors per round trip; an unpublished word is polled again
    if (tid < BINS) {
        uint32_t excl = 0;
        if (t > 0) {
            int32_t pred = (int32_t)t - 1;
            uint32_t spins = 0;
            bool failed = false;
            while (true) {
                uint32_t w[kRsLook];
#pragma unroll
                for (int u = 0; u < kRsLook; ++u)
                    w[u] = pred - u >= 0 ? ld_relaxed32(&lookback[(size_t)(pred - u) * BINS + tid]) : kStPre;
                int used = 0;
                bool done = false;
#pragma unroll
                for (int u = 0; u < kRsLook; ++u) {
                    if (done || used < u || (w[u] >> 30) == 0u) continue;
                    excl += w[u] & kStMask;
                    used = u + 1;
                    done = (w[u] >> 30) == 2u;
                }
                if (done) break;
                pred -= used;
                if (used < kRsLook) {
                    if (++spins > (1u << 22)) { failed = true; break; }
                    __nanosleep(32);
                }
            }
            if (failed) atomicOr(err, ERR_SORT_LOOKBACK);
            st_relaxed32(&lb[tid], kStPre | ((excl + cnt) & kStMask));
        }
        s_gbase[tid] = gstart[tid] + excl - dstart;
    }
    __syncthreads();
    // coalesced write-out: consecutive threads write consecutive keys of each digit run
    // (a position past n would mean corrupt histograms: it is skipped and reported once per thread)
    bool bad = false;
    auto write_one = [&](uint32_t i) {
        const uint32_t k = s_key[i];
        const uint32_t pos = s_gbase[(k >> shift) & (BINS - 1)] + i;
        const bool ok = pos < n;
        bad |= !ok;
        if (ok) {
            kout[pos] = k;
            vout[pos] = s_val[i];
        }
    };
    if (whole) {
#pragma unroll
        for (int q = 0; q < IPT; ++q) write_one((uint32_t)(q * kRsThreads + tid));
    } else {
        for (uint32_t i = tid; i < tile_n; i += kRsThreads) write_one(i);
    }
    if (bad) atomicOr(err, ERR_BAD_INDEX);
}

void radix_release(RadixScratch& s) {
    if (s.mem) cudaFree(s.mem);
    s = RadixScratch();
}

// Tiles of a sort of n pairs, and one onesweep pass over them; the staging lives in dynamic shared memory
// (above 48 KB for large tiles).
template <int BITS>
static uint32_t onesweep_tiles(uint32_t n) {
    const uint32_t tile = n <= kRsSmallMax ? RsShape<BITS, kRsIptSmall>::tile : RsShape<BITS, kRsIptLarge<BITS>>::tile;
    return (n + tile - 1) / tile;
}
template <int BITS, int IPT>
static void onesweep_launch_t(bool early, uint32_t tiles, const uint32_t* ik, const uint32_t* iv, uint32_t* ok, uint32_t* ov, uint32_t n,
                              int shift, const uint32_t* gstart, uint32_t* lookback, uint32_t* counter, uint32_t* err,
                              cudaStream_t st) {
    // set on every launch: the attributes belong to the current device's context
    constexpr size_t stage = RsShape<BITS, IPT>::stage;
    cudaFuncSetAttribute(k_onesweep<BITS, IPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stage);
    cudaFuncSetAttribute(k_onesweep<BITS, IPT>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    launch_pdl_if(early, k_onesweep<BITS, IPT>, dim3(tiles), dim3(kRsThreads), stage, st, ik, iv, ok, ov, n, shift, gstart, lookback,
               counter, err);
}
template <int BITS>
static void onesweep_launch(bool early, uint32_t tiles, const uint32_t* ik, const uint32_t* iv, uint32_t* ok, uint32_t* ov,
                            uint32_t n, int shift, const uint32_t* gstart, uint32_t* lookback, uint32_t* counter,
                            uint32_t* err, cudaStream_t st) {
    if (n <= kRsSmallMax)
        onesweep_launch_t<BITS, kRsIptSmall>(early, tiles, ik, iv, ok, ov, n, shift, gstart, lookback, counter, err, st);
    else
        onesweep_launch_t<BITS, kRsIptLarge<BITS>>(early, tiles, ik, iv, ok, ov, n, shift, gstart, lookback, counter, err, st);
}

template <int BITS>
static cudaError_t radix_impl(RadixScratch& s, uint32_t* ka, uint32_t* va, uint32_t* kb, uint32_t* vb, uint32_t n,
                              int key_bits, uint32_t* err, bool placed, bool early, cudaStream_t st) {
    constexpr int BINS = 1 << BITS;
    int passes = std::max(1, (key_bits + BITS - 1) / BITS);
    if (passes > kMaxPasses) return cudaErrorInvalidValue;
    const uint32_t tiles = onesweep_tiles<BITS>(n);
    // [digit histograms][tile counters][lookback words], cleared together
    constexpr size_t kCounterWords = 32;  // the lookback rows start on a 128-byte line
    const size_t hw = ((size_t)passes * BINS + 31) / 32 * 32,
                 words = hw + kCounterWords + (size_t)passes * std::max(tiles, 1u) * BINS;
    cudaError_t e;
    if (words * 4 > s.bytes) {
        // room for every smaller sort too, so that none of them allocates (it may be captured): just below the
        // line between the tile sizes there are more tiles than just above it
        const uint32_t most = std::max(tiles, onesweep_tiles<BITS>(std::min(n, kRsSmallMax)));
        const size_t room = (hw + kCounterWords + (size_t)passes * std::max(most, 1u) * BINS) * 4;
        if (s.mem) cudaFree(s.mem);
        s.mem = nullptr;
        s.bytes = 0;
        if ((e = cudaMalloc(&s.mem, room)) != cudaSuccess) return e;
        s.bytes = room;
    }
    uint32_t* hist = (uint32_t*)s.mem;
    uint32_t* counters = hist + hw;
    uint32_t* lookback = counters + kCounterWords;
    cudaMemsetAsync(hist, 0, words * 4, st);
    if (n == 0) return cudaGetLastError();
    // ping-pong so that the last pass writes (kb, vb)
    uint32_t *ik = ka, *iv = va, *ok = kb, *ov = vb;
    if (passes % 2 == 0) { ok = ka; ov = va; ik = kb; iv = vb; }
    launch_pdl_if(early, k_radix_hist<BITS>, dim3(std::min<uint32_t>((n + 4095) / 4096, 1184u)), dim3(256), 0, st, placed ? ik : ka, n, passes, hist);
    launch_pdl_if(early, k_radix_hist_scan<BITS>, dim3(passes), dim3(BINS < 32 ? 32 : BINS), 0, st, hist);
    if (passes % 2 == 0 && !placed) {
        // first pass reads the input from (ka, va): copy it to (kb, vb) so the parity works out
        cudaMemcpyAsync(kb, ka, (size_t)n * 4, cudaMemcpyDeviceToDevice, st);
        cudaMemcpyAsync(vb, va, (size_t)n * 4, cudaMemcpyDeviceToDevice, st);
    }
    for (int p = 0; p < passes; ++p) {
        onesweep_launch<BITS>(early, tiles, ik, iv, ok, ov, n, p * BITS, hist + p * BINS,
                              lookback + (size_t)p * tiles * BINS, counters + p, err, st);
        std::swap(ik, ok);
        std::swap(iv, ov);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------- no-allocation sort
// Callers that may not allocate device memory (a host application that owns the whole GPU memory
// budget through its own pool, or a real-time frame loop where a cudaMalloc would stall or is
// forbidden) use gpsb_sort_pairs_noalloc. Its scratch (digit histograms, tile counters and the
// lookback words) is this file-scope array, sized for kNoAllocMaxN pairs with up to 32-bit keys
// (4 passes of 8-bit digits): about 1.25 MB that every GPU which loads the library keeps until the
// process exits.
constexpr uint32_t kNoAllocMaxN = 1u << 21;
constexpr uint32_t kNoAllocTiles = (kNoAllocMaxN + RsShape<8, kRsIptLarge<8>>::tile - 1) / RsShape<8, kRsIptLarge<8>>::tile;
static_assert((kRsSmallMax + RsShape<8, kRsIptSmall>::tile - 1) / RsShape<8, kRsIptSmall>::tile <= kNoAllocTiles, "the no-allocation scratch holds the small tiles");
constexpr uint32_t kNoAllocPasses = 4;
constexpr size_t kNoAllocHistWords = kNoAllocPasses * 256;
constexpr size_t kNoAllocCounterWords = 16;  // per-pass tile counters (padded)
constexpr size_t kNoAllocWords = kNoAllocHistWords + kNoAllocCounterWords + (size_t)kNoAllocPasses * kNoAllocTiles * 256;
static __device__ __align__(256) uint32_t g_noalloc_sort_scratch[kNoAllocWords];

cudaError_t radix_sort_pairs(RadixScratch& s, uint32_t* ka, uint32_t* va, uint32_t* kb, uint32_t* vb, uint32_t n,
                             int key_bits, int digit_bits, uint32_t* err, cudaStream_t st, bool placed, bool early) {
    if (digit_bits == 4) return radix_impl<4>(s, ka, va, kb, vb, n, key_bits, err, placed, early, st);
    if (digit_bits == 6) return radix_impl<6>(s, ka, va, kb, vb, n, key_bits, err, placed, early, st);
    return radix_impl<8>(s, ka, va, kb, vb, n, key_bits, err, placed, early, st);
}

// Device address of g_noalloc_sort_scratch on the current device. In host code the array's name is
// only a host-side stand-in, so the address comes from cudaGetSymbolAddress with the device
// current. It is looked up again on every call whose stream is not capturing (so a device reset,
// which reloads the module, never leaves a stale address behind) and kept per device ordinal for
// calls made while `st` is being captured into a graph, which must follow one uncaptured call.
static void* noalloc_scratch_address(cudaStream_t st, cudaError_t* err, bool* capture_without_setup) {
    static std::mutex mu;
    static void* addr[256] = {};
    *capture_without_setup = false;
    int dev = 0;
    *err = cudaGetDevice(&dev);
    if (*err != cudaSuccess) return nullptr;
    if (dev < 0 || dev >= 256) {
        *err = cudaErrorInvalidDevice;
        return nullptr;
    }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    *err = cudaStreamIsCapturing(st, &cs);
    if (*err != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (cs == cudaStreamCaptureStatusNone) {
        void* p = nullptr;
        *err = cudaGetSymbolAddress(&p, g_noalloc_sort_scratch);
        if (*err != cudaSuccess) return nullptr;
        addr[dev] = p;
    } else if (!addr[dev]) {
        *capture_without_setup = true;
    }
    return addr[dev];
}

// ============================================================================ sorted path
constexpr uint64_t kBin64Pixels = 4ull << 20;  // frames from this size on may use 64 x 64 bins
constexpr ull kMaxEntries = 1ull << 30;        // of the entry lists
// Screen bins of the blend (tw x th pixels).
struct TileGeom {
    uint32_t tw, th, tiles_x, tiles_y;
};

__device__ __forceinline__ uint32_t rect_tiles(uint2 r) {
    if (r.x == 0xFFFFFFFFu) return 0u;
    uint32_t w = (r.y & 0xFFFFu) - (r.x & 0xFFFFu) + 1u, h = (r.y >> 16) - (r.x >> 16) + 1u;
    return w * h;
}
// the rectangle in bins of twice the size
__device__ __forceinline__ uint2 halved(uint2 r) { return make_uint2((r.x >> 1) & 0x7FFF7FFFu, (r.y >> 1) & 0x7FFF7FFFu); }
__device__ __forceinline__ uint2 coarser(uint2 r) { return r.x == 0xFFFFFFFFu ? r : halved(r); }
// Whether the frame's bins are doubled, from its numbers of entries with either size (decided on the device, where
// the depth sort's result is counted, and on the host alike). Larger bins have fewer entries to write and sort,
// but every region of 8 x 8 pixels tests four times the area's records: they win where splats cover several
// bins. Whole frame, 32 / 64 pixels, against the ratio of their entries: 6M splats at 3840x2160, 2.62 / 2.08 ms at
// 2.7 (distance 7), 2.42 / 2.02 at 2.36, 2.13 / 1.90 at 2.10, 1.64 / 2.09 at 1.85 (distance 20), 2.23 / 4.66 at
// 1.4 (distance 60); 560k at 2560x1700: 0.82 / 0.79 at 2.47, 0.84 / 0.84 at 2.18, 0.73 / 0.76 at 1.94, 0.54 / 0.66
// at 1.72. Frames below 4 Mpixel keep 32 pixels (560k at 1280x720, ratio 1.83: 0.44 / 0.51).
__host__ __device__ inline bool double_bins(const ull* entries) { return entries[0] > 2u * entries[1] || entries[0] > kMaxEntries; }

// sp_project (gps_splat.wgsl:737-777) + bin rectangle (kBoth: entries with bins of twice the size counted too)
template <bool kBoth>
__global__ void __launch_bounds__(128) k_sp_project(FrameConst f, TileGeom tg, const float4* __restrict__ splats,
                                                     const float* __restrict__ sh, uint32_t* keys, uint32_t* vals,
                                                     float4* rec, uint2* rect, ull* stats, ull* entries, int full) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    ull demand = 0;
    uint32_t bins = 0, bins2 = 0;  // bins of the splat's rectangle, and of twice the size; their sums size the entry lists
    if (i < f.N) {
        if (full) {
            keys[i] = 0xFFFFFFu;
            vals[i] = i;
            rect[i] = make_uint2(0xFFFFFFFFu, 0u);
        }
        float4 g0 = __ldg(&splats[4 * (size_t)i]), g1 = __ldg(&splats[4 * (size_t)i + 1]);
        float4 g2 = __ldg(&splats[4 * (size_t)i + 2]), g3 = __ldg(&splats[4 * (size_t)i + 3]);
        Proj pr = project(f, g0, g1, g2);
        float o = clamp_(g0.w, F_(0.0), F_(1.0));
        bool vis = pr.ok && o > F_(0.0);
        if (vis) {
            float ex = gxc::kOffscreenSigma * sqrt_(pr.a), ey = gxc::kOffscreenSigma * sqrt_(pr.c);
            vis = !(pr.mx + ex < F_(0.0) || pr.mx - ex >= (float)f.W || pr.my + ey < F_(0.0) || pr.my - ey >= (float)f.H);
        }
        if (vis) {
            float det = pr.a * pr.c - pr.b * pr.b;
            float en = f.density * (float)f.S * F_(2.0) * gxc::kPi * sqrt_(det) * dilog(o);
            if (en > F_(0.0)) demand = f2u(fmin_(en, F_(4.0e9)));
        }
        if (full && vis && !(o < gxc::kSpMinAlpha)) {
            float K = sqrt_(F_(2.0) * gx::log(div_(o, gxc::kSpMinAlpha)));
            float ex = K * sqrt_(pr.a), ey = K * sqrt_(pr.c);
            if (!(pr.mx + ex < F_(0.0) || pr.mx - ex >= (float)f.W || pr.my + ey < F_(0.0) || pr.my - ey >= (float)f.H)) {
                float tr2 = F_(0.5) * (pr.a + pr.c);
                float disc = sqrt_(fmax_(tr2 * tr2 - (pr.a * pr.c - pr.b * pr.b), F_(0.0)));
                float l1 = tr2 + disc;
                float l2 = fmax_(tr2 - disc, F_(1e-12));
                float v1x = F_(1.0), v1y = F_(0.0);
                if (fabsf(pr.b) > F_(1e-12)) {
                    float ux = l1 - pr.c, uy = pr.b;
                    float len = sqrt_(ux * ux + uy * uy);
                    v1x = div_(ux, len);
                    v1y = div_(uy, len);
                } else if (pr.a < pr.c) {
                    v1x = F_(0.0);
                    v1y = F_(1.0);
                }
                float v2x = -v1y, v2y = v1x;
                float s1 = sqrt_(l1), s2 = sqrt_(l2);
                rec[3 * (size_t)i] = make_float4(pr.mx, pr.my, o, K);
                rec[3 * (size_t)i + 1] = make_float4(div_(v1x, s1), div_(v1y, s1), div_(v2x, s2), div_(v2y, s2));
                rec[3 * (size_t)i + 2] = splat_colour(f, sh, i, g0, g3);
                keys[i] = 0xFFFFFEu - (f2b(pr.depth) >> 8u);
                // pixel-centre bounding box of the ellipse r2 <= K^2, padded, in tiles
                float bx = K * sqrtf(l1 * v1x * v1x + l2 * v2x * v2x) * 1.001f + 1.0f;
                float by = K * sqrtf(l1 * v1y * v1y + l2 * v2y * v2y) * 1.001f + 1.0f;
                float x0f = floorf(pr.mx - bx - 0.5f), x1f = ceilf(pr.mx + bx - 0.5f);
                float y0f = floorf(pr.my - by - 0.5f), y1f = ceilf(pr.my + by - 0.5f);
                if (x1f >= 0.0f && y1f >= 0.0f && x0f <= (float)(f.W - 1) && y0f <= (float)(f.H - 1)) {
                    uint32_t x0 = (uint32_t)fmaxf(x0f, 0.0f), y0 = (uint32_t)fmaxf(y0f, 0.0f);
                    uint32_t x1 = (uint32_t)fminf(x1f, (float)(f.W - 1)), y1 = (uint32_t)fminf(y1f, (float)(f.H - 1));
                    const uint2 r = make_uint2((x0 / tg.tw) | ((y0 / tg.th) << 16), (x1 / tg.tw) | ((y1 / tg.th) << 16));
                    rect[i] = r;
                    bins = rect_tiles(r);
                    if (kBoth) bins2 = rect_tiles(coarser(r));
                }
            }
        }
    }
    for (int o = 16; o; o >>= 1) demand += __shfl_xor_sync(0xffffffffu, demand, o);
    if constexpr (!kBoth) {
        if ((threadIdx.x & 31) == 0 && demand) atomicAdd(&stats[ST_PROBE], demand);
        if (full) {
            ull b = bins;
            for (int o = 16; o; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
            if ((threadIdx.x & 31) == 0 && b) atomicAdd(entries, b);
        }
    } else {
        // one addition per block: a third one per warp made a frame of 6M splats 6 % longer. A frame has at most
        // 2^25 bins (its accumulator bounds it), so a warp's fit 32 bits.
        __shared__ ull s_sum[3][4];
        const uint32_t b = __reduce_add_sync(0xffffffffu, bins), b2 = __reduce_add_sync(0xffffffffu, bins2);
        if ((threadIdx.x & 31) == 0) {
            s_sum[0][threadIdx.x >> 5] = demand;
            s_sum[1][threadIdx.x >> 5] = b;
            s_sum[2][threadIdx.x >> 5] = b2;
        }
        __syncthreads();
        if (threadIdx.x < 3u) {
            const ull* w = s_sum[threadIdx.x];
            const ull sum = w[0] + w[1] + w[2] + w[3];
            if (sum) atomicAdd(threadIdx.x ? entries + (threadIdx.x - 1u) : &stats[ST_PROBE], sum);
        }
    }
}

// ---- bin entries: for every splat in depth order, one (bin, splat id) pair per bin of its rectangle.
// A block takes kEbSplats sorted splats, a warp kEbSplats / 8 of them in groups of 32 (one per lane).
constexpr int kEbT = 256, kEbGroups = 8, kEbSplats = kEbT * kEbGroups;

// sorted position of group g of this thread
__device__ __forceinline__ uint32_t entry_splat(int g) {
    return blockIdx.x * kEbSplats + (threadIdx.x >> 5) * (32 * kEbGroups) + g * 32 + (threadIdx.x & 31);
}
__device__ __forceinline__ uint2 sorted_rect(const uint32_t* __restrict__ vals_sorted, const uint2* __restrict__ rect, uint32_t j,
                                             uint32_t n, bool twice) {
    const uint2 r = j < n ? rect[__ldg(&vals_sorted[j])] : make_uint2(0xFFFFFFFFu, 0u);  // unbinned splats have no rectangle
    return twice ? coarser(r) : r;
}

// entries of every block's splats; choose: the bins may be doubled, by the numbers of entries
__global__ void __launch_bounds__(kEbT) k_entry_sums(const uint32_t* __restrict__ vals_sorted, const uint2* __restrict__ rect,
                                                     const ull* entries, bool choose, uint32_t n, uint32_t* sums) {
    __shared__ uint32_t s[kEbT / 32];
    const bool twice = choose && double_bins(entries);
    uint32_t v = 0;
#pragma unroll
    for (int g = 0; g < kEbGroups; ++g) v += rect_tiles(sorted_rect(vals_sorted, rect, entry_splat(g), n, twice));
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < kEbT / 32; ++w) t += s[w];
        sums[blockIdx.x] = t;
    }
}
// single block: exclusive scan of the block sums, in place
__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t* sums, uint32_t nb) {
    __shared__ uint32_t s[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t base = 0;
    for (uint32_t b0 = 0; b0 < nb; b0 += 1024) {
        const uint32_t i = b0 + threadIdx.x, c = i < nb ? sums[i] : 0u;
        uint32_t incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = s[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += v;
            }
            s[lane] = w;  // inclusive over the warps
        }
        __syncthreads();
        if (i < nb) sums[i] = base + (warp ? s[warp - 1] : 0u) + incl - c;
        base += s[31];
        __syncthreads();
    }
}
// first entry of every sorted splat
__global__ void __launch_bounds__(kEbT) k_entry_offsets(const uint32_t* __restrict__ vals_sorted, const uint2* __restrict__ rect,
                                                        const uint32_t* __restrict__ sums, const ull* entries, bool choose, uint32_t n,
                                                        uint32_t* __restrict__ offs) {
    const bool twice = choose && double_bins(entries);
    __shared__ uint32_t s[kEbT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t c[kEbGroups], v = 0;
#pragma unroll
    for (int g = 0; g < kEbGroups; ++g) {
        c[g] = rect_tiles(sorted_rect(vals_sorted, rect, entry_splat(g), n, twice));
        v += c[g];
    }
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) s[warp] = v;
    __syncthreads();
    uint32_t base = sums[blockIdx.x];
    for (int w = 0; w < warp; ++w) base += s[w];
#pragma unroll
    for (int g = 0; g < kEbGroups; ++g) {
        uint32_t incl = c[g];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t a = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += a;
        }
        const uint32_t j = entry_splat(g);
        if (j < n) offs[j] = base + incl - c[g];
        base += __shfl_sync(0xffffffffu, incl, 31);
    }
}
// The entries. A warp writes kEwEntries consecutive ones, whatever the splats' sizes: it finds the
// first one's splat by a binary search in the offsets and steps on 32 entries at a time, the splats
// that begin within a step found by one bit per lane. (One thread per splat writing its entries one by
// one took 4.4 ms at 6M splats, 3840x2160, where some splats cover the whole frame; one warp per 32
// splats 0.85 ms, as the nearest splats, neighbours in depth order, are the largest.)
constexpr uint32_t kEwEntries = 512;
template <bool kTwice>
__global__ void __launch_bounds__(256) k_entries(const uint32_t* __restrict__ vals_sorted, const uint2* __restrict__ rect,
                                                 const uint32_t* __restrict__ offs, uint32_t n, uint32_t tiles_x, uint32_t m,
                                                 uint32_t* __restrict__ ekey, uint32_t* __restrict__ eval) {
    const uint32_t lane = threadIdx.x & 31u, upto = 0xFFFFFFFFu >> (31u - lane);
    auto bins_of = [&](uint32_t splat) { return kTwice ? halved(rect[splat]) : rect[splat]; };  // a splat with entries
    const uint32_t first = ((blockIdx.x * 256u + threadIdx.x) >> 5) * kEwEntries;
    if (first >= m) return;
    const uint32_t last = m - first < kEwEntries ? m : first + kEwEntries;
    // splat of entry `first`: the last j with offs[j] <= first (it has entries: the next offset is larger)
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1u) {
        const uint32_t step = (hi - lo + 31u) / 32u, idx = lo + (lane + 1u) * step;
        const uint32_t c = __popc(__ballot_sync(0xffffffffu, idx < hi && __ldg(&offs[idx]) <= first));
        const uint32_t nh = lo + (c + 1u) * step;
        lo += c * step;
        hi = nh < hi ? nh : hi;
    }
    uint32_t j = lo;
    uint32_t co = __ldg(&offs[j]), nx = j + 1u < n ? __ldg(&offs[j + 1u]) : m;
    uint32_t id = __ldg(&vals_sorted[j]);
    uint2 r = bins_of(id);
    for (uint32_t p = first; p < last; p += 32u) {
        uint32_t myid = id, o = co;
        uint2 mr = r;
        while (nx - p < 32u && nx < m) {  // splats that begin within the step, 32 candidates at a time
            const uint32_t jj = j + 1u + lane;
            const uint32_t of = jj < n ? __ldg(&offs[jj]) : m;
            const uint32_t d = of - p;
            // a splat without entries shares its offset with the next one: the last of equals counts
            const uint32_t nxt = __shfl_down_sync(0xffffffffu, of, 1);
            const uint32_t after = lane < 31u ? nxt : (jj + 1u < n ? __ldg(&offs[jj + 1u]) : m);
            const bool starts = jj < n && d < 32u && after > of;
            const uint32_t mask = __ballot_sync(0xffffffffu, starts);
            const uint32_t bits = __reduce_or_sync(0xffffffffu, starts ? 1u << d : 0u);
            uint32_t sid = 0;
            uint2 sr = make_uint2(0u, 0u);
            if (starts) {
                sid = __ldg(&vals_sorted[jj]);
                sr = bins_of(sid);
            }
            // the c-th starting splat of the mask serves this lane's entry
            const uint32_t c = __popc(bits & upto);
            uint32_t src = c - 1u;
            if (mask & (mask + 1u)) src = c ? __fns(mask, 0u, (int)c) : 0u;  // empty splats among them
            const uint32_t a = __shfl_sync(0xffffffffu, sid, src & 31u), b = __shfl_sync(0xffffffffu, of, src & 31u);
            const uint32_t rx = __shfl_sync(0xffffffffu, sr.x, src & 31u), ry = __shfl_sync(0xffffffffu, sr.y, src & 31u);
            if (c) {
                myid = a;
                o = b;
                mr = make_uint2(rx, ry);
            }
            // step on to the last splat that began here, or past 32 empty ones
            const uint32_t seen = __popc(__ballot_sync(0xffffffffu, jj < n && d < 32u));
            if (mask) {
                const uint32_t l = 31u - __clz(mask);
                id = __shfl_sync(0xffffffffu, sid, l);
                co = __shfl_sync(0xffffffffu, of, l);
                r = make_uint2(__shfl_sync(0xffffffffu, sr.x, l), __shfl_sync(0xffffffffu, sr.y, l));
            }
            j += seen;
            nx = j + 1u < n ? __ldg(&offs[j + 1u]) : m;
            if (seen < 32u) break;
        }
        const uint32_t pos = p + lane;
        if (pos < last) {
            const uint32_t t = pos - o, w = (mr.y & 0xFFFFu) - (mr.x & 0xFFFFu) + 1u, ty = t / w;
            ekey[pos] = ((mr.x >> 16) + ty) * tiles_x + (mr.x & 0xFFFFu) + (t - ty * w);
            eval[pos] = myid;
        }
        // p + 32 may fall on the next splat's first entry
        while (nx == p + 32u && nx < m) {
            ++j;
            co = nx;
            nx = j + 1u < n ? __ldg(&offs[j + 1u]) : m;
            if (nx > co) {
                id = __ldg(&vals_sorted[j]);
                r = bins_of(id);
            }
        }
    }
}

// first entry of every bin (bin b: [ranges[b], ranges[b + 1])): one warp each, a 32-ary search in the
// sorted keys
__global__ void __launch_bounds__(128) k_bin_ranges(const uint32_t* __restrict__ ekey, uint32_t m, uint32_t bins, uint32_t* ranges) {
    const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (b > bins) return;
    uint32_t lo = 0, n = m;  // the first position with key >= b lies in [lo, lo + n]
    while (n) {
        const uint32_t step = (n + 31u) / 32u, idx = lane * step;
        const uint32_t c = __popc(__ballot_sync(0xffffffffu, idx < n && __ldg(&ekey[lo + idx]) < b));
        if (c == 0u) break;
        // key[lo + (c - 1) step] < b, and key[lo + c step] >= b where that is within the range
        const uint32_t next = (c - 1u) * step + 1u, stop = c * step < n ? c * step : n;
        lo += next;
        n = stop - next;
    }
    if (lane == 0) ranges[b] = lo;
}

// Blending, nearest splats first, per pixel the arithmetic of one thread per pixel. One warp, a block of
// its own, per region of RW x RH pixels (8 x 8, two pixels a lane) of a screen bin: it reads the bin's
// entries 32 at a time, each lane tests one record against the region, and the warp steps only through
// those that can touch it. Bound: instruction issue and, at the end, the longest regions; warps
// of their own end by themselves and leave their place to the next.
// Measured (B200), 560k splats at 1280x720 with 32 x 32 bins: 8 x 8 regions 203 us, 16 x 8 279, 8 x 4 218;
// bins of 16 / 64 pixels 201 / 308 us, but more entries to sort, or longer lists to test; 6M splats at
// 3840x2160 with 64 x 64 bins: 1.19 ms, 1.22, 1.42. (A block per 16 x 16 tile with every record tested by
// every pixel: 340 us and 1.87 ms; blocks of 8 warps per 32 x 32 bin 430 us, waiting for their
// slowest warp.)
template <int RW, int RH>
__global__ void __launch_bounds__(32) k_blend(uint32_t W, uint32_t H, uint32_t tiles_x, uint32_t bw, uint32_t bh,
                                              uint32_t regions_x, const uint32_t* __restrict__ ranges,
                                              const uint32_t* __restrict__ eid, const float4* __restrict__ rec, float bg0,
                                              float bg1, float bg2, float4* accum) {
    constexpr int PX = RW * RH / 32, LH = 32 / RW;  // a lane's pixels are LH rows apart
    __shared__ float4 s_a[32], s_b[32], s_c[32];
    __shared__ __align__(8) float s_exp[gx::kExpNodes * 2];
    const int lane = threadIdx.x;
    for (int k = lane; k < gx::kExpNodes * 2; k += 32) s_exp[k] = gx::kExpTabD[k];
    const uint32_t rx = (blockIdx.x % regions_x) * RW, ry = (blockIdx.x / regions_x) * RH;
    const uint32_t tile = (ry / bh) * tiles_x + rx / bw;
    const uint32_t px = rx + (lane % RW), py = ry + (lane / RW);  // pixels (px, py + LH j)
    const float pcx = (float)px + F_(0.5);
    const float mcx = (float)rx + 0.5f * RW, mcy = (float)ry + 0.5f * RH;
    constexpr float hx = 0.5f * (RW - 1), hy = 0.5f * (RH - 1);
    float T[PX], cr[PX], cg[PX], cb[PX];
    bool live = false;
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        T[j] = px < W && py + LH * j < H ? F_(1.0) : F_(0.0);  // a pixel is done below 1e-4
        cr[j] = cg[j] = cb[j] = F_(0.0);
        live |= T[j] > F_(0.0);
    }
    const int begin = (int)ranges[tile];
    int end = (int)ranges[tile + 1];
    // the records of the next 32 entries and the ids of the 32 after them are on their way meanwhile
    float4 na, nb, nc;
    uint32_t nid = 0;
    auto fetch_id = [&](int e) { if (e - 1 - lane >= begin) nid = __ldg(&eid[e - 1 - lane]); };
    auto fetch = [&](int e) {
        if (e - 1 - lane >= begin) {
            na = __ldg(&rec[3 * (size_t)nid]);
            nb = __ldg(&rec[3 * (size_t)nid + 1]);
            nc = __ldg(&rec[3 * (size_t)nid + 2]);
        }
    };
    fetch_id(end);
    fetch(end);
    fetch_id(end - 32);
    for (; end > begin; end -= 32) {
        // can the record touch the region? |(u, v)| at its middle less the largest change of u and v over it
        // (and of their roundings) against K
        bool hit = false;
        if (end - 1 - lane >= begin) {
            const float dx = mcx - na.x, dy = mcy - na.y;
            const float ux = dx * nb.x, uy = dy * nb.y, vx = dx * nb.z, vy = dy * nb.w;
            const float eu = hx * fabsf(nb.x) + hy * fabsf(nb.y) + 1e-6f * (fabsf(ux) + fabsf(uy)) + 0.01f;
            const float ev = hx * fabsf(nb.z) + hy * fabsf(nb.w) + 1e-6f * (fabsf(vx) + fabsf(vy)) + 0.01f;
            const float u = fmaxf(fabsf(ux + uy) - eu, 0.0f), v = fmaxf(fabsf(vx + vy) - ev, 0.0f);
            hit = !(u * u + v * v > na.w * na.w * 1.001f);
        }
        uint32_t todo = __ballot_sync(0xffffffffu, hit);
        __syncwarp();
        if (hit) {
            s_a[lane] = na;
            s_b[lane] = nb;
            s_c[lane] = nc;
        }
        __syncwarp();
        fetch(end - 32);
        fetch_id(end - 64);
        while (todo) {
            const int q = __ffs(todo) - 1;
            todo &= todo - 1u;
            const float4 a = s_a[q], b = s_b[q];
            const float dx = pcx - a.x, ub = dx * b.x, vb = dx * b.z, kk = a.w * a.w;
            bool in[PX], any = false;
            float r2[PX];
#pragma unroll
            for (int j = 0; j < PX; ++j) {
                const float dy = ((float)(py + LH * j) + F_(0.5)) - a.y;
                const float u = ub + dy * b.y, v = vb + dy * b.w;
                r2[j] = u * u + v * v;
                in[j] = !(r2[j] > kk) && !(T[j] < F_(1e-4));
                any |= in[j];
            }
            if (!any) continue;
            const float4 c = s_c[q];
#pragma unroll
            for (int j = 0; j < PX; ++j) {
                if (!in[j]) continue;
                const float alpha = fmin_(a.z * gx::exp_mid(-F_(0.5) * r2[j], s_exp), F_(0.99));
                if (alpha < gxc::kSpMinAlpha) continue;
                const float wgt = T[j] * alpha;
                cr[j] = cr[j] + wgt * c.x;
                cg[j] = cg[j] + wgt * c.y;
                cb[j] = cb[j] + wgt * c.z;
                T[j] = T[j] * (F_(1.0) - alpha);
            }
        }
        live = false;
#pragma unroll
        for (int j = 0; j < PX; ++j) live |= !(T[j] < F_(1e-4));
        if (!__any_sync(0xffffffffu, live)) break;
    }
#pragma unroll
    for (int j = 0; j < PX; ++j)
        if (px < W && py + LH * j < H)
            accum[(size_t)(py + LH * j) * W + px] = make_float4(cr[j] + T[j] * bg0, cg[j] + T[j] * bg1, cb[j] + T[j] * bg2, F_(1.0));
}

void sorted_release(SortedState& s) {
    void* ptrs[] = {s.keys_a, s.vals_a, s.keys_b, s.vals_b, s.rec, s.tiles, s.sums, s.offs, s.total,
                    s.ent_key_a, s.ent_val_a, s.ent_key_b, s.ent_val_b, s.ranges};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (s.host_total) cudaFreeHost(s.host_total);
    if (s.counted) cudaEventDestroy(s.counted);
    radix_release(s.rs_keys);
    radix_release(s.rs_tiles);
    s = SortedState();
}

template <int RW, int RH>
static void blend_launch(const SortedState& s, const FrameConst& f, const TileGeom& tg, float4* accum, cudaStream_t st) {
    const uint32_t rx = (f.W + RW - 1) / RW, ry = (f.H + RH - 1) / RH;
    k_blend<RW, RH><<<rx * ry, 32, 0, st>>>(f.W, f.H, tg.tiles_x, tg.tw, tg.th, rx, (uint32_t*)s.ranges, (uint32_t*)s.ent_val_b,
                                            (float4*)s.rec, f.bg[0], f.bg[1], f.bg[2], accum);
}

cudaError_t sorted_render(SortedState& s, const FrameConst& f, const float4* splats, const float* sh, float4* accum,
                          unsigned long long* stats, uint32_t* err, uint32_t* launches, bool full, cudaStream_t st,
                          std::string* what) {
    const uint32_t n = f.N;
    cudaError_t e;
    if (n > s.cap_n) {
        s.cap_n = 0;  // nothing is usable until the last allocation has succeeded
        void** bufs[] = {&s.keys_a, &s.vals_a, &s.keys_b, &s.vals_b, &s.offs};
        for (void** b : bufs) {
            if (*b) cudaFree(*b);
            *b = nullptr;
            if ((e = cudaMalloc(b, (size_t)std::max(n, 1u) * 4 + 64)) != cudaSuccess) { *what = "sorted buffers"; return e; }
        }
        for (void** b : {&s.rec, &s.tiles, &s.sums}) {
            if (*b) cudaFree(*b);
            *b = nullptr;
        }
        if ((e = cudaMalloc(&s.rec, (size_t)std::max(n, 1u) * 48)) != cudaSuccess) { *what = "sorted records"; return e; }
        if ((e = cudaMalloc(&s.tiles, (size_t)std::max(n, 1u) * 8)) != cudaSuccess) { *what = "sorted rectangles"; return e; }
        if ((e = cudaMalloc(&s.sums, ((size_t)n / kEbSplats + 1) * 4)) != cudaSuccess) { *what = "entry sums"; return e; }
        if (!s.total && (e = cudaMalloc(&s.total, 64)) != cudaSuccess) { *what = "entry total"; return e; }
        if (!s.host_total && (e = cudaMallocHost(&s.host_total, 64)) != cudaSuccess) { *what = "pinned total"; return e; }
        if (!s.counted && (e = cudaEventCreateWithFlags(&s.counted, cudaEventDisableTiming)) != cudaSuccess) { *what = "event"; return e; }
        s.cap_n = n;
    }
    // Bins of the blend: the tuned shape, by default 32 x 32, doubled in large frames where that is the faster
    // (double_bins). All are multiples of the blend's 8 x 8 regions.
    TileGeom tg;
    tg.tw = s.tw;
    tg.th = s.th;
    if (!s.tw) tg.tw = tg.th = 32u;
    const bool choose = !s.tw && (uint64_t)f.W * f.H >= kBin64Pixels;
    auto count_bins = [&] {
        tg.tiles_x = (f.W + tg.tw - 1) / tg.tw;
        tg.tiles_y = (f.H + tg.th - 1) / tg.th;
    };
    count_bins();
    cudaMemsetAsync(stats + ST_PROBE, 0, 8, st);  // the probe reports the last view (sorted.rs:316-322)
    if (full) cudaMemsetAsync(s.total, 0, 16, st);
    auto project = full && choose ? k_sp_project<true> : k_sp_project<false>;
    project<<<(n + 127) / 128, 128, 0, st>>>(f, tg, splats, sh, (uint32_t*)s.keys_a, (uint32_t*)s.vals_a, (float4*)s.rec,
                                             (uint2*)s.tiles, stats, (ull*)s.total, full ? 1 : 0);
    if ((e = cudaGetLastError()) != cudaSuccess) { *what = "sp_project kernel"; return e; }
    *launches = 1;
    if (!full) return cudaSuccess;
    // the number of bin entries sizes their buffers: it comes back while the depth sort runs
    cudaMemcpyAsync(s.host_total, s.total, 16, cudaMemcpyDeviceToHost, st);
    if ((e = cudaEventRecord(s.counted, st)) != cudaSuccess) { *what = "sorted path"; return e; }
    e = radix_sort_pairs(s.rs_keys, (uint32_t*)s.keys_a, (uint32_t*)s.vals_a, (uint32_t*)s.keys_b, (uint32_t*)s.vals_b, n, 24,
                         s.digit_bits, err, st);
    if (e != cudaSuccess) { *what = "depth sort"; return e; }
    const uint32_t nb = (n + kEbSplats - 1) / kEbSplats;
    *launches += radix_sort_launches(24, s.digit_bits) + 3;
    k_entry_sums<<<nb, kEbT, 0, st>>>((uint32_t*)s.vals_b, (uint2*)s.tiles, (ull*)s.total, choose, n, (uint32_t*)s.sums);
    k_scan_sums<<<1, 1024, 0, st>>>((uint32_t*)s.sums, nb);
    k_entry_offsets<<<nb, kEbT, 0, st>>>((uint32_t*)s.vals_b, (uint2*)s.tiles, (uint32_t*)s.sums, (ull*)s.total, choose, n,
                                          (uint32_t*)s.offs);
    if ((e = cudaEventSynchronize(s.counted)) != cudaSuccess) { *what = "sorted path"; return e; }
    const ull* totals = (const ull*)s.host_total;
    const bool twice = choose && double_bins(totals);
    const ull total = totals[twice ? 1 : 0];
    if (twice) {
        tg.tw *= 2u;
        tg.th *= 2u;
        count_bins();
    }
    const uint32_t n_tiles = tg.tiles_x * tg.tiles_y;
    if (total > kMaxEntries) { *what = "more than 2^30 tile entries"; return cudaErrorInvalidValue; }
    const uint32_t m = (uint32_t)total;
    if (m > s.cap_entries) {
        void** bufs[] = {&s.ent_key_a, &s.ent_val_a, &s.ent_key_b, &s.ent_val_b};
        size_t want = (size_t)m + m / 4 + 1024;
        s.cap_entries = 0;
        for (void** b : bufs) {
            if (*b) cudaFree(*b);
            *b = nullptr;
            if ((e = cudaMalloc(b, want * 4)) != cudaSuccess) { *what = "tile entries"; return e; }
        }
        s.cap_entries = (uint32_t)want;
    }
    if (n_tiles > s.n_tiles || !s.ranges) {
        if (s.ranges) cudaFree(s.ranges);
        s.ranges = nullptr;
        if ((e = cudaMalloc(&s.ranges, ((size_t)n_tiles + 1) * 4)) != cudaSuccess) { *what = "tile ranges"; return e; }
        s.n_tiles = n_tiles;
    }
    if (m) {
        int tbits = 1;
        while ((1u << tbits) < n_tiles) ++tbits;
        // the entries start in the buffer from which the sort's passes end in (ent_key_b, ent_val_b)
        const bool even = ((tbits + 7) / 8) % 2 == 0;
        auto entries = twice ? k_entries<true> : k_entries<false>;
        entries<<<(m + 8 * kEwEntries - 1) / (8 * kEwEntries), 256, 0, st>>>(
            (uint32_t*)s.vals_b, (uint2*)s.tiles, (uint32_t*)s.offs, n, tg.tiles_x, m,
            (uint32_t*)(even ? s.ent_key_b : s.ent_key_a), (uint32_t*)(even ? s.ent_val_b : s.ent_val_a));
        e = radix_sort_pairs(s.rs_tiles, (uint32_t*)s.ent_key_a, (uint32_t*)s.ent_val_a, (uint32_t*)s.ent_key_b,
                             (uint32_t*)s.ent_val_b, m, tbits, 8, err, st, true);
        if (e != cudaSuccess) { *what = "tile sort"; return e; }
        *launches += 1 + radix_sort_launches(tbits, 8);
    }
    k_bin_ranges<<<n_tiles / 4 + 1, 128, 0, st>>>((uint32_t*)s.ent_key_b, m, n_tiles, (uint32_t*)s.ranges);
    blend_launch<8, 8>(s, f, tg, accum, st);
    *launches += 2;
    if ((e = cudaGetLastError()) != cudaSuccess) { *what = "blend kernel"; return e; }
    return cudaSuccess;
}

cudaError_t sorted_read(SortedState& s, uint32_t* keys, uint32_t* vals, uint32_t n, cudaStream_t st) {
    if (!s.keys_b || n > s.cap_n) return cudaErrorInvalidValue;
    cudaMemcpyAsync(keys, s.keys_b, (size_t)n * 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(vals, s.vals_b, (size_t)n * 4, cudaMemcpyDeviceToHost, st);
    return cudaStreamSynchronize(st);
}

// ============================================================================ composite
__device__ __forceinline__ float oetf(float c) {
    if (c <= F_(0.0031308)) return F_(12.92) * c;
    return F_(1.055) * gx::pow(c, gxc::kInv2p4) - F_(0.055);
}
__device__ __forceinline__ void lin_px(const float4* accum, uint32_t W, uint32_t H, int px, int py, float* c) {
    int qx = min(max(px, 0), (int)W - 1), qy = min(max(py, 0), (int)H - 1);
    float4 a = __ldg(&accum[(size_t)qy * W + qx]);
    float d = fmax_(a.w, F_(1.0));
    c[0] = div_(a.x, d);
    c[1] = div_(a.y, d);
    c[2] = div_(a.z, d);
}
__device__ __forceinline__ float mixc(float a, float b, float t) { return a * (F_(1.0) - t) + b * t; }

__global__ void k_composite(const float4* __restrict__ accum, uint32_t W, uint32_t H, float exposure, uint32_t gamma_on,
                            uint32_t out_w, uint32_t out_h, uchar4* out) {
    uint32_t X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y;
    if (X >= out_w || Y >= out_h) return;
    float uvx = div_((float)X + F_(0.5), (float)out_w), uvy = div_((float)Y + F_(0.5), (float)out_h);
    float qx = uvx * (float)W - F_(0.5), qy = uvy * (float)H - F_(0.5);
    float fx0 = floorf(qx), fy0 = floorf(qy);
    int px = (int)fx0, py = (int)fy0;
    float fx = qx - fx0, fy = qy - fy0;
    float c00[3], c10[3], c01[3], c11[3];
    lin_px(accum, W, H, px, py, c00);
    lin_px(accum, W, H, px + 1, py, c10);
    lin_px(accum, W, H, px, py + 1, c01);
    lin_px(accum, W, H, px + 1, py + 1, c11);
    unsigned char o[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float top = mixc(c00[k], c10[k], fx), bot = mixc(c01[k], c11[k], fx);
        float c = mixc(top, bot, fy) * exposure;
        c = clamp_(c, F_(0.0), F_(1.0));
        if (gamma_on) c = oetf(c);
        o[k] = (unsigned char)f2u(gx::rint_(c * F_(255.0)));
    }
    out[(size_t)Y * out_w + X] = make_uchar4(o[0], o[1], o[2], 255);
}

void launch_composite(const float4* accum, uint32_t W, uint32_t H, float exposure, uint32_t gamma_on, uint32_t out_w,
                      uint32_t out_h, uchar4* out, cudaStream_t st) {
    dim3 grid((out_w + 255) / 256, out_h);
    k_composite<<<grid, 256, 0, st>>>(accum, W, H, exposure, gamma_on, out_w, out_h, out);
}

}  // namespace gpsb

// ============================================================================ C ABI: no-allocation sort
namespace gpsb {
void set_global_error(const char* msg);  // renderer.cpp: message of gpsb_last_error(NULL)
}
static thread_local char g_noalloc_error[256];

extern "C" gpsb_status gpsb_sort_pairs_noalloc(uint32_t* keys_in, uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                                               uint32_t n, uint32_t key_bits, void* cuda_stream, uint32_t* err_dev) {
    using namespace gpsb;
    g_noalloc_error[0] = 0;
    if (n > kNoAllocMaxN) {
        snprintf(g_noalloc_error, sizeof g_noalloc_error,
                 "gpsb_sort_pairs_noalloc: %u pairs exceed the fixed scratch of %u pairs", n, kNoAllocMaxN);
        set_global_error(g_noalloc_error);
        return GPSB_ERR_LIMIT;
    }
    if (key_bits < 1 || key_bits > 32) {
        snprintf(g_noalloc_error, sizeof g_noalloc_error, "gpsb_sort_pairs_noalloc: key_bits must be 1..32");
        set_global_error(g_noalloc_error);
        return GPSB_ERR_INVALID_ARGUMENT;
    }
    if (n == 0) return GPSB_OK;
    if (!keys_in || !vals_in || !keys_out || !vals_out || !err_dev) {
        snprintf(g_noalloc_error, sizeof g_noalloc_error, "gpsb_sort_pairs_noalloc: null buffer or error word");
        set_global_error(g_noalloc_error);
        return GPSB_ERR_INVALID_ARGUMENT;
    }
    cudaStream_t st = (cudaStream_t)cuda_stream;
    cudaError_t e;
    bool capture_without_setup = false;
    uint32_t* base = (uint32_t*)noalloc_scratch_address(st, &e, &capture_without_setup);
    if (!base) {
        if (capture_without_setup)
            snprintf(g_noalloc_error, sizeof g_noalloc_error,
                     "gpsb_sort_pairs_noalloc: the first call on a device must come before any stream capture");
        else
            snprintf(g_noalloc_error, sizeof g_noalloc_error, "gpsb_sort_pairs_noalloc: scratch address: %s",
                     cudaGetErrorString(e));
        set_global_error(g_noalloc_error);
        return capture_without_setup ? GPSB_ERR_STATE : GPSB_ERR_CUDA;
    }
    const int passes = (int)((key_bits + 7) / 8);
    const uint32_t tiles = onesweep_tiles<8>(n);
    uint32_t* hist = base;
    uint32_t* counters = base + kNoAllocHistWords;
    uint32_t* err = err_dev;
    uint32_t* lookback = base + kNoAllocHistWords + kNoAllocCounterWords;
    // the array keeps the previous call's contents: clear what this call needs at zero
    e = cudaMemsetAsync(base, 0, (kNoAllocHistWords + kNoAllocCounterWords + (size_t)passes * tiles * 256) * 4, st);
    uint32_t *ik = keys_in, *iv = vals_in, *ok = keys_out, *ov = vals_out;
    if (e == cudaSuccess && passes % 2 == 0) {
        // an even number of passes ends in the first buffer: start from a copy in the output
        e = cudaMemcpyAsync(keys_out, keys_in, (size_t)n * 4, cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(vals_out, vals_in, (size_t)n * 4, cudaMemcpyDeviceToDevice, st);
        ik = keys_out; iv = vals_out; ok = keys_in; ov = vals_in;
    }
    if (e == cudaSuccess) {
        launch_pdl(k_radix_hist<8>, dim3(std::min<uint32_t>((n + 4095) / 4096, 1184u)), dim3(256), 0, st, ik, n, passes, hist);
        launch_pdl(k_radix_hist_scan<8>, dim3(passes), dim3(256), 0, st, hist);
        for (int p = 0; p < passes; ++p) {
            onesweep_launch<8>(true, tiles, ik, iv, ok, ov, n, p * 8, hist + p * 256, lookback + (size_t)p * tiles * 256,
                               counters + p, err, st);
            std::swap(ik, ok);
            std::swap(iv, ov);
        }
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        snprintf(g_noalloc_error, sizeof g_noalloc_error, "gpsb_sort_pairs_noalloc: %s", cudaGetErrorString(e));
        set_global_error(g_noalloc_error);
        return GPSB_ERR_CUDA;
    }
    return GPSB_OK;
}
