// sph_sort.cu -- Compute::sort (SPH/Compute/Compute.cpp:265-326) for sm_100a.
//
// The reference hashes every particle to a 24-bit Morton cell key
// (sort.metal:15-44), sorts (key, index) pairs with four stable 8-bit LSD
// passes of hist/scan/sum/scatter dispatches (sort.metal:46-129), then
// re-initialises all 2^24 cell entries and finds each cell's first and last
// sorted index with atomics (sort.metal:131-148).
//
// Here:
//  * k_hash_hist computes the keys and, in the same sweep, the global digit
//    histograms of all passes (the one-sweep "upsweep"); it also clears only
//    the cell entries the previous sort filled, instead of all 2^24;
//  * k_onesweep does one stable 8-bit pass per launch: warp-level ranking
//    with ballots, a decoupled look-back across tiles for each digit (every
//    wait is bounded and raises a health bit instead of hanging), scatter;
//    the top byte of the 24-bit keys is always zero, so three passes give the
//    reference's four-pass order exactly;
//  * k_cells writes each occupied cell's (first, last) sorted index from
//    neighbouring keys, without atomics.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>

#include "sph_internal.h"

namespace sph {

namespace {

constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1u;
constexpr uint32_t kArrived = 1u << 27;  // group words: tiles added, above the sum of their counts
static_assert(RadixSorter::kGroup * RadixSorter::kThreads * RadixSorter::kMaxItems < kArrived &&
                  RadixSorter::kGroup < 32, "group words");
constexpr int kSpinLimit = 1 << 22;

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Blocks of the key kernels: each ends in one set of 768 global atomics, which
// took the time with 2368 blocks (N = 1e6: 28 of the sort's 131 us).
constexpr int kHashThreads = 512;
constexpr int kHashBlocks = 296;
int hash_grid(int n) { return std::max(1, std::min(kHashBlocks, (n + kHashThreads - 1) / kHashThreads)); }

// Keys of the cell grid + all three digit histograms; clears the previous
// sort's occupied cells, octets and units first (they are read from the previous
// sorted keys, which live in the buffer the first pass is about to overwrite).
__global__ void __launch_bounds__(kHashThreads)
    k_hash_hist(const float4 *__restrict__ pos4, int n, uint32_t *__restrict__ keys, uint32_t *__restrict__ vals,
                uint32_t *__restrict__ hist, const uint32_t *__restrict__ prev_keys, uint2 *__restrict__ cell_range,
                uint2 *__restrict__ octets, uint2 *__restrict__ units, int clear_prev) {
    __shared__ uint32_t sh[3][256];
    for (int i = threadIdx.x; i < 3 * 256; i += blockDim.x) (&sh[0][0])[i] = 0u;
    __syncthreads();
#pragma unroll 2
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (clear_prev) {
            const uint32_t pk = prev_keys[i], before = i ? prev_keys[i - 1] : ~pk;
            if (before != pk) cell_range[pk] = make_uint2(0xffffffffu, 0u);
            if ((before ^ pk) >> 3) octets[pk >> 3] = make_uint2(0xffffffffu, 0xffffffffu);
            if ((before ^ pk) >> (3 * kUnitShift)) units[pk >> (3 * kUnitShift)] = make_uint2(0xffffffffu, 0xffffffffu);
        }
        const float4 p = __ldg(pos4 + i);
        const uint32_t k = cell_key(p.x, p.y, p.z);
        keys[i] = k;
        vals[i] = (uint32_t)i;
        atomicAdd(&sh[0][k & 255u], 1u);
        atomicAdd(&sh[1][(k >> 8) & 255u], 1u);
        atomicAdd(&sh[2][(k >> 16) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * 256; i += blockDim.x) {
        const uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
}

// The valid lanes of the warp whose 8-bit digit equals this lane's, by a ballot
// per bit: match_any takes a round per distinct digit.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool ok) {
    uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// One stable 8-bit LSD pass over tiles of 256 x ITEMS keys.
template <int ITEMS>
__global__ void __launch_bounds__(RadixSorter::kThreads)
    k_onesweep(const uint32_t *__restrict__ keys_in, const uint32_t *__restrict__ vals_in,
               uint32_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out, int n, int shift,
               const uint32_t *__restrict__ hist, uint32_t *status, int tiles, uint32_t *counter, uint32_t *health,
               uint32_t *failed, int spin_limit) {
    constexpr int T = RadixSorter::kThreads, I = ITEMS, W = T / 32, G = RadixSorter::kGroup;
    // tiles, groups read at a time (the polls of all waiting tiles meet in a few
    // lines of L2: with twice as many, N = 1e6 in tiles of 2048 keys takes 171
    // instead of 93 us)
    constexpr int kWindow = 4, kGroupWindow = 4;
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_warp[W][256];
    __shared__ uint32_t s_base[256];
    __shared__ uint32_t s_scan[W];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(counter, 1u);
    for (int i = tid; i < W * 256; i += T) (&s_warp[0][0])[i] = 0u;
    // exclusive prefix of the global histogram over digits
    const uint32_t count = hist[tid];
    uint32_t incl = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    uint32_t global_excl = incl - count;
#pragma unroll
    for (int w = 0; w < W; ++w)
        if (w < warp) global_excl += s_scan[w];
    const uint32_t tile = s_tile;
    const int64_t base = (int64_t)tile * (T * I) + (int64_t)warp * (I * 32);
    const uint32_t lt = lanemask_lt();

    uint32_t k[I], v[I], rank[I];
#pragma unroll
    for (int it = 0; it < I; ++it) {
        int64_t idx = base + it * 32 + lane;
        bool ok = idx < n;
        k[it] = ok ? keys_in[idx] : 0u;
        v[it] = ok ? vals_in[idx] : 0u;
    }
#pragma unroll
    for (int it = 0; it < I; ++it) {
        const bool ok = base + it * 32 + lane < n;
        const uint32_t d = (k[it] >> shift) & 255u;
        const uint32_t peers = digit_peers(d, ok);
        const uint32_t before = s_warp[warp][d];
        rank[it] = before + __popc(peers & lt);
        __syncwarp();
        if (ok && (peers & lt) == 0u) s_warp[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit: offsets of the warps inside the tile, and the tile total
    uint32_t tile_count = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        uint32_t c = s_warp[w][tid];
        s_warp[w][tid] = tile_count;
        tile_count += c;
    }
    // Decoupled look-back for digit `tid` (the words carry the counts
    // themselves: nothing else has to be ordered).  All tiles of a sort of 1e6
    // keys run at once, so that most words hold only their own tile's count and
    // a walk over single tiles reads all before it.  So a tile also adds its
    // count to its group's word, and the walk goes by tiles to the group's start
    // and then by groups, whichever of a group's sum and its last tile's prefix
    // is there.
    uint32_t excl = 0;
    volatile uint32_t *vs = status;
    uint32_t *const groups = status + (size_t)tiles * 256;
    volatile uint32_t *vg = groups;
    const int64_t group = tile / G, first = group * G;
    vs[(size_t)tile * 256 + tid] = (tile == 0 ? kFlagPrefix : kFlagAgg) | tile_count;
    if (tiles > G) atomicAdd(groups + group * 256 + tid, kArrived | tile_count);
    int spins = 0;
    bool done = tile == 0;
    auto wait = [&]() {  // false: given up
        if (++spins > spin_limit) {
            raise_health(health, SPH_HEALTH_SORT_TIMEOUT);
            if (failed) *failed = 1u;
            return false;
        }
        __nanosleep(32);
        return true;
    };
    for (int64_t j = (int64_t)tile - 1; !done && j >= first;) {
        uint32_t s[kWindow];
#pragma unroll
        for (int q = 0; q < kWindow; ++q) s[q] = j - q >= first ? vs[(size_t)(j - q) * 256 + tid] : 0u;
        int got = 0;
#pragma unroll
        for (int q = 0; q < kWindow; ++q) {
            const uint32_t flag = s[q] & ~kValueMask;
            if (!done && got == q && flag != 0u) {
                excl += s[q] & kValueMask;
                ++got;
                done = flag == kFlagPrefix;
            }
        }
        j -= got;
        if (got == 0 && !wait()) done = true;
    }
    for (int64_t j = group - 1; !done && j >= 0;) {
        uint32_t s[kGroupWindow], e[kGroupWindow];
#pragma unroll
        for (int q = 0; q < kGroupWindow; ++q) {
            s[q] = j - q >= 0 ? vg[(size_t)(j - q) * 256 + tid] : 0u;
            e[q] = j - q >= 0 ? vs[(size_t)((j - q) * G + G - 1) * 256 + tid] : 0u;
        }
        int got = 0;
#pragma unroll
        for (int q = 0; q < kGroupWindow; ++q) {
            const bool prefix = (e[q] & ~kValueMask) == kFlagPrefix;
            if (!done && got == q && (prefix || s[q] / kArrived == G)) {
                excl += prefix ? e[q] & kValueMask : s[q] % kArrived;
                ++got;
                done = prefix;
            }
        }
        j -= got;
        if (got == 0 && !wait()) done = true;
    }
    if (tile != 0) vs[(size_t)tile * 256 + tid] = kFlagPrefix | ((excl + tile_count) & kValueMask);
    s_base[tid] = global_excl + excl;
    __syncthreads();
#pragma unroll
    for (int it = 0; it < I; ++it) {
        int64_t idx = base + it * 32 + lane;
        if (idx < n) {
            uint32_t d = (k[it] >> shift) & 255u;
            uint32_t dst = s_base[d] + s_warp[warp][d] + rank[it];
            if (dst < (uint32_t)n) {  // only a timed-out look-back can break this
                keys_out[dst] = k[it];
                vals_out[dst] = v[it];
            }
        }
    }
}

void launch_onesweep(const uint32_t *keys_in, const uint32_t *vals_in, uint32_t *keys_out, uint32_t *vals_out, int n,
                     int shift, const uint32_t *hist, uint32_t *status, uint32_t *counter, uint32_t *health,
                     uint32_t *failed, int spin_limit, cudaStream_t st, bool withhold = false) {
    const int tiles = RadixSorter::tiles(n), items = RadixSorter::items(n);
    auto *kernel = items == 4 ? k_onesweep<4> : items == 8 ? k_onesweep<8> : k_onesweep<16>;
    kernel<<<withhold ? tiles - 1 : tiles, RadixSorter::kThreads, 0, st>>>(
        keys_in, vals_in, keys_out, vals_out, n, shift, hist, status, tiles, counter, health, failed, spin_limit);
}

// Self-test: the tickets of all passes start behind the first tile.
__global__ void k_withhold(uint32_t *counters) { counters[threadIdx.x] = 1u; }

// Each occupied cell's (first, last) sorted index, and each occupied octet's
// (cell key >> 3) and unit's (cell key >> 6).  Of keys that are not sorted there
// are no ranges: all cells stay empty (a first index behind the last would be a
// run over most of memory).
__global__ void k_cells(const uint32_t *__restrict__ keys, int n, uint2 *__restrict__ cell_range,
                        uint2 *__restrict__ octets, uint2 *__restrict__ units, const uint32_t *__restrict__ failed) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || *failed) return;
    const uint32_t k = keys[i], u = k >> (3 * kUnitShift);
    const uint32_t before = i ? keys[i - 1] : ~k, after = i < n - 1 ? keys[i + 1] : ~k;
    if (before != k) cell_range[k].x = (uint32_t)i;
    if (after != k) cell_range[k].y = (uint32_t)i;
    if ((before ^ k) >> 3) octets[k >> 3].x = (uint32_t)i;
    if ((after ^ k) >> 3) octets[k >> 3].y = (uint32_t)i;
    if ((before >> (3 * kUnitShift)) != u) units[u].x = (uint32_t)i;
    if ((after >> (3 * kUnitShift)) != u) units[u].y = (uint32_t)i;
}

__global__ void k_init_cells(uint2 *cell_range, uint32_t count) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
        cell_range[i] = make_uint2(0xffffffffu, 0u);
}

}  // namespace

sph_status sort_alloc(RadixSorter &s, int n) {
    s.n_cap = n;
    constexpr int kMinTile = RadixSorter::kThreads * RadixSorter::kMinItems;
    const size_t rows = RadixSorter::rows(std::max(1, (n + kMinTile - 1) / kMinTile));
    constexpr size_t kHead = 256 * RadixSorter::kMaxPasses + RadixSorter::kMaxPasses + 1;
    size_t nb = sizeof(uint32_t) * (size_t)(n > 0 ? n : 1);
    cudaError_t e = cudaSuccess;
    for (int b = 0; b < 2; ++b) {
        if (e == cudaSuccess) e = cudaMalloc(&s.keys[b], nb);
        if (e == cudaSuccess) e = cudaMalloc(&s.vals[b], nb);
        // (in range from the start: a sort that fails leaves entries unwritten)
        if (e == cudaSuccess) e = cudaMemset(s.keys[b], 0, nb);
        if (e == cudaSuccess) e = cudaMemset(s.vals[b], 0, nb);
    }
    if (e == cudaSuccess) e = cudaMalloc(&s.hist, sizeof(uint32_t) * (kHead + 256 * rows * RadixSorter::kMaxPasses));
    s.counters = s.hist + 256 * RadixSorter::kMaxPasses;
    s.failed = s.counters + RadixSorter::kMaxPasses;
    s.status = s.hist + kHead;
    return cuda_status(e, "sort_alloc");
}

void sort_free(RadixSorter &s) {
    for (int b = 0; b < 2; ++b) {
        cudaFree(s.keys[b]);
        cudaFree(s.vals[b]);
        s.keys[b] = s.vals[b] = nullptr;
    }
    cudaFree(s.hist);
    s.hist = s.status = s.counters = s.failed = nullptr;
}

void radix_clear(RadixSorter &s, int n, int bits, cudaStream_t st) {
    const size_t words = (size_t)(s.status - s.hist) + 256 * RadixSorter::rows(RadixSorter::tiles(n)) * ((bits + 7) / 8);
    cudaMemsetAsync(s.hist, 0, sizeof(uint32_t) * words, st);
}

int radix_sort_pairs(RadixSorter &s, int n, int bits, cudaStream_t st, uint32_t *health, bool withhold) {
    const int passes = (bits + 7) / 8;
    int cur = 0;
    if (n <= 0) return 0;
    if (withhold) k_withhold<<<1, RadixSorter::kMaxPasses, 0, st>>>(s.counters);
    for (int p = 0; p < passes; ++p) {
        launch_onesweep(s.keys[cur], s.vals[cur], s.keys[cur ^ 1], s.vals[cur ^ 1], n, 8 * p, s.hist + 256 * p,
                        s.status + 256 * RadixSorter::rows(RadixSorter::tiles(n)) * p, s.counters + p, health, s.failed,
                        s.spin_limit, st, withhold);
        cur ^= 1;
    }
    return cur;
}

void launch_init_cells(sph_ctx *ctx, cudaStream_t st) {
    k_init_cells<<<148 * 8, 256, 0, st>>>(ctx->cell_range, kNumCells);
    cudaMemsetAsync(ctx->octets, 0xff, sizeof(uint2) * kNumOctets, st);
    cudaMemsetAsync(ctx->units, 0xff, sizeof(uint2) * kNumUnits, st);
    ctx->cells_have_prev = false;
}

sph_status launch_sort(sph_ctx *ctx, cudaStream_t st, bool withhold) {
    RadixSorter &s = ctx->cell_sort;
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    radix_clear(s, n, 24, st);
    const int prev = ctx->cell_final;
    // the previous sorted keys live in keys[prev]; the hash writes keys[0] and
    // the first pass writes keys[1], so clearing must use keys[prev] before that
    uint32_t *clear_src = s.keys[prev];
    if (prev == 0) {
        // never the case with 3 passes (result in buffer 1); kept for safety
        launch_init_cells(ctx, st);
    }
    k_hash_hist<<<hash_grid(n), kHashThreads, 0, st>>>(ctx->pos4, n, s.keys[0], s.vals[0], s.hist, clear_src,
                                                       ctx->cell_range, ctx->octets, ctx->units,
                                                       (ctx->cells_have_prev && prev == 1) ? 1 : 0);
    int fin = radix_sort_pairs(s, n, 24, st, ctx->health, withhold);
    ctx->cell_final = fin;
    k_cells<<<(n + 255) / 256, 256, 0, st>>>(s.keys[fin], n, ctx->cell_range, ctx->octets, ctx->units,
                                              s.failed);
    ctx->cells_have_prev = true;
    return cuda_status(cudaGetLastError(), "sort");
}

}  // namespace sph

// ---------------------------------------------------------------------------
// Cell sort without allocation.
//
// Some callers cannot allocate device memory at all: code that runs inside a
// host framework which owns every allocation (a pool or arena it hands out,
// memory-accounting or sandboxing layers), or code that must not call
// cudaMalloc/cudaFree on a latency-critical thread because those calls may
// synchronise the device.  For them, sph_sort_cells_noalloc computes the same
// sorted (cell key, particle index) pairs as sph_sort from positions the
// caller already holds on the device, using only caller-provided inputs and
// outputs plus one fixed scratch array compiled into this library.
//
// The scratch is a file-scope __device__ array, so every GPU that loads the
// library carries it (kNoAllocScratchBytes, about 2.8 MiB) until the process
// exits.  On the host, the array's name is only a stand-in symbol, not a
// device address; its device address is looked up with cudaGetSymbolAddress
// on every call, for the device current at that call (the first lookup on a
// device loads the module there, which is why the first call should come
// before any stream capture).  Every call shares the array and it keeps the
// last call's contents, so the parts that must start at zero (histograms,
// tile tickets, the health word and the look-back words this call's size
// uses) are cleared on the caller's stream at each call, and calls whose work
// overlaps on the GPU (different streams without ordering, or several host
// threads) race on it.  A look-back wait that gives up raises the health word
// inside the scratch; sph_sort_cells_noalloc_health reads it back.
// ---------------------------------------------------------------------------
namespace sph {
namespace {

constexpr int kNoAllocPasses = 3;  // 24-bit cell keys
constexpr int kNoAllocTiles = SPH_SORT_NOALLOC_MAX_N / (RadixSorter::kThreads * RadixSorter::kMinItems);
static_assert(SPH_SORT_NOALLOC_MAX_N % (RadixSorter::kThreads * RadixSorter::kMinItems) == 0, "whole tiles");
constexpr size_t kNoAllocKeysOff = 0;
constexpr size_t kNoAllocValsOff = kNoAllocKeysOff + sizeof(uint32_t) * SPH_SORT_NOALLOC_MAX_N;
// the words that must be zero when a call starts sit together from here on:
// histograms, tile tickets, the health word, then the look-back words of the
// three passes, each pass using 256 x (rows of this call) words
constexpr size_t kNoAllocHistOff = kNoAllocValsOff + sizeof(uint32_t) * SPH_SORT_NOALLOC_MAX_N;
constexpr size_t kNoAllocCountOff = kNoAllocHistOff + sizeof(uint32_t) * 256 * kNoAllocPasses;
constexpr size_t kNoAllocHealthOff = kNoAllocCountOff + sizeof(uint32_t) * kNoAllocPasses;
constexpr size_t kNoAllocStatusOff = kNoAllocHealthOff + sizeof(uint32_t);
constexpr size_t kNoAllocScratchBytes = kNoAllocStatusOff + sizeof(uint32_t) * 256 * RadixSorter::rows(kNoAllocTiles) * kNoAllocPasses;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// sort.metal:15-44 from xyz-interleaved positions, plus the digit histograms
// of the three passes (same keys as k_hash_hist; no cell table to clear).
__global__ void k_hash_hist_xyz(const float *__restrict__ pos, int n, uint32_t *__restrict__ keys,
                                uint32_t *__restrict__ vals, uint32_t *__restrict__ hist) {
    __shared__ uint32_t sh[3][256];
    for (int i = threadIdx.x; i < 3 * 256; i += blockDim.x) (&sh[0][0])[i] = 0u;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = cell_key(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]);
        keys[i] = k;
        vals[i] = (uint32_t)i;
        atomicAdd(&sh[0][k & 255u], 1u);
        atomicAdd(&sh[1][(k >> 8) & 255u], 1u);
        atomicAdd(&sh[2][(k >> 16) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * 256; i += blockDim.x) {
        const uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
}

// Device address of the scratch array on the current device.
sph_status noalloc_scratch(unsigned char **out) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_status(e, "sph_sort_cells_noalloc: cudaGetSymbolAddress");
    *out = static_cast<unsigned char *>(p);
    return SPH_OK;
}

}  // namespace

}  // namespace sph

extern "C" sph_status sph_sort_cells_noalloc(const float *pos_xyz, int32_t n, uint32_t *cell_key,
                                            uint32_t *cell_index, void *stream) {
    using namespace sph;
    if (n < 0 || n > SPH_SORT_NOALLOC_MAX_N) {
        set_error("sph_sort_cells_noalloc: n = %d is outside 0..%d (the size of the library's fixed scratch)", n,
                  SPH_SORT_NOALLOC_MAX_N);
        return SPH_ERR_INVALID_ARG;
    }
    if (n == 0) return SPH_OK;
    if (!pos_xyz || !cell_key || !cell_index) {
        set_error("sph_sort_cells_noalloc: null device pointer");
        return SPH_ERR_INVALID_ARG;
    }
    unsigned char *s = nullptr;
    sph_status st = noalloc_scratch(&s);
    if (st != SPH_OK) return st;
    cudaStream_t cs = (cudaStream_t)stream;
    const size_t rows = RadixSorter::rows(RadixSorter::tiles(n));
    uint32_t *tk = reinterpret_cast<uint32_t *>(s + kNoAllocKeysOff);
    uint32_t *tv = reinterpret_cast<uint32_t *>(s + kNoAllocValsOff);
    uint32_t *hist = reinterpret_cast<uint32_t *>(s + kNoAllocHistOff);
    uint32_t *counters = reinterpret_cast<uint32_t *>(s + kNoAllocCountOff);
    uint32_t *health = reinterpret_cast<uint32_t *>(s + kNoAllocHealthOff);
    uint32_t *status = reinterpret_cast<uint32_t *>(s + kNoAllocStatusOff);
    const size_t zero_bytes = (kNoAllocStatusOff - kNoAllocHistOff) + sizeof(uint32_t) * 256 * rows * kNoAllocPasses;
    cudaError_t e = cudaMemsetAsync(s + kNoAllocHistOff, 0, zero_bytes, cs);
    if (e != cudaSuccess) return cuda_status(e, "sph_sort_cells_noalloc: clear scratch");
    k_hash_hist_xyz<<<hash_grid(n), kHashThreads, 0, cs>>>(pos_xyz, n, tk, tv, hist);
    // three stable 8-bit passes: scratch -> out -> scratch -> out
    uint32_t *kin[kNoAllocPasses] = {tk, cell_key, tk};
    uint32_t *vin[kNoAllocPasses] = {tv, cell_index, tv};
    uint32_t *kout[kNoAllocPasses] = {cell_key, tk, cell_key};
    uint32_t *vout[kNoAllocPasses] = {cell_index, tv, cell_index};
    for (int p = 0; p < kNoAllocPasses; ++p)
        launch_onesweep(kin[p], vin[p], kout[p], vout[p], n, 8 * p, hist + 256 * p,
                        status + 256 * rows * p, counters + p, health, nullptr, kSpinLimit, cs);
    return cuda_status(cudaGetLastError(), "sph_sort_cells_noalloc");
}

extern "C" sph_status sph_sort_cells_noalloc_health(void *stream, uint32_t *word) {
    using namespace sph;
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_status(e, "sph_sort_cells_noalloc_health: stream");
    uint32_t w = 0;
    e = cudaMemcpyFromSymbol(&w, g_noalloc_scratch, sizeof(uint32_t), kNoAllocHealthOff, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_status(e, "sph_sort_cells_noalloc_health: read");
    if (word) *word = w;
    if (w & SPH_HEALTH_SORT_TIMEOUT) {
        set_error("sph_sort_cells_noalloc: a look-back wait gave up (health 0x%x); the outputs are incomplete", w);
        return SPH_ERR_TIMEOUT;
    }
    return SPH_OK;
}

// ---------------------------------------------------------------------------
// Self-test of the bounded look-back wait.  One k_onesweep tile is launched
// whose ticket is preset to 1, so it waits on tile 0's status words, which
// nothing writes: the wait must give up after spin_limit polls, raise
// SPH_HEALTH_SORT_TIMEOUT and return.  The tile holds no elements (n = 0), so
// it reads and writes no key or value.  With ctx the context's sorter scratch
// and health word are used (sph_synchronize then reports SPH_ERR_TIMEOUT);
// without, the allocation-free sort's static scratch is used
// (sph_sort_cells_noalloc_health then reports it).
// ---------------------------------------------------------------------------
namespace sph {
namespace {
__global__ void k_selftest_prepare(uint32_t *hist, uint32_t *status, uint32_t *counter) {
    const int t = threadIdx.x;  // 256 threads
    hist[t] = 0u;
    status[t] = 0u;
    status[256 + t] = 0u;
    status[512 + t] = 0u;  // the group's word
    if (t == 0) *counter = 1u;
}
}  // namespace
}  // namespace sph

extern "C" sph_status sph_selftest_lookback_timeout(sph_ctx *ctx, int32_t spin_limit, void *stream) {
    using namespace sph;
    if (spin_limit < 1 || spin_limit > (1 << 22)) {
        set_error("sph_selftest_lookback_timeout: spin_limit %d is outside 1..%d", spin_limit, 1 << 22);
        return SPH_ERR_INVALID_ARG;
    }
    cudaStream_t cs = (cudaStream_t)stream;
    uint32_t *hist, *status, *counter, *health, *kbuf, *vbuf;
    if (ctx) {
        cudaSetDevice(ctx->device);
        RadixSorter &r = ctx->cell_sort;  // status holds >= 4 x 256 words
        hist = r.hist;
        status = r.status;
        counter = r.counters;
        health = ctx->health;
        kbuf = r.keys[0];
        vbuf = r.vals[0];
    } else {
        unsigned char *s = nullptr;
        sph_status st = noalloc_scratch(&s);
        if (st != SPH_OK) return st;
        hist = reinterpret_cast<uint32_t *>(s + kNoAllocHistOff);
        counter = reinterpret_cast<uint32_t *>(s + kNoAllocCountOff);
        health = reinterpret_cast<uint32_t *>(s + kNoAllocHealthOff);
        status = reinterpret_cast<uint32_t *>(s + kNoAllocStatusOff);
        kbuf = reinterpret_cast<uint32_t *>(s + kNoAllocKeysOff);
        vbuf = reinterpret_cast<uint32_t *>(s + kNoAllocValsOff);
    }
    // the key/value buffers are valid device memory, though n = 0 touches none
    k_selftest_prepare<<<1, 256, 0, cs>>>(hist, status, counter);
    k_onesweep<RadixSorter::kMinItems><<<1, RadixSorter::kThreads, 0, cs>>>(kbuf, vbuf, kbuf, vbuf, 0, 0, hist, status, 2,
                                                                            counter, health, nullptr, spin_limit);
    return cuda_status(cudaGetLastError(), "sph_selftest_lookback_timeout");
}

// The same for what follows a sort whose waits gave up: a tree build and a cell
// sort whose first tiles are withheld.
extern "C" sph_status sph_selftest_sort_timeout(sph_ctx *ctx, int32_t spin_limit, void *stream) {
    using namespace sph;
    if (!ctx || ctx->params.tree_source != SPH_TREE_GPU || RadixSorter::tiles(ctx->n) < 2 || spin_limit < 1 ||
        spin_limit > (1 << 22)) {
        set_error("sph_selftest_sort_timeout: needs a context with the GPU tree and more than one sort tile, and a "
                  "spin limit in 1..%d", 1 << 22);
        return SPH_ERR_INVALID_ARG;
    }
    cudaSetDevice(ctx->device);
    RadixSorter *const sorters[] = {&ctx->tb.sorter, &ctx->cell_sort};
    // (what an up pass over a tree that is none leaves behind)
    cudaMemsetAsync(ctx->tree.arrived, 1, sizeof(int32_t) * ctx->tree.node_cap, (cudaStream_t)stream);
    for (RadixSorter *r : sorters) r->spin_limit = spin_limit;
    sph_status s = launch_tree_build(ctx, (cudaStream_t)stream, true);
    if (s == SPH_OK) s = launch_sort(ctx, (cudaStream_t)stream, true);
    for (RadixSorter *r : sorters) r->spin_limit = kSpinLimit;
    return s;
}
