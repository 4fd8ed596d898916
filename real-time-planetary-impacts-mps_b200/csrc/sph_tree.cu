// sph_tree.cu -- the octree build, moved from the reference's detached CPU
// thread (SPH/octree/octree.cpp:14-141 via Compute::updateOctreeData,
// Compute.cpp:510-516) onto the GPU.
//
// Tree definition (restated on the CPU by the oracle's ora_tree_build_morton):
//   * keys: each coordinate quantised to D = max_tree_depth bits over the
//     bounding cube (side = largest extent), interleaved with x on bit 0 of
//     each triplet (the reference's morton3D convention);
//   * particles stable-sorted by key (one-sweep radix sort, ties by index);
//   * a node is a leaf if it holds <= max_children_in_leaf particles or sits
//     at depth D; otherwise its children are the non-empty octants of the next
//     key triplet (octant bit x = 1, y = 2, z = 4, the reference's order);
//   * flattened in DFS preorder in the reference's int format
//     (leaf [n, dataPtr, ids...], branch [0, dataPtr, 8 child offsets or -1]),
//     with per-level node lists in DFS order, so the same up/down passes run
//     on it.  The split is geometric (cube midpoints) instead of the
//     reference's per-subset mean.
//
// Build: bounding box -> keys (+ digit histograms) -> sort -> three kernels.
// The nodes follow from the sorted keys alone: with cl(a, b) the number of
// leading triplets that two keys share, the run of particles of a node at
// level l starts at i exactly when cl(i - 1, i) < l, it holds more than
// leafcap particles exactly when cl(i, i + leafcap) >= l, and it is a node
// exactly when its parent's run does.  So each particle knows, from a few
// neighbouring keys, the levels first .. last at which nodes start at it (all
// branches but the last), and an exclusive scan over the particles gives every
// node's DFS offset, data pointer and place in its level's lists:
//   k_tree_mark   levels and ints of each particle's nodes; block totals; the
//                 last block to finish scans them
//   k_tree_write  scans within the block, nodes, level lists, particle ids
//   k_tree_link   the first node at each particle links itself into its
//                 parent (the only node whose parent starts elsewhere)
// With one set of launches per level (82 in all, most of them too small to
// fill the device) the build was half of a gravity pass: tree, up and down
// together, N = 1e6, leaf 32: 2.12 -> 1.62 ms; N = 1e5, leaf 4: 1.25 -> 0.86 ms.
// Every launch size is a host-side upper bound and the true counts stay on
// the device, so the whole build can be captured in a CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>

#include "sph_internal.h"

namespace sph {

namespace {

__device__ __forceinline__ uint32_t f2ord(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Blocks of the passes that end in one set of global atomics per block.
constexpr int kReduceThreads = 512;
constexpr int kReduceBlocks = 296;
int reduce_grid(int n) { return std::max(1, std::min(kReduceBlocks, (n + kReduceThreads - 1) / kReduceThreads)); }

__global__ void k_bbox_init(uint32_t *bb) {
    if (threadIdx.x < 3) bb[threadIdx.x] = 0xffffffffu;
    else if (threadIdx.x < 6) bb[threadIdx.x] = 0u;
}

// Few blocks (kReduceBlocks), each reduced to one value per bound before its
// six atomics: with one set of atomics per warp of 2368 blocks the atomics
// took the time (N = 1e6: 82 us).
__global__ void __launch_bounds__(kReduceThreads) k_bbox(const float4 *__restrict__ pos4, int n, uint32_t *bb) {
    __shared__ uint32_t s[6][kReduceThreads / 32];
    float lo[3] = {3.402823466e+38f, 3.402823466e+38f, 3.402823466e+38f};
    float hi[3] = {-3.402823466e+38f, -3.402823466e+38f, -3.402823466e+38f};
#pragma unroll 4
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = __ldg(pos4 + i);
        lo[0] = fminf(lo[0], p.x);
        lo[1] = fminf(lo[1], p.y);
        lo[2] = fminf(lo[2], p.z);
        hi[0] = fmaxf(hi[0], p.x);
        hi[1] = fmaxf(hi[1], p.y);
        hi[2] = fmaxf(hi[2], p.z);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, f2ord(lo[a]));
        const uint32_t h = __reduce_max_sync(0xffffffffu, f2ord(hi[a]));
        if (lane == 0) {
            s[a][warp] = l;
            s[3 + a][warp] = h;
        }
    }
    __syncthreads();
    if (warp < 6) {
        const uint32_t v = s[warp][lane < kReduceThreads / 32 ? lane : 0];
        const uint32_t r = warp < 3 ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
        if (lane == 0) {
            if (warp < 3) atomicMin(bb + warp, r);
            else atomicMax(bb + warp, r);
        }
    }
}

__global__ void k_tree_keys(const float4 *__restrict__ pos4, int n, int depth, const uint32_t *__restrict__ bb,
                            uint32_t *__restrict__ keys, uint32_t *__restrict__ vals, uint32_t *__restrict__ hist,
                            int passes) {
    __shared__ uint32_t sh[RadixSorter::kMaxPasses][256];
    for (int i = threadIdx.x; i < RadixSorter::kMaxPasses * 256; i += blockDim.x) (&sh[0][0])[i] = 0u;
    __syncthreads();
    const float lx = ord2f(bb[0]), ly = ord2f(bb[1]), lz = ord2f(bb[2]);
    const float hx = ord2f(bb[3]), hy = ord2f(bb[4]), hz = ord2f(bb[5]);
    float span = fmaxf(hx - lx, fmaxf(hy - ly, hz - lz));
    if (!(span > 0.f)) span = 1.f;
    const int cells = 1 << depth;
    const float scale = __fdiv_rn((float)cells, span);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 p = pos4[i];
        int qx = (int)__fmul_rn(__fsub_rn(p.x, lx), scale);
        int qy = (int)__fmul_rn(__fsub_rn(p.y, ly), scale);
        int qz = (int)__fmul_rn(__fsub_rn(p.z, lz), scale);
        qx = min(max(qx, 0), cells - 1);
        qy = min(max(qy, 0), cells - 1);
        qz = min(max(qz, 0), cells - 1);
        uint32_t k = morton3((uint32_t)qx, (uint32_t)qy, (uint32_t)qz);
        keys[i] = k;
        vals[i] = (uint32_t)i;
        for (int q = 0; q < passes; ++q) atomicAdd(&sh[q][(k >> (8 * q)) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) {
        uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
}

// ---- nodes from the sorted keys ------------------------------------------------
constexpr int kTreeThreads = 1024;  // particles per block of the three kernels
// Scanned over the particles: nodes, ints, nodes per level (D + 1), branches
// per level (D); D <= 10.
constexpr int kTreeSeqs = 2 + 11 + 10;
constexpr uint8_t kNoNodes = 0xff;

// The sorted keys.  After a sort whose look-back gave up they are in no order,
// and the rules below would make a tree without bounds on its nodes: then the
// particles' places stand for their keys, spread evenly over the key range, so
// that the tree is a whole one (of no meaning; the health word says so).
__device__ __noinline__ uint32_t place_key(int i, int n, int bits) {
    return (uint32_t)(((uint64_t)(uint32_t)i << bits) / (uint32_t)n);
}
struct TreeKeys {
    const uint32_t *k;
    const uint32_t *failed;
    int n, bits;
    bool bad;  // read once per kernel (load)
    __device__ __forceinline__ void load() { bad = *failed != 0u; }
    __device__ __forceinline__ uint32_t operator[](int i) const { return bad ? place_key(i, n, bits) : k[i]; }
};

struct TreeArgs {
    TreeKeys keys;
    const uint32_t *order;  // particle ids in key order
    int n, depth, leafcap, blocks;
    uint8_t *levels;        // [n] first | last << 4 level of the nodes starting at each particle, or kNoNodes
    int32_t *ints;          // [n] ints of the nodes starting at each particle
    int32_t *at_int, *at_node;  // [n] their first offset and data pointer
    int64_t *totals;        // [kTreeSeqs][blocks] block totals, scanned in place by the last block
    uint32_t *ticket;       // blocks of k_tree_mark that are done
    int32_t *tree, *level_nodes, *level_count, *list_slot, *parent, *arrived, *meta;
    int2 *node_range;       // by data pointer, leaves: (first particle in key order, count)
    int64_t level_cap, tree_cap, node_cap;
    uint32_t *health;
};

// Leading triplets shared by two keys of `depth` triplets.
__device__ __forceinline__ int shared_levels(uint32_t a, uint32_t b, int depth) {
    const uint32_t x = a ^ b;
    return x ? depth - 1 - (31 - __clz(x)) / 3 : depth;
}

// First index in (i, hi] whose key leaves i's run at `level` (hi when none
// does before it).
__device__ __forceinline__ int run_end(const TreeKeys &keys, uint32_t key, int i, int hi, int level, int depth) {
    int lo = i + 1;
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if (shared_levels(key, keys[mid], depth) >= level) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// First index of the run of i at `level`, not looked for before `lo`: steps
// back that double, then a binary search, since most runs are short.
__device__ __forceinline__ int run_start(const TreeKeys &keys, uint32_t key, int i, int lo, int level, int depth) {
    int in = i, out = lo - 1, step = 1;  // in: in the run; out: before it (or before lo)
    while (in - step >= lo) {
        if (shared_levels(key, keys[in - step], depth) < level) {
            out = in - step;
            break;
        }
        in -= step;
        step += step;
    }
    while (in - out > 1) {
        const int mid = out + ((in - out) >> 1);
        if (shared_levels(key, keys[mid], depth) >= level) in = mid;
        else out = mid;
    }
    return in;
}

__device__ __forceinline__ void unpack_levels(uint8_t v, int &first, int &last) {
    first = v & 15;
    last = v == kNoNodes ? -1 : v >> 4;  // none: an empty range
}

__global__ void __launch_bounds__(kTreeThreads) k_tree_mark(TreeArgs a) {
    __shared__ int32_t s_tot[kTreeSeqs];
    __shared__ bool s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i = blockIdx.x * kTreeThreads + tid;
    const int D = a.depth, n = a.n;
    a.keys.load();
    if (tid < kTreeSeqs) s_tot[tid] = 0;
    __syncthreads();
    int first = 0, last = -1, ints = 0;
    if (i < n) {
        const uint32_t key = a.keys[i];
        const int c = i ? shared_levels(a.keys[i - 1], key, D) : -1;
        bool nodes = c < D;
        if (nodes && c >= 0) {
            // the run of level c that holds i - 1 and i is a branch: it has
            // leafcap particles besides i within leafcap places of it
            const bool right = i + a.leafcap - 1 < n && shared_levels(a.keys[i + a.leafcap - 1], key, D) >= c;
            const bool left = i >= a.leafcap && shared_levels(a.keys[i - a.leafcap], key, D) >= c;
            if (!right && !left) {
                const int s = run_start(a.keys, key, i, max(i - a.leafcap, 0), c, D);
                const int e = run_end(a.keys, key, i, min(i + a.leafcap, n), c, D);
                nodes = e - s > a.leafcap;
            }
        }
        if (nodes) {
            const int far = i + a.leafcap;
            const int q = far < n ? shared_levels(key, a.keys[far], D) : -1;
            first = c + 1;
            last = max(first, min(D, q + 1));
            // the leaf's run ends within leafcap places unless it is cut off by the depth
            const int e = q >= last ? run_end(a.keys, key, far, n, last, D)
                                    : run_end(a.keys, key, i, min(far, n), last, D);
            ints = 10 * (last - first) + 2 + (e - i);
        }
        a.levels[i] = nodes ? (uint8_t)(first | (last << 4)) : kNoNodes;
        a.ints[i] = ints;
    }
    const int nodes = __reduce_add_sync(0xffffffffu, last - first + 1);
    const int wints = __reduce_add_sync(0xffffffffu, ints);
    if (lane == 0) {
        atomicAdd(&s_tot[0], nodes);
        atomicAdd(&s_tot[1], wints);
    }
    for (int l = 0; l <= D; ++l) {
        const unsigned on = __ballot_sync(0xffffffffu, first <= l && l <= last);
        const unsigned br = __ballot_sync(0xffffffffu, first <= l && l < last);
        if (lane == 0 && on) {
            atomicAdd(&s_tot[2 + l], __popc(on));
            if (br) atomicAdd(&s_tot[3 + D + l], __popc(br));
        }
    }
    __syncthreads();
    const int seqs = 3 + 2 * D;
    if (tid < seqs) a.totals[(size_t)tid * a.blocks + blockIdx.x] = s_tot[tid];
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    // the last block to get here: one warp scans each sequence of block totals
    __threadfence();
    if (tid == 0) *a.ticket = 0u;
    if (warp < seqs) {
        int64_t *t = a.totals + (size_t)warp * a.blocks;
        int64_t carry = 0;
        int64_t v = lane < a.blocks ? __ldcg(t + lane) : 0;
        for (int b = lane; b - lane < a.blocks; b += 32) {
            const int64_t next = b + 32 < a.blocks ? __ldcg(t + b + 32) : 0;
            int64_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (b < a.blocks) t[b] = carry + x - v;
            carry += __shfl_sync(0xffffffffu, x, 31);
            v = next;
        }
        if (lane == 0) {
            if (warp < 2) a.meta[1 + warp] = (int32_t)carry;
            else if (warp < 3 + D) a.level_count[warp - 2] = (int32_t)carry;
        }
    }
    if (tid < 16 && tid > D) a.level_count[tid] = 0;
}

__global__ void __launch_bounds__(kTreeThreads) k_tree_write(TreeArgs a) {
    __shared__ int32_t s_at[kTreeSeqs][32];  // first value of each warp
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i = blockIdx.x * kTreeThreads + tid;
    const int D = a.depth, seqs = 3 + 2 * D;
    a.keys.load();
    const unsigned lt = (1u << lane) - 1u;
    int first, last;
    unpack_levels(i < a.n ? a.levels[i] : kNoNodes, first, last);
    const bool has = last >= 0;
    if (!has) first = 0;
    const int nodes = has ? last - first + 1 : 0;
    const int ints = has ? a.ints[i] : 0;
    int xn = nodes, xi = ints;  // inclusive scans over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int yn = __shfl_up_sync(0xffffffffu, xn, o), yi = __shfl_up_sync(0xffffffffu, xi, o);
        if (lane >= o) {
            xn += yn;
            xi += yi;
        }
    }
    if (lane == 31) {
        s_at[0][warp] = xn;
        s_at[1][warp] = xi;
    }
    for (int l = 0; l <= D; ++l) {
        const unsigned on = __ballot_sync(0xffffffffu, first <= l && l <= last);
        const unsigned br = __ballot_sync(0xffffffffu, first <= l && l < last);
        if (lane == 0) {
            s_at[2 + l][warp] = __popc(on);
            if (l < D) s_at[3 + D + l][warp] = __popc(br);
        }
    }
    __syncthreads();
    if (warp < seqs) {
        const int v = s_at[warp][lane];
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        s_at[warp][lane] = (int32_t)a.totals[(size_t)warp * a.blocks + blockIdx.x] + x - v;
    }
    __syncthreads();
    const int dp0 = s_at[0][warp] + xn - nodes;
    const int off0 = s_at[1][warp] + xi - ints;
    const int64_t leaf_off = (int64_t)off0 + 10 * (last - first);
    // a node whose record or data pointer lies past the storage is left out
    // and flagged (k_tree_link leaves it out too)
    const bool fits = has && (int64_t)off0 + ints <= a.tree_cap && (int64_t)dp0 + nodes <= a.node_cap;
    if (has && !fits) raise_health(a.health, SPH_HEALTH_TREE_CAPACITY);
    if (has) {
        a.at_int[i] = off0;
        a.at_node[i] = dp0;
    }
    const uint32_t key = has ? a.keys[i] : 0u;
    for (int l = 0; l <= D; ++l) {
        const bool on = first <= l && l <= last, br = first <= l && l < last;
        const unsigned m_on = __ballot_sync(0xffffffffu, on), m_br = __ballot_sync(0xffffffffu, br);
        if (!on || !fits) continue;
        const int off = off0 + 10 * (l - first), dp = dp0 + (l - first);
        a.level_nodes[(size_t)l * a.level_cap + s_at[2 + l][warp] + __popc(m_on & lt)] = off;
        a.list_slot[dp] = br ? s_at[3 + D + l][warp] + __popc(m_br & lt) : -1;
        a.arrived[dp] = 0;
        if (l > first) a.parent[dp] = off - 10;
        else if (l == 0) a.parent[dp] = -1;
        int32_t *T = a.tree + off;
        T[1] = dp;
        if (br) {
            T[0] = 0;
            // the child that starts at this particle is the next record
            const int o = (int)((key >> (3 * (D - l - 1))) & 7u);
#pragma unroll
            for (int k = 0; k < 8; ++k) T[2 + k] = k == o ? off + 10 : -1;
        } else {
            const int cnt = ints - 2 - 10 * (last - first);
            T[0] = cnt;
            a.node_range[dp] = make_int2(i, cnt);
        }
    }
    // the leaves' particle ids, a warp per leaf
    for (unsigned m = __ballot_sync(0xffffffffu, fits); m; m &= m - 1u) {
        const int src = __ffs(m) - 1;
        const int64_t off = __shfl_sync(0xffffffffu, leaf_off, src) + 2;
        const int cnt = __shfl_sync(0xffffffffu, ints - 2 - 10 * (last - first), src);
        const int p0 = i - lane + src;
        for (int k = lane; k < cnt; k += 32) a.tree[off + k] = (int32_t)a.order[p0 + k];
    }
}

__global__ void __launch_bounds__(256) k_tree_link(TreeArgs a) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < 1 || i >= a.n) return;
    int first, last;
    unpack_levels(a.levels[i], first, last);
    if (last < 0 || first < 1) return;
    const int off = a.at_int[i], dp = a.at_node[i];
    a.keys.load();
    if ((int64_t)off + a.ints[i] > a.tree_cap || (int64_t)dp + (last - first + 1) > a.node_cap) return;
    const uint32_t key = a.keys[i];
    const int level = first - 1;  // the parent's
    const int s = run_start(a.keys, key, i, 0, level, a.depth);
    int pf, pl;
    unpack_levels(a.levels[s], pf, pl);
    const int poff = a.at_int[s] + 10 * (level - pf);
    a.tree[poff + 2 + (int)((key >> (3 * (a.depth - first))) & 7u)] = off;
    a.parent[dp] = poff;
}

}  // namespace

sph_status tree_alloc(sph_ctx *ctx) {
    TreeBuild &tb = ctx->tb;
    if (tb.bbox) return SPH_OK;
    const int n = ctx->n;
    sph_status s = sort_alloc(tb.sorter, n);
    if (s != SPH_OK) return s;
    const size_t blocks = (size_t)(n + kTreeThreads - 1) / kTreeThreads;
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t r) {
        if (e == cudaSuccess) e = r;
    };
    chk(cudaMalloc(&tb.levels, sizeof(uint8_t) * (size_t)n));
    chk(cudaMalloc(&tb.ints, sizeof(int32_t) * (size_t)n));
    chk(cudaMalloc(&tb.at_int, sizeof(int32_t) * (size_t)n));
    chk(cudaMalloc(&tb.at_node, sizeof(int32_t) * (size_t)n));
    chk(cudaMalloc(&tb.totals, sizeof(int64_t) * kTreeSeqs * blocks));
    chk(cudaMalloc(&tb.ticket, sizeof(uint32_t)));
    if (e == cudaSuccess) chk(cudaMemset(tb.ticket, 0, sizeof(uint32_t)));
    chk(cudaMalloc(&tb.bbox, sizeof(uint32_t) * 8));
    return cuda_status(e, "tree_alloc");
}

void tree_free(sph_ctx *ctx) {
    TreeBuild &tb = ctx->tb;
    sort_free(tb.sorter);
    cudaFree(tb.levels);
    cudaFree(tb.ints);
    cudaFree(tb.at_int);
    cudaFree(tb.at_node);
    cudaFree(tb.totals);
    cudaFree(tb.ticket);
    cudaFree(tb.bbox);
    cudaFree(tb.walk_queues);
    cudaFree(tb.kp4);
    cudaFree(tb.walk_counter);
    tb = TreeBuild();
}

sph_status launch_tree_build(sph_ctx *ctx, cudaStream_t st, bool withhold) {
    sph_status s = tree_alloc(ctx);
    if (s != SPH_OK) return s;
    TreeBuild &tb = ctx->tb;
    Tree &tr = ctx->tree;
    const int n = ctx->n;
    const int D = ctx->params.max_tree_depth;
    const int leafcap = std::min(ctx->params.max_children_in_leaf, n);  // more is the same
    const int bits = 3 * D;
    const int passes = (bits + 7) / 8;
    uint32_t *bb = (uint32_t *)tb.bbox;

    k_bbox_init<<<1, 32, 0, st>>>(bb);
    k_bbox<<<reduce_grid(n), kReduceThreads, 0, st>>>(ctx->pos4, n, bb);
    radix_clear(tb.sorter, n, bits, st);
    k_tree_keys<<<reduce_grid(n), kReduceThreads, 0, st>>>(ctx->pos4, n, D, bb, tb.sorter.keys[0], tb.sorter.vals[0],
                                                           tb.sorter.hist, passes);
    const int fin = radix_sort_pairs(tb.sorter, n, bits, st, ctx->health, withhold);
    TreeArgs a;
    a.keys = TreeKeys{tb.sorter.keys[fin], tb.sorter.failed, n, bits, false};
    a.order = tb.sorter.vals[fin];
    a.n = n;
    a.depth = D;
    a.leafcap = leafcap;
    a.blocks = (n + kTreeThreads - 1) / kTreeThreads;
    a.levels = tb.levels;
    a.ints = tb.ints;
    a.at_int = tb.at_int;
    a.at_node = tb.at_node;
    a.totals = tb.totals;
    a.ticket = tb.ticket;
    a.tree = tr.tree;
    a.level_nodes = tr.level_nodes;
    a.level_count = tr.level_count;
    a.list_slot = tr.list_slot;
    a.parent = tr.parent;
    a.arrived = tr.arrived;
    a.meta = tr.meta;
    a.node_range = tr.node_range;
    a.level_cap = tr.level_cap;
    a.tree_cap = tr.tree_cap;
    a.node_cap = tr.node_cap;
    a.health = ctx->health;
    tb.order = a.order;
    k_tree_mark<<<a.blocks, kTreeThreads, 0, st>>>(a);
    k_tree_write<<<a.blocks, kTreeThreads, 0, st>>>(a);
    k_tree_link<<<(n + 255) / 256, 256, 0, st>>>(a);

    // upper bounds of the level sizes: a level's nodes are children of the
    // branches above it, each of which holds more than leafcap particles
    tr.n_levels_host = D + 1;
    const int64_t branches = (int64_t)n / ((int64_t)leafcap + 1);
    int64_t bound = 1;
    for (int l = 0; l < 16; ++l) {
        tr.level_count_host[l] = (l <= D) ? (int)bound : 0;
        bound = std::max<int64_t>(1, std::min<int64_t>(n, 8 * std::min(bound, branches)));
    }
    tr.valid = true;
    return cuda_status(cudaGetLastError(), "tree build");
}

}  // namespace sph

extern "C" sph_status sph_selftest_tree_capacity(sph_ctx *ctx, void *stream) {
    using namespace sph;
    if (!ctx || ctx->params.tree_source != SPH_TREE_GPU) {
        set_error("sph_selftest_tree_capacity: needs a context with the GPU tree");
        return SPH_ERR_INVALID_ARG;
    }
    cudaSetDevice(ctx->device);
    const int64_t cap = ctx->tree.tree_cap;
    ctx->tree.tree_cap = 16;  // room for one branch record at most
    const sph_status s = launch_tree_build(ctx, (cudaStream_t)stream);
    ctx->tree.tree_cap = cap;
    ctx->tree.valid = false;  // the next tree build replaces the partial one
    return s;
}
