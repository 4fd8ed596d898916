// sph_hydro.cu -- density, acceleration and step passes for sm_100a.
//
// density      SPH/Shaders/density.metal:12-239        (Compute.cpp:179-208)
// acceleration SPH/Shaders/accelerations.metal:12-141  (Compute.cpp:210-240)
// step         SPH/Shaders/step.metal:12-46            (Compute.cpp:242-263)
// snapshot     SPH/Shaders/render.metal:49-66          (Compute.cpp:396-448)
//
// Particles are taken in sorted (Morton cell) order, and neighbour data are read
// from sorted, 16-byte records (sp4/sv4, then sA/sB/sC written by the density
// epilogue), so every cell's particles are one contiguous run of float4 loads
// instead of the reference's index-chased float3 gathers.
//
// Product build: the density pass searches once, over tiles of cells staged in
// shared memory, and writes every particle's neighbour list (k_lists); eight
// lanes a particle iterate h over the list (k_density_list) and sum the
// acceleration over the same list (k_acceleration_list), or over one that the
// acceleration tiles search for (k_acceleration_tile).  Particles that no tile
// or list serves are walked for, a warp each (k_density_deferred,
// k_acceleration_deferred; group_walk).
//
// Parity build: one thread a particle walks the reference's cells in its order
// (k_density, k_acceleration).  The reference's 128-entry per-thread neighbour
// cache (density.metal:67-70) is replaced by rescanning the same cell box with
// the same filters: the visited set and order are identical (density_particle),
// and no thread carries 1 KiB of local memory.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "sph_f32x2.cuh"
#include "sph_internal.h"

namespace sph {

namespace {

// Margin on the distance from a particle to a cell box: positions near 318 Mm
// carry ~3e-5 Mm of float32 rounding, and a particle's cell comes from
// floor(x / CELL_WIDTH); 2e-4 Mm keeps every particle of a cell inside its box.
constexpr float kCellMargin = 2e-4f;

// Square root of a pair distance.  The parity build keeps the correctly
// rounded sqrtf of the reference; the product uses the hardware reciprocal
// square root (within 2 ulp), a rounding-level difference.
__device__ __forceinline__ float pair_sqrt(float r2) {
#ifdef SPH_PARITY
    return sqrtf(r2);
#else
    return r2 > 1e-30f ? r2 * rsqrt_hw(r2) : 0.f;
#endif
}

// 1 / r for a pair at r = pair_sqrt(r2) > 0: the correctly rounded quotient
// in the parity build, the hardware reciprocal square root in the product.
__device__ __forceinline__ float pair_rinv(float r2, float r) {
#ifdef SPH_PARITY
    return 1.f / r;
#else
    (void)r;
    return rsqrt_hw(r2);
#endif
}

// a / b in the pair arithmetic: the correctly rounded quotient in the parity
// build, the hardware approximation (within 2 ulp) in the product.
__device__ __forceinline__ float pdiv(float a, float b) {
#ifdef SPH_PARITY
    return a / b;
#else
    return a * rcp_hw(b);
#endif
}

// Lanes per particle of the parity build's passes: one, which sums in the
// reference's sequential order.
constexpr int kParityLanes = 1;
// Lanes per particle of the deferred particles' walk, a whole warp: its cost
// is the walk over the thousands of cells of a box that no tile can hold, one
// look-up per lane at a time, and a few particles at the end of a pass are
// nothing but latency (N = 2e4, 3 particles: the density pass 434 us
// with 8 lanes a particle, 278 with 32).
constexpr int kWalkLanes = 32;

// Squared distance from (px, py, pz) to the box of cell (x, y, z), each axis
// gap shortened by the margin.
__device__ __forceinline__ float cell_gap2(float px, float py, float pz, int x, int y, int z) {
    const float w = kCellWidth;
    const float gx = fmaxf(fmaxf((float)x * w - px, px - (float)(x + 1) * w) - kCellMargin, 0.f);
    const float gy = fmaxf(fmaxf((float)y * w - py, py - (float)(y + 1) * w) - kCellMargin, 0.f);
    const float gz = fmaxf(fmaxf((float)z * w - pz, pz - (float)(z + 1) * w) - kCellMargin, 0.f);
    return gx * gx + gy * gy + gz * gz;
}

__global__ void k_gather(int n, const uint32_t *__restrict__ cidx, const float4 *__restrict__ pos4,
                         const float4 *__restrict__ vel4, float4 *__restrict__ sp4, float4 *__restrict__ sv4) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint32_t i = cidx[k];
    sp4[k] = pos4[i];
    sv4[k] = vel4[i];
}

// ---- neighbour walk shared by the lanes of one particle -------------------
//
// Each particle gets a group of L consecutive lanes (the parity build's one or
// the deferred walk's whole warp).  The group
// walks the particle's own cell box of radius 2h in the reference's order
// (x outer, z inner; sorted index within a cell): its lanes look up L cells
// at a time (cells farther than the search radius are not looked up), the
// particles of those cells are numbered consecutively, and lane `sub` takes
// every L-th of them.  So each lane sees a slice of exactly the candidates the
// reference's box walk visits, the lanes stay busy although a cell holds only
// a few particles.  Partial sums are combined across the
// group by a butterfly (every lane ends with the same bits).  With L = 1 the
// walk is the reference's sequential order exactly.

template <int L>
__device__ __forceinline__ unsigned group_mask(int lane) {
    return L == 32 ? 0xffffffffu : (((1u << L) - 1u) << (lane & ~(L - 1)));
}
template <int L>
__device__ __forceinline__ float group_sum(float v, unsigned gm) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(gm, v, o, L);
    return v;
}
template <int L>
__device__ __forceinline__ int group_sum_i(int v, unsigned gm) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(gm, v, o, L);
    return v;
}
template <int L>
__device__ __forceinline__ float group_max(float v, unsigned gm) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v = fmax_ref(v, __shfl_xor_sync(gm, v, o, L));
    return v;
}

// s_off / s_start: this warp's 32-entry scratch in shared memory; gbase =
// the group's first lane within the warp.
template <int L, class Body>
__device__ __forceinline__ void group_walk(float px, float py, float pz, float h, float r2cull,
                                           const uint2 *__restrict__ cells, int sub, unsigned gm, int gbase,
                                           uint32_t *s_off, uint32_t *s_start, Body &&body) {
    const CellBox b = cell_box(px, py, pz, h);
    const int ny = b.hi1 - b.lo1 + 1, nz = b.hi2 - b.lo2 + 1;
    const int nyz = ny * nz;
    const int nc = (b.hi0 - b.lo0 + 1) * nyz;
    for (int c0 = 0; c0 < nc; c0 += L) {
        const int c = c0 + sub;
        uint32_t st = 0u, cnt = 0u;
        if (c < nc) {
            const int ix = c / nyz, rem = c - ix * nyz;
            const int iy = rem / nz, iz = rem - iy * nz;
            const int x = b.lo0 + ix, y = b.lo1 + iy, z = b.lo2 + iz;
            if (cell_gap2(px, py, pz, x, y, z) <= r2cull) {
                const uint2 r = __ldg(cells + cell_index_of(x, y, z));
                if (r.x != 0xffffffffu) {
                    st = r.x;
                    cnt = r.y - r.x + 1u;
                }
            }
        }
        if (L == 1) {
            for (uint32_t k = st; k < st + cnt; ++k) body(k);
            continue;
        }
        uint32_t inc = cnt;
#pragma unroll
        for (int o = 1; o < L; o <<= 1) {
            const uint32_t y = __shfl_up_sync(gm, inc, o, L);
            if (sub >= o) inc += y;
        }
        const uint32_t tot = __shfl_sync(gm, inc, L - 1, L);
        if (tot == 0u) continue;
        s_off[gbase + sub] = inc - cnt;
        s_start[gbase + sub] = st;
        __syncwarp(gm);
        for (uint32_t j = sub; j < tot; j += L) {
            int q = 0;  // the last cell whose first candidate number is <= j
#pragma unroll
            for (int step = L / 2; step > 0; step >>= 1)
                if (s_off[gbase + q + step] <= j) q += step;
            body(s_start[gbase + q] + (j - s_off[gbase + q]));
        }
        __syncwarp(gm);
    }
}

// Collect, in the walk's order, the indices of the candidates of the
// particle's box of radius 2 hbox that pass `test` into the group's list in
// shared memory: each round of L candidates is ordered by a ballot, so the
// list keeps the reference's visiting order.  Whenever the list could
// overflow, `drain(count)` consumes it and the list restarts; a drain that
// returns false keeps the list instead and the walk only counts from then on,
// so the return value (the number of candidates found) may exceed cap.
template <int L, class Test, class Drain>
__device__ __forceinline__ int group_collect(float px, float py, float pz, float hbox, float r2cull,
                                             const uint2 *__restrict__ cells, int sub, unsigned gm, int gbase,
                                             uint32_t *s_off, uint32_t *s_start, uint32_t *list, int cap,
                                             Test &&test, Drain &&drain) {
    const CellBox b = cell_box(px, py, pz, hbox);
    const int ny = b.hi1 - b.lo1 + 1, nz = b.hi2 - b.lo2 + 1;
    const int nyz = ny * nz;
    const int nc = (b.hi0 - b.lo0 + 1) * nyz;
    int cnt = 0;
    for (int c0 = 0; c0 < nc; c0 += L) {
        const int c = c0 + sub;
        uint32_t st = 0u, n_in = 0u;
        if (c < nc) {
            const int ix = c / nyz, rem = c - ix * nyz;
            const int iy = rem / nz, iz = rem - iy * nz;
            const int x = b.lo0 + ix, y = b.lo1 + iy, z = b.lo2 + iz;
            if (cell_gap2(px, py, pz, x, y, z) <= r2cull) {
                const uint2 r = __ldg(cells + cell_index_of(x, y, z));
                if (r.x != 0xffffffffu) {
                    st = r.x;
                    n_in = r.y - r.x + 1u;
                }
            }
        }
        uint32_t inc = n_in;
#pragma unroll
        for (int o = 1; o < L; o <<= 1) {
            const uint32_t y = __shfl_up_sync(gm, inc, o, L);
            if (sub >= o) inc += y;
        }
        const uint32_t tot = __shfl_sync(gm, inc, L - 1, L);
        if (tot == 0u) continue;
        s_off[gbase + sub] = inc - n_in;
        s_start[gbase + sub] = st;
        __syncwarp(gm);
        for (uint32_t j0 = 0; j0 < tot; j0 += L) {
            const uint32_t j = j0 + sub;
            uint32_t k = 0u;
            bool hit = false;
            if (j < tot) {
                int q = 0;  // the last cell whose first candidate number is <= j
#pragma unroll
                for (int step = L / 2; step > 0; step >>= 1)
                    if (s_off[gbase + q + step] <= j) q += step;
                k = s_start[gbase + q] + (j - s_off[gbase + q]);
                hit = test(k);
            }
            const unsigned hm = (__ballot_sync(gm, hit) >> gbase) & (L == 32 ? 0xffffffffu : ((1u << L) - 1u));
            const int nh = __popc(hm);
            if (cnt + nh > cap) {
                if (!drain(cnt)) {
                    cnt += nh;  // overflow: keep counting, store nothing more
                    continue;
                }
                cnt = 0;
            }
            if (hit) list[cnt + __popc(hm & ((1u << sub) - 1u))] = k;
            cnt += nh;
            __syncwarp(gm);
        }
        __syncwarp(gm);
    }
    return cnt;
}

// Neighbour lists that the density tiles leave for the acceleration pass, so
// that it need not look for the same neighbours again.  A particle's list
// holds every particle within 2 kTileListReach x max(its h, the other's h),
// the h at the start of the density pass (the last h a list was built for, its
// own), as far as its box of cells reaches: all pairs the acceleration pass can
// accept, unless a neighbour's h has outgrown its start by more than
// kTileListReach: the largest such h is kept per 64-cell unit in `grown`, and a
// particle's list is complete as long as that h reaches no further than it.
struct NeighbourLists {
    uint32_t *entries;  // [last - first][kTileList] sorted indices
    int first, last;    // the sorted particles whose lists are in it
    uint8_t *count;     // [n], kNoList: none
    float *reach2;      // [n] everything within this squared distance is listed;
                        // negative: nothing else is (no use to the acceleration pass)
    int *grown;         // [units] float bits, 0: none
};
constexpr uint8_t kNoList = 0xff;

struct DensityArgs {
    int n;
    const uint32_t *cidx;
    const uint32_t *skey;  // sorted cell keys (tile passes)
    const uint2 *cells;
    const uint2 *octets;   // 8-cell octet ranges and
    const uint2 *units;    // 64-cell unit ranges (coarse tiles)
    uint8_t *cflags;       // per 512-cell block: holds a coarse-tile particle
    int coarse;            // coarse tiles on
    uint8_t *mode;         // [n] the pass that takes each sorted particle (kMode*), written by k_density_plan
    float *first_h;        // [n] the largest h its first sweep can have, and
    float *start_h;        // [n] the h its staged box is built for, written by k_density_plan
    NeighbourLists lists;  // out, for the acceleration pass
    const float4 *sp4, *sv4;
    float *h, *rho, *f, *P, *c, *B;
    const float *u;
    const int32_t *mat;
    const uint8_t *active;
    float4 *sA, *sB, *sC;
    int32_t *globals;
    uint32_t *health;
    EosTables eos;
    float eta;            // convergence tolerance of the h iteration (DENSITY_ETA in the reference)
    const float *seed;    // learned starting h per particle, or null (the plain guess, h itself)
    float *nn_out;        // neighbour count per particle, or null
    uint32_t *stats;      // [0] sweeps, [1] fallbacks, [2] most sweeps, [3] particles; or null
};

// A learned seed whose first sweep moves h by more than this relative amount
// is abandoned for the plain initial guess.
constexpr float kSeedFallback = 0.05f;

// Per-particle neighbour list of the density pass, in shared memory: the
// sorted indices of every candidate within kListReach x the smoothing length
// the list was built for, in the reference's visiting order.  The iteration's
// sweeps and the gradient sweep read it instead of walking the cells again
// (recomputing each distance exactly as the walk does); a sweep whose radius
// the list does not cover rebuilds it, and a particle whose list overflows
// walks the cells in every sweep.
constexpr int kListMax = 192;       // list entries per particle
// particles per block: 16 groups, but never fewer than a warp's worth of lanes
template <int L>
__host__ __device__ constexpr int parts_per_block() { return 16 * L >= 32 ? 16 : 32 / L; }
constexpr float kListReach = 1.15f; // list radius / (2 h)

__device__ __forceinline__ void mark_grown(const DensityArgs &a, uint32_t p, float h);

// density.metal:12-239 for one sorted particle per lane group.  The group
// keeps the reference's per-particle iteration state (h, the int max_h, the
// cached scan's h and neighbour count) identically in all its lanes.
// w_off / w_start: the warp's 32-entry walk scratch; list: the group's
// kListMax-entry neighbour list.
template <int L>
__device__ __forceinline__ void density_particle(const DensityArgs &a, int index, int sub, unsigned gm, int gbase,
                                                 uint32_t *w_off, uint32_t *w_start, uint32_t *list) {
    const uint32_t ind = a.cidx[index];
    const float4 me = a.sp4[index];
    const float4 mv = a.sv4[index];
    if (!a.active[ind]) {
        // density.metal:40-55: EOS only
        if (sub != 0) return;
        float2 pc = eos_lookup(a.eos, a.mat[ind], a.rho[ind], a.u[ind]);
        a.P[ind] = pc.x;
        a.c[ind] = pc.y;
        float hi = a.h[ind], rho = a.rho[ind], fi = a.f[ind];
        a.sA[index] = make_float4(me.x, me.y, me.z, hi);
        a.sB[index] = make_float4(mv.x, mv.y, mv.z, pc.y);
        a.sC[index] = make_float4(me.w, (fi * pc.x / (rho * rho)), rho, a.B[ind]);
        return;
    }
    const float px = me.x, py = me.y, pz = me.z, mi = me.w;
    const float h_plain = a.h[ind];
    float hi = h_plain;
    // a learned seed replaces the plain guess when it is finite and within a
    // factor two of it
    bool seeded = false;
    if (a.seed) {
        const float sd = a.seed[ind];
        if (sd >= 0.5f * h_plain && sd <= 2.f * h_plain && sd <= kMaxH) {
            hi = sd;
            seeded = true;
        }
    }
    bool first = true, fell_back = false;
    int sweeps = 0;
    int max_h = 0;  // an int in the reference (truncates h < 1 to 0)
    float h2x4 = 4.f * hi * hi;
    float h1 = 1.f / hi;
    float dens = 0.f;
    float eps = 1.f;
    int count = 0;
    // State of the reference's neighbour cache, which holds the neighbours of
    // the last full scan: that scan's h (box and filter), and its count capped
    // at N_NEIGHBOURS_ESTIM.  A "cached" sweep is a rescan with those filters.
    int nn = 0;
    float hs = hi, hs2x4 = h2x4;
    const uint2 *cells = a.cells;
    const float4 *sp4 = a.sp4;
    // the list: entries within sqrt(list_r2); n_list < 0 = none
    int n_list = -1;
    float list_r2 = 0.f;
    auto build = [&](float hb) {
        const float rl = 2.f * hb * kListReach;
        list_r2 = rl * rl;
        const float r2max = list_r2;
        n_list = group_collect<L>(
            px, py, pz, hb * kListReach, r2max, cells, sub, gm, gbase, w_off, w_start, list, kListMax,
            [&](uint32_t k) {
                const float4 q = __ldg(sp4 + k);
                const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
                return dx * dx + dy * dy + dz * dz <= r2max;
            },
            [](int) { return false; });
        __syncwarp(gm);
    };
    while (eps > a.eta && count < kMaxNR) {
        const bool cached = hi < (float)max_h && nn < kNeighbourCache;
        if (!cached) {
            hs = hi;
            hs2x4 = h2x4;
        }
        const float h2 = hi + hi;
        if (n_list < 0 || (n_list <= kListMax && hs2x4 > list_r2)) build(hs);
        float part = 0.f;
        int found = 0;
        if (n_list <= kListMax) {
#pragma unroll 4
            for (int i = sub; i < n_list; i += L) {
                const float4 q = __ldg(sp4 + list[i]);
                const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (r2 > hs2x4) continue;
                const float r = pair_sqrt(r2);
                if (cached && r > h2) continue;
                ++found;
                part += kernel_w(r, h1) * q.w;
            }
        } else {
            group_walk<L>(px, py, pz, hs, hs2x4, cells, sub, gm, gbase, w_off, w_start, [&](uint32_t k) {
                const float4 q = __ldg(sp4 + k);
                const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (r2 > hs2x4) return;
                const float r = pair_sqrt(r2);
                if (cached && r > h2) return;
                ++found;
                part += kernel_w(r, h1) * q.w;
            });
        }
        dens = group_sum<L>(part, gm);
        if (!cached) nn = min(group_sum_i<L>(found, gm), kNeighbourCache);
        float nh = fmin_ref(kResolutionEta * powf(mi / dens, 1.f / 3), kMaxH);
        nh = 0.5f * (hi + nh);
        eps = fabsf(nh - hi) / hi;
        ++sweeps;
        if (first && seeded && eps > kSeedFallback) {
            // the seed disagrees with its own first sweep: start again from
            // the plain guess, with the iteration state of a fresh start
            first = false;
            fell_back = true;
            hi = h_plain;
            h1 = 1.f / hi;
            h2x4 = 4.f * hi * hi;
            max_h = 0;
            nn = 0;
            eps = 1.f;
            continue;
        }
        first = false;
        if (eps > a.eta) {
            max_h = (int)fmax_ref((float)max_h, hi);
            hi = nh;
            h1 = 1.f / hi;
            h2x4 = 4.f * hi * hi;
            count++;
        }
    }
    // gradient sweep (density.metal:145-213): below N_NEIGHBOURS_ESTIM the
    // cached neighbours (last full scan) within 2h; above, a full scan at h
    // that adds to the converged density again
    const bool gcached = nn < kNeighbourCache;
    const float gh = gcached ? hs : hi;
    const float g2 = gcached ? hs2x4 : h2x4;
    const float h2 = hi + hi;
    const float vix = mv.x, viy = mv.y, viz = mv.z;
    const float4 *sv4 = a.sv4;
    float pdens = 0.f, dens_h = 0.f, vdiv = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
    auto grad = [&](uint32_t k, float r, float mj, float dx, float dy, float dz) {
        if (!gcached) pdens += kernel_w(r, h1) * mj;
        dens_h += mj * kernel_dwdh(r, h1);
        if (r > 1e-12f) {
            const float r1 = 1.f / r;
            const float4 vj = __ldg(sv4 + k);
            const float vx = vj.x - vix, vy = vj.y - viy, vz = vj.z - viz;
            const float sc = kernel_gradw_scale(r, h1);
            const float gx = sc * (dx * r1), gy = sc * (dy * r1), gz = sc * (dz * r1);
            vdiv += mj * (vx * gx + vy * gy + vz * gz);
            cx += mj * (vy * gz - vz * gy);
            cy += mj * (vz * gx - vx * gz);
            cz += mj * (vx * gy - vy * gx);
        }
    };
    if (n_list <= kListMax && g2 > list_r2) build(gh);
    if (n_list <= kListMax) {
#pragma unroll 4
        for (int i = sub; i < n_list; i += L) {
            const uint32_t k = list[i];
            const float4 q = __ldg(sp4 + k);
            const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (r2 > g2) continue;
            const float r = pair_sqrt(r2);
            if (gcached && r > h2) continue;
            grad(k, r, q.w, dx, dy, dz);
        }
    } else {
        group_walk<L>(px, py, pz, gh, g2, cells, sub, gm, gbase, w_off, w_start, [&](uint32_t k) {
            const float4 q = __ldg(sp4 + k);
            const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (r2 > g2) return;
            const float r = pair_sqrt(r2);
            if (gcached && r > h2) return;
            grad(k, r, q.w, dx, dy, dz);
        });
    }
    if (!gcached) dens += group_sum<L>(pdens, gm);
    dens_h = group_sum<L>(dens_h, gm);
    vdiv = group_sum<L>(vdiv, gm);
    cx = group_sum<L>(cx, gm);
    cy = group_sum<L>(cy, gm);
    cz = group_sum<L>(cz, gm);
    if (a.stats) {
        // counters of the iteration (one group member per particle)
        const unsigned am = __activemask();
        const uint32_t mine = sub == 0 ? 1u : 0u;
        const uint32_t sw = __reduce_add_sync(am, mine * (uint32_t)sweeps);
        const uint32_t fb = __reduce_add_sync(am, mine * (fell_back ? 1u : 0u));
        const uint32_t mx = __reduce_max_sync(am, mine * (uint32_t)sweeps);
        const uint32_t np = __reduce_add_sync(am, mine);
        if ((threadIdx.x & 31) == (uint32_t)(__ffs(am) - 1)) {
            atomicAdd(a.stats + 0, sw);
            if (fb) atomicAdd(a.stats + 1, fb);
            atomicMax(a.stats + 2, mx);
            atomicAdd(a.stats + 3, np);
        }
    }
    if (sub != 0) return;
    if (a.nn_out) a.nn_out[ind] = (float)nn;
    vdiv = fabsf(vdiv) / dens;
    float acurl = sqrtf(cx * cx + cy * cy + cz * cz) / dens;
    float fi = 1.f / (1.f + (hi / (3.f * dens)) * dens_h);
    float2 pc = eos_lookup(a.eos, a.mat[ind], dens, a.u[ind]);
    float bal = vdiv / (vdiv + acurl + 1e-4f * (pc.y / hi));
#ifndef SPH_PARITY
    mark_grown(a, (uint32_t)index, hi);
#endif
    a.h[ind] = hi;
    a.rho[ind] = dens;
    a.f[ind] = fi;
    a.P[ind] = pc.x;
    a.c[ind] = pc.y;
    a.B[ind] = bal;
    if (!(dens == dens) || !(pc.x == pc.x)) raise_health(a.health, SPH_HEALTH_NAN_DENSITY);
    a.sA[index] = make_float4(px, py, pz, hi);
    a.sB[index] = make_float4(vix, viy, viz, pc.y);
    a.sC[index] = make_float4(mi, (fi * pc.x / (dens * dens)), dens, bal);
}

#ifdef SPH_PARITY
// One lane group per sorted particle, every particle.
template <int L>
__global__ void __launch_bounds__(parts_per_block<L>() * L) k_density(DensityArgs a) {
    extern __shared__ uint32_t s_lists[];
    __shared__ uint32_t s_off[parts_per_block<L>() * L], s_start[parts_per_block<L>() * L];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, sub = lane & (L - 1), gbase = lane & ~(L - 1);
    const int index = t / L;
    if (index >= a.n) return;  // whole groups leave together
    if (t == 0) a.globals[1] = (int32_t)(kDT0 * 1 / kDtMin1);  // density.metal:34-36
    density_particle<L>(a, index, sub, group_mask<L>(lane), gbase, s_off + (threadIdx.x & ~31),
                        s_start + (threadIdx.x & ~31), s_lists + (size_t)(threadIdx.x / L) * kListMax);
}
#endif

// The particles the tile pass handed on (sorted indices idx[0, *count)),
// one lane group each, grid-stride.
template <int L>
__global__ void __launch_bounds__(parts_per_block<L>() * L)
    k_density_deferred(DensityArgs a, const uint32_t *__restrict__ idx, const uint32_t *__restrict__ count) {
    extern __shared__ uint32_t s_lists[];
    __shared__ uint32_t s_off[parts_per_block<L>() * L], s_start[parts_per_block<L>() * L];
    const int lane = threadIdx.x & 31, sub = lane & (L - 1), gbase = lane & ~(L - 1);
    const uint32_t cnt = *count;
    constexpr int per_block = parts_per_block<L>();
    for (uint32_t base = blockIdx.x * per_block; base < cnt; base += gridDim.x * per_block) {
        const uint32_t j = base + threadIdx.x / L;
        if (j < cnt)
            density_particle<L>(a, (int)idx[j], sub, group_mask<L>(lane), gbase, s_off + (threadIdx.x & ~31),
                                s_start + (threadIdx.x & ~31), s_lists + (size_t)(threadIdx.x / L) * kListMax);
    }
}

// ---- density over neighbour lists (product build) ---------------------------
//
// k_lists finds every particle's neighbours over tiles: a tile is an aligned
// Morton block of cells -- 64 cells (4 x 4 x 4), or, where such a block holds
// many particles, its 16-cell quarters or its octets -- so its particles are
// one contiguous run of the sorted order.  A CTA takes tiles from a ticket
// counter; per tile it stages, once, every particle of the box of cells that
// the tile's lists can reach (position, sorted index, starting h) into shared
// memory, in cell order x-major, then y, z innermost, so a row of cells along z
// is one contiguous run of staged slots.  Warps then take the tile's particles
// four at a time (lists_tile_warp) and write their lists.
//
// k_density_list iterates h from the lists alone, eight lanes a particle: the
// distances and masses stay in registers through the sweeps, and no sweep
// touches memory.  The acceleration pass reads the same lists.  (Search and
// iteration were one kernel, whose registers and shared memory left room for
// 24 warps per SM and whose 77 KB of code did not fit the instruction caches:
// N = 1e6, 3.05 ms the pass; the two kernels 2.06.)
//
// A particle whose list box reaches more than kTileReach units beyond its own,
// whose h is at least MAX_SMOOTHING_LENGTH (where the reference's neighbour
// cache comes into play), whose list overflows or whose growing h leaves its
// list is handed to k_density_deferred, which runs the per-particle walk above;
// so is every particle of a tile whose box exceeds the shared-memory budget.
#ifndef SPH_TILE_LANES
#define SPH_TILE_LANES 8
#endif
constexpr int kTileLanes = SPH_TILE_LANES;                  // lanes per particle
constexpr int kTileGpw = 32 / kTileLanes;                   // particles per warp
constexpr int kTileCellsMax = 1024;                         // units of a tile's staged box
#ifndef SPH_TILE_REACH_CELLS
#define SPH_TILE_REACH_CELLS 3
#endif
constexpr int kTileReach = SPH_TILE_REACH_CELLS;            // units a list box may extend past its own
constexpr int kTileList = 192;                              // list entries per particle
#ifndef SPH_TILE_LIST_REACH
#define SPH_TILE_LIST_REACH 1.08f
#endif
// list radius / (2 h), for the h that k_density_plan expects: a list costs as
// much as several sweeps, and a particle whose h outgrows it is walked for on
// its own
constexpr float kTileListReach = SPH_TILE_LIST_REACH;
// staged box radius / (2 h): room for the second, wider search of a particle
// that finds too few neighbours
constexpr float kTileStageReach = 1.25f;
// list and box radius / (2 h) of lists that serve a first sweep and no more, and
// the h whose kTileListReach is that, for h = 1
constexpr float kFirstReach = 1.00001f, kNarrow = kFirstReach / kTileListReach;
// neighbours within 2 kTileListReach h of a particle at its fixed point,
// 4/3 pi (2 RESOLUTION_ETA kTileListReach)^3
constexpr float kListFull = 4.18879f * 8.f * kResolutionEta * kResolutionEta * kResolutionEta * kTileListReach *
                            kTileListReach * kTileListReach;
// Neighbours a particle's lanes keep in registers, as pairs per lane, through
// the sweeps of its iteration; longer lists are read again in every sweep.
constexpr int kRegPairs = 6;
constexpr int kRegList = 2 * kRegPairs * kTileLanes;        // 96 (a list holds ~85)

// CTAs of the tile passes.  Cell tiles: three of 320 threads fill an SM's
// registers (64 each) and shared memory.  Coarse tiles stage more per particle,
// and one that overflows is taken again unit by unit, a few particles at a
// time: two larger CTAs (N = 1e5, whose boxes are mostly coarse, two steps: 2032
// us with the cell tiles' shape, 1791 with this; the cell tiles with this shape
// 2.18 ms at N = 1e6 instead of 2.02).
template <int U>
struct ListTile {
    static constexpr int kThreads = U == 0 ? 320 : 512;
    static constexpr int kCtas = U == 0 ? 3 : 2;      // per SM
    static constexpr int kStage = U == 0 ? 2944 : 4096;  // staged particles
};
template <int U>
struct ListShared {
    float4 pos[ListTile<U>::kStage];       // staged (x, y, z, m)
    uint32_t gidx[ListTile<U>::kStage];    // staged sorted index
    float hs[ListTile<U>::kStage];         // staged starting h
    uint32_t off[kTileCellsMax + 1];       // first staged slot of each box unit; off[units] = staged count
    int box[6];                            // staged box: lo x y z, hi x y z (unwrapped cell coordinates)
    int hmax_bits;                         // largest staged starting h (float bits; h > 0)
    uint32_t wsum[ListTile<U>::kThreads / 32];
    uint32_t rows[ListTile<U>::kThreads / 32][32];  // each warp's rows: staged slot minus flat index
    uint32_t start, end, tile, next;
    int defer_all;
    int need;                              // some particle of the range needs the warp pass
    int narrow;                            // lists of first sweeps only
    float reach;                           // staged box radius / (2 h), h the first sweep's when narrow
};

// The list box of a tile particle at smoothing length hb: the cells within
// 2 hb reach, widened by 1e-3 of a cell so that float rounding of the cell
// coordinates (|x| / CELL_WIDTH < 2^12, a few 1e-4 of a cell) never drops a
// cell.
__device__ __forceinline__ void tile_box(float px, float py, float pz, float hb, CellBox &b,
                                         float reach = kTileListReach) {
    constexpr float iw = 1.f / kCellWidth;
    constexpr float widen = 1e-3f;
    const float rl = 2.f * hb * reach;
    b.lo0 = (int)floorf((px - rl) * iw - widen);
    b.lo1 = (int)floorf((py - rl) * iw - widen);
    b.lo2 = (int)floorf((pz - rl) * iw - widen);
    b.hi0 = (int)floorf((px + rl) * iw + widen);
    b.hi1 = (int)floorf((py + rl) * iw + widen);
    b.hi2 = (int)floorf((pz + rl) * iw + widen);
}

// Units (of 1 << shift cells) from cell lo to cell hi, or a number past any
// limit where these span more than the grid's period: particles of one tile are
// only alike modulo the grid, and a box that holds two of them a period apart
// would stage the cells between them twice.  (64 bits: lo and hi are anything.)
__device__ __forceinline__ int box_extent(int lo, int hi, int shift) {
    const int64_t e = (int64_t)(hi >> shift) - (lo >> shift) + 1;
    return e > (kCellsPerDim >> shift) ? 1 << 20 : (int)e;
}
__device__ __forceinline__ int64_t box_units(int nx, int ny, int nz) { return (int64_t)nx * ny * nz; }

// The particle's h is final: note it when the lists of its neighbours may lack
// it (a little early, for the rounding of the lists' squared reach; NaN counts
// as grown).
__device__ __forceinline__ void mark_grown(const DensityArgs &a, uint32_t p, float h) {
    if (!(h <= (kTileListReach - 1e-4f) * a.start_h[p]))
        atomicMax(a.lists.grown + (a.skey[p] >> (3 * kUnitShift)), __float_as_int(h));
}

// Tiling units of the staged box: cells (shift 0, the cell tiles), 2 x 2 x 2
// octets (shift 1) or 4 x 4 x 4-cell units (shift 2) for the coarse tiles,
// which take the octets whenever their box has few enough of them: finer
// units stage fewer particles and trim the lists' rows closer (h of 2 cells,
// reach 5: half the staged particles), while at a reach of 7 cells and more
// their 200 rows cost more than they trim.
template <int U>
__device__ __forceinline__ int unit_shift(const int (&box)[6]) {
    if (U == 0) return 0;
    return box_units(box_extent(box[0], box[3], 1), box_extent(box[1], box[4], 1), box_extent(box[2], box[5], 1)) <=
                   kTileCellsMax
               ? 1
               : kUnitShift;
}
// The (first, last) sorted range of unit (x, y, z); first is 0xffffffff when
// it is empty.
__device__ __forceinline__ uint2 unit_range(const uint2 *cells, const uint2 *octets, const uint2 *units, int shift,
                                            int x, int y, int z) {
    const int mask = (kCellsPerDim >> shift) - 1;
    const uint2 *t = shift == 0 ? cells : shift == 1 ? octets : units;
    return __ldg(t + morton3((uint32_t)(x & mask), (uint32_t)(y & mask), (uint32_t)(z & mask)));
}

// Whether a cell box reaches at most kTileReach tiling units (cells for U = 0,
// 64-cell units for U = kUnitShift) past the unit of cell (ox, oy, oz).
template <int U>
__device__ __forceinline__ bool within_reach(int ox, int oy, int oz, const CellBox &b) {
    return (ox >> U) - (b.lo0 >> U) <= kTileReach && (b.hi0 >> U) - (ox >> U) <= kTileReach &&
           (oy >> U) - (b.lo1 >> U) <= kTileReach && (b.hi1 >> U) - (oy >> U) <= kTileReach &&
           (oz >> U) - (b.lo2 >> U) <= kTileReach && (b.hi2 >> U) - (oz >> U) <= kTileReach;
}

// The pass that takes a density particle whose iteration starts from list
// radius 2 hb kTileListReach: 0 the cell tiles, kUnitShift the coarse tiles
// (a box past kTileReach cells, within kTileReach units), -1 the per-particle
// pass (h at MAX_H, where the reference's neighbour cache comes into play, or
// coarse tiles off).
__device__ __forceinline__ int density_mode(float px, float py, float pz, float hb, int coarse) {
    if (!(hb < kMaxH)) return -1;
    constexpr float iw = 1.f / kCellWidth;
    CellBox b;
    tile_box(px, py, pz, hb, b);
    const int ox = (int)floorf(px * iw), oy = (int)floorf(py * iw), oz = (int)floorf(pz * iw);
    if (within_reach<0>(ox, oy, oz, b)) return 0;
    if (coarse && within_reach<kUnitShift>(ox, oy, oz, b)) return kUnitShift;
    return -1;
}

// Staging: a warp copies the particles of its lanes' units (cnt and first of
// PER consecutive units per lane), which are consecutive
// staged slots from the warp's first: 32 slots at a time, each lane finding the
// lane and unit its slot belongs to, so that a unit with many particles is
// shared out.  excl, incl: the lane's slots within the warp.  copy(slot
// within the warp's, sorted index, unit counted from the warp's first).
template <int PER, class Copy>
__device__ __forceinline__ void stage_units(const uint32_t (&cnt)[PER], const uint32_t (&first)[PER], uint32_t excl,
                                            uint32_t incl, int lane, Copy &&copy) {
    constexpr unsigned kFull = 0xffffffffu;
    const uint32_t total = __shfl_sync(kFull, incl, 31);
#pragma unroll 2
    for (uint32_t vb = 0; vb < total; vb += 32u) {
        const uint32_t v = vb + (uint32_t)lane;
        int j = 0;  // the last lane whose first slot is <= v
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
            const uint32_t e = __shfl_sync(kFull, excl, j + step);
            if (e <= v) j += step;
        }
        uint32_t at = v - __shfl_sync(kFull, excl, j);
        uint32_t g = 0u;
        int unit = 0;
        bool found = false;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const uint32_t c = __shfl_sync(kFull, cnt[k], j), f = __shfl_sync(kFull, first[k], j);
            if (!found) {
                if (at < c) {
                    g = f + at;
                    unit = PER * j + k;
                    found = true;
                } else {
                    at -= c;
                }
            }
        }
        if (v < total) copy(v, g, unit);
    }
}

// The starting h of an active particle's iteration (the learned seed when it
// is accepted, as in density_particle) and the h its staged box is built for.
__device__ __forceinline__ float tile_start_h(const DensityArgs &a, uint32_t ind, float h_plain, bool &seeded) {
    seeded = false;
    if (a.seed) {
        const float sd = a.seed[ind];
        if (sd >= 0.5f * h_plain && sd <= 2.f * h_plain && sd <= kMaxH) {
            seeded = true;
            return sd;
        }
    }
    return h_plain;
}

// The pass that takes a sorted particle, decided once per pass by tile_plan
// from the particle's starting h: the density pass changes h as it goes, so a
// second look could give a particle to two passes (10 % of them on a 2e5
// impact) or to none.
constexpr uint8_t kModeWalk = 0xfe;      // the per-particle pass
constexpr uint8_t kModeInactive = 0xff;  // no neighbours needed (cell-tile pass)
constexpr uint8_t kModeList = 0xfd;      // acceleration: the density pass's list
static_assert(kUnitShift < kModeWalk, "0 and kUnitShift: the tile passes");

// A warp: the tiles of the 128-cell block `blk` (the cells whose keys differ
// in the low seven bits, 4 x 4 x 8), four cells per lane, so an octet is two
// lanes, a 16-cell quarter of a half four, a 64-cell half sixteen: the block
// is one tile when it holds at most big_max particles, else each half is one
// when it holds at most block_max, else each quarter when it holds at most
// half_max, else each octet.  (first, one past last) per tile, in ticket
// order; ctr[0] counts tiles.
__device__ __forceinline__ void plan_block(uint32_t blk, const uint2 *cells, uint2 *tiles, uint32_t *ctr,
                                           uint32_t block_max, uint32_t half_max, uint32_t big_max, int lane) {
    constexpr unsigned kFull = 0xffffffffu;
    uint32_t f = 0xffffffffu, l = 0u;
    const uint4 *c4 = reinterpret_cast<const uint4 *>(cells + (size_t)blk * 128u + 4u * (uint32_t)lane);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const uint4 r = __ldg(c4 + j);
        if (r.x != 0xffffffffu) f = min(f, r.x), l = max(l, r.y + 1u);
        if (r.z != 0xffffffffu) f = min(f, r.z), l = max(l, r.w + 1u);
    }
    uint32_t first = 0u, end = 0u;  // the tile this lane leads
    bool fits = false;              // a larger block already holds the lane's cells
    uint32_t lf[5], ll[5];          // ranges of 2, 4, 8, 16 and 32 lanes
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        f = min(f, __shfl_xor_sync(kFull, f, 1 << k));
        l = max(l, __shfl_xor_sync(kFull, l, 1 << k));
        lf[k] = f;
        ll[k] = l;
    }
    auto take = [&](int k, uint32_t most) {
        if (fits || ll[k] <= lf[k] || ll[k] - lf[k] > most) return;
        fits = true;
        if ((lane & ((2 << k) - 1)) == 0) {
            first = lf[k];
            end = ll[k];
        }
    };
    take(4, big_max);
    take(3, block_max);
    take(1, half_max);
    take(0, 0xffffffffu);
    const unsigned m = __ballot_sync(kFull, end > first);
    uint32_t at = 0u;
    if (lane == 0) at = atomicAdd(ctr, (uint32_t)__popc(m));
    at = __shfl_sync(kFull, at, 0);
    if (end > first) tiles[at + (uint32_t)__popc(m & ((1u << lane) - 1u))] = make_uint2(first, end);
}

// One thread per sorted particle: its pass (Mode(p), which also flags the
// 512-cell blocks that hold a coarse-tile particle), and, a warp per occupied
// 128-cell block that starts among its particles, the tiles.  (With one thread
// per block, whose 128 cell reads ran one after another, the tiles alone took
// 20 us at N = 1e6.)
template <class Mode>
__device__ __forceinline__ void tile_plan(int n, const uint32_t *skey, const uint2 *cells, uint8_t *cflags,
                                          uint8_t *mode, uint2 *tiles, uint32_t *ctr, uint32_t block_max,
                                          uint32_t half_max, uint32_t big_max, Mode &&of) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint32_t key = 0u;
    bool start = false;
    if (k < n) {
        key = skey[k];
        start = k == 0 || ((skey[k - 1] ^ key) >> 7) != 0u;
        const uint8_t m = of(k);
        mode[k] = m;
        if (m == kUnitShift) cflags[key >> (3 * kUnitShift + 3)] = 1;
    }
    for (unsigned s = __ballot_sync(0xffffffffu, start); s; s &= s - 1u)
        plan_block(__shfl_sync(0xffffffffu, key, __ffs(s) - 1) >> 7, cells, tiles, ctr, block_max, half_max, big_max,
                   lane);
}

__global__ void __launch_bounds__(256) k_density_plan(DensityArgs a, uint2 *tiles, uint32_t *ctr, uint32_t block_max,
                                                      uint32_t half_max, uint32_t big_max) {
    if (blockIdx.x == 0 && threadIdx.x == 0)
        a.globals[1] = (int32_t)(kDT0 * 1 / kDtMin1);  // density.metal:34-36
    tile_plan(a.n, a.skey, a.cells, a.cflags, a.mode, tiles, ctr, block_max, half_max, big_max, [&](int p) -> uint8_t {
        const uint32_t ind = a.cidx[p];
        const float4 me = a.sp4[p];
        const float h_plain = a.h[ind];
        const bool on = a.active[ind];
        bool seeded;
        float hb = fmaxf(tile_start_h(a, ind, h_plain, seeded), h_plain);
        a.first_h[p] = hb;
        // the list is built for the h the iteration is on its way to, as the
        // last pass's density (moved on by the step) has it
        if (on && hb < kMaxH) {
            const float to = kResolutionEta * cbrtf(me.w / a.rho[ind]);
            hb = fmaxf(hb, fminf(fminf(to, 1.2f * hb), 0.999f * kMaxH));
        }
        a.start_h[p] = hb;
        a.lists.count[p] = kNoList;
        if (!on) return kModeInactive;
        const int m = density_mode(me.x, me.y, me.z, hb, a.coarse);
        return m < 0 ? kModeWalk : (uint8_t)m;
    });
}

// Coarse tiles: at the first sorted particle of every 512-cell block (2 x 2 x
// 2 units) that a cell-tile pass flagged, the block's (first, one past last)
// sorted range; the flag is cleared for the next pass.  ctr[0] counts tiles.
__global__ void k_coarse_starts(int n, const uint32_t *__restrict__ skey, const uint2 *__restrict__ units,
                                uint8_t *__restrict__ flags, uint2 *__restrict__ tiles, uint32_t *ctr) {
    constexpr int kShift = 3 * kUnitShift + 3;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t blk = skey[k] >> kShift;
    if (k > 0 && (skey[k - 1] >> kShift) == blk) return;
    if (!flags[blk]) return;
    flags[blk] = 0;
    uint32_t l = (uint32_t)k + 1u;
    for (int j = 0; j < 8; ++j) {
        const uint2 r = units[blk * 8u + (uint32_t)j];
        if (r.x != 0xffffffffu) l = max(l, r.y + 1u);
    }
    tiles[atomicAdd(ctr, 1u)] = make_uint2((uint32_t)k, l);
}

// 1 / (4 pi h^3), h1 = 1 / h: the norm of the cubic spline summed as
// (2 - q)+^3 - 4 (1 - q)+^3.
__device__ __forceinline__ float kernel_norm(float h1) { return 0.25f * kPi1 * h1 * h1 * h1; }

// Where the spheres of a warp's four particles can reach, as one box of
// centres and the largest radius (their z ranges row by row would be four
// times the work for few slots less: the four are neighbours in cell order).
struct Reach4 {
    float x0, x1, y0, y1, z0, z1, r2;
    // r2 < 0: a group that takes no part
    __device__ __forceinline__ Reach4(float px, float py, float pz, float rr) {
        constexpr unsigned kFull = 0xffffffffu;
        constexpr int L = kTileLanes;
        const float big = 3e38f;
        const bool on = rr >= 0.f;
        x0 = on ? px : big, y0 = on ? py : big, z0 = on ? pz : big;
        x1 = on ? px : -big, y1 = on ? py : -big, z1 = on ? pz : -big;
        r2 = rr;
#pragma unroll
        for (int o = L; o < 32; o <<= 1) {
            x0 = fminf(x0, __shfl_xor_sync(kFull, x0, o));
            y0 = fminf(y0, __shfl_xor_sync(kFull, y0, o));
            z0 = fminf(z0, __shfl_xor_sync(kFull, z0, o));
            x1 = fmaxf(x1, __shfl_xor_sync(kFull, x1, o));
            y1 = fmaxf(y1, __shfl_xor_sync(kFull, y1, o));
            z1 = fmaxf(z1, __shfl_xor_sync(kFull, z1, o));
            r2 = fmaxf(r2, __shfl_xor_sync(kFull, r2, o));
        }
    }
    // The z range of the row (x, y) of units (w wide, iw = 1 / w) that a sphere
    // can reach; false when none does.
    __device__ __forceinline__ bool row(int x, int y, float w, float iw, int &zl, int &zh) const {
        const float gx = fmaxf(fmaxf((float)x * w - x1, x0 - (float)(x + 1) * w) - kCellMargin, 0.f);
        const float gy = fmaxf(fmaxf((float)y * w - y1, y0 - (float)(y + 1) * w) - kCellMargin, 0.f);
        const float left = r2 - (gx * gx + gy * gy);
        if (left < 0.f) return false;
        const float dz = left * rsqrt_hw(fmaxf(left, 1e-30f)) + kCellMargin;
        zl = (int)floorf((z0 - dz) * iw - 1e-3f);
        zh = (int)floorf((z1 + dz) * iw + 1e-3f);
        return true;
    }
};

// One warp: the neighbour lists of sorted particles p0 .. p0 + 3 of the staged
// tile (lane group g = lane / 8 takes p0 + g) whose pass is U (0 cell tiles,
// kUnitShift coarse tiles; the staged box is counted in units).  The search is
// transposed: each lane takes one staged slot of a row and tests it against all
// four particles.  A list holds the staged particles within 2 kTileListReach x
// the particle's starting h or x their own (see NeighbourLists).
template <int U>
__device__ __forceinline__ void lists_tile_warp(const DensityArgs &a, ListShared<U> &S, uint32_t p0, uint32_t end,
                                                int lane) {
    constexpr int L = kTileLanes;
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int kBig = 0x3fffffff;
    constexpr float kFar2 = 4.f * kTileListReach * kTileListReach;
    const int g = lane / L, sub = lane & (L - 1);
    const uint32_t p = p0 + (uint32_t)g;
    bool want = p < end && a.mode[p] == U;
    float4 me = make_float4(3e38f, 3e38f, 3e38f, 0.f);  // (a group without a particle is nowhere near)
    float hb = 0.f;
    // the staged box in its units
    const int us = unit_shift<U>(S.box);
    const float uw = kCellWidth * (float)(1 << us), uiw = (1.f / kCellWidth) / (float)(1 << us);
    const int lo0 = S.box[0] >> us, lo1 = S.box[1] >> us, lo2 = S.box[2] >> us;
    const int hi0 = S.box[3] >> us, hi1 = S.box[4] >> us, hi2 = S.box[5] >> us;
    const int ny = hi1 - lo1 + 1, nz = hi2 - lo2 + 1;
    if (want) {
        me = a.sp4[p];
        hb = S.narrow ? kNarrow * a.first_h[p] : a.start_h[p];
    }
    // a second search: wider, for the particles that found too few neighbours
    // for their h to stay within the first one's reach (a body's surface at its
    // first step), or just as far as the iteration's first sweep needs, for
    // those that found more than a list holds (a body that contracts)
    float hscale = S.narrow ? 0.f : kFar2;  // 0: the neighbours' own reach does not count
    bool narrow = false;
    for (int round = 0; round < 2; ++round) {
        CellBox b;
        b.lo0 = b.lo1 = b.lo2 = kBig;
        b.hi0 = b.hi1 = b.hi2 = -kBig;
        if (want) {
            tile_box(me.x, me.y, me.z, hb, b);
            if (round == 1 && !narrow && ((b.lo0 >> us) < lo0 || (b.lo1 >> us) < lo1 || (b.lo2 >> us) < lo2 ||
                               (b.hi0 >> us) > hi0 || (b.hi1 >> us) > hi1 || (b.hi2 >> us) > hi2)) {
                hb = a.start_h[p] * (kTileStageReach / kTileListReach);  // what is staged for it
                tile_box(me.x, me.y, me.z, hb, b);
            }
            b.lo0 = max(b.lo0 >> us, lo0), b.lo1 = max(b.lo1 >> us, lo1), b.lo2 = max(b.lo2 >> us, lo2);
            b.hi0 = min(b.hi0 >> us, hi0), b.hi1 = min(b.hi1 >> us, hi1), b.hi2 = min(b.hi2 >> us, hi2);
        }
        const float r2 = kFar2 * hb * hb;
        const int u0 = __reduce_min_sync(kFull, b.lo0), u1 = __reduce_min_sync(kFull, b.lo1),
                  u2 = __reduce_min_sync(kFull, b.lo2);
        const int v0 = __reduce_max_sync(kFull, b.hi0), v1 = __reduce_max_sync(kFull, b.hi1),
                  v2 = __reduce_max_sync(kFull, b.hi2);
        if (u0 > v0) return;  // nothing (more) to search for
        const float hm = fmaxf(hb, __int_as_float(S.hmax_bits));
        const Reach4 reach(me.x, me.y, me.z, want ? kFar2 * hm * hm : -1.f);
        F2 nx[kTileGpw / 2], ny2[kTileGpw / 2], nz2[kTileGpw / 2];  // minus the positions, two particles each
        float qr[kTileGpw];
        const float qpx = want ? me.x : 3e38f;
#pragma unroll
        for (int k = 0; k < kTileGpw; ++k) qr[k] = __shfl_sync(kFull, r2, k * L);
#pragma unroll
        for (int k = 0; k < kTileGpw / 2; ++k) {
            nx[k] = f2(-__shfl_sync(kFull, qpx, 2 * k * L), -__shfl_sync(kFull, qpx, (2 * k + 1) * L));
            ny2[k] = f2(-__shfl_sync(kFull, me.y, 2 * k * L), -__shfl_sync(kFull, me.y, (2 * k + 1) * L));
            nz2[k] = f2(-__shfl_sync(kFull, me.z, 2 * k * L), -__shfl_sync(kFull, me.z, (2 * k + 1) * L));
        }
        uint32_t *const out =
            a.lists.entries + (size_t)(p0 - (uint32_t)a.lists.first) * kTileList;  // of particle k: + k kTileList
        int cnt[kTileGpw] = {};
        const unsigned below = (1u << lane) - 1u;
        uint32_t *const rows_of = S.rows[threadIdx.x >> 5];
        // Rows (x, y) of the union box, 32 at a time, one per lane; each row is
        // trimmed to the z cells that the four spheres can reach, and the trimmed
        // rows are walked as one flat sequence of staged slots, 32 slots per step.
        const int nyu = v1 - u1 + 1;
        const int rows = (v0 - u0 + 1) * nyu;
        for (int rb = 0; rb < rows; rb += 32) {
            const int r = rb + lane;
            uint32_t len = 0u, s0 = 0u;
            if (r < rows) {
                const int x = u0 + r / nyu, y = u1 + r % nyu;
                int zl, zh;
                if (reach.row(x, y, uw, uiw, zl, zh)) {
                    zl = max(zl, u2);
                    zh = min(zh, v2);
                    if (zl <= zh) {
                        const int c0 = ((x - lo0) * ny + (y - lo1)) * nz;
                        s0 = S.off[c0 + (zl - lo2)];
                        len = S.off[c0 + (zh - lo2) + 1] - s0;
                    }
                }
            }
            uint32_t pre = len;  // inclusive scan of the row lengths
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(kFull, pre, o);
                if (lane >= o) pre += t;
            }
            const uint32_t excl = pre - len;
            const uint32_t total = __shfl_sync(kFull, pre, 31);
            // rows that have slots, in order: the staged slot of flat index v
            // in row j is rows[j] + v
            const unsigned some = __ballot_sync(kFull, len > 0u);
            __syncwarp();
            if (len) rows_of[__popc(some & below)] = s0 - excl;
            __syncwarp();
            int row0 = -1;  // the last row that starts before the step's slots
            for (uint32_t vb = 0; vb < total; vb += 32u) {
                const uint32_t v = vb + (uint32_t)lane;
                const uint32_t at0 = excl - vb;
                const unsigned starts = __reduce_or_sync(kFull, len && at0 < 32u ? 1u << at0 : 0u);
                const int j = row0 + __popc(starts & ((below << 1) | 1u));
                row0 += __popc(starts);
                const uint32_t s = rows_of[j] + v;
                float4 q = make_float4(-3e38f, -3e38f, -3e38f, 0.f);
                float hr = 0.f;
                uint32_t gi = 0u;
                if (v < total) {
                    q = S.pos[s];
                    const float h = S.hs[s];
                    hr = hscale * h * h;
                    gi = S.gidx[s];
                }
                const F2 qx = f2(q.x), qy = f2(q.y), qz = f2(q.z);
#pragma unroll
                for (int k = 0; k < kTileGpw / 2; ++k) {
                    const F2 dx = qx + nx[k], dy = qy + ny2[k], dz = qz + nz2[k];
                    float d[2];
                    unpack(fma2(dz, dz, fma2(dy, dy, dx * dx)), d[0], d[1]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int g2 = 2 * k + i;
                        const bool hit = d[i] <= fmaxf(qr[g2], hr);
                        const unsigned bal = __ballot_sync(kFull, hit);
                        const int at = cnt[g2] + __popc(bal & below);
                        if (hit && at < kTileList) out[g2 * kTileList + at] = gi;
                        cnt[g2] += __popc(bal);
                    }
                }
            }
        }
        if (want) {
            int c = 0;
#pragma unroll
            for (int k = 0; k < kTileGpw; ++k)
                if (g == k) c = cnt[k];
            if (sub == 0) {
                a.lists.count[p] = c <= kTileList ? (uint8_t)c : kNoList;
                a.lists.reach2[p] = hscale > 0.f ? r2 : -r2;
            }
            const float to = hb * cbrtf(kListFull / (float)max(c, 1));
            narrow = c > kTileList;
            want = round == 0 && !S.narrow && (narrow || (to > kTileListReach * hb && to < kMaxH));
            if (want) hb = narrow ? kNarrow * a.first_h[p] : fminf(1.02f * to, 0.999f * kMaxH);
        }
        // (a warp's second searches are alike: rare, and the test of a slot
        // stays the same for all)
        if (__any_sync(kFull, want && narrow)) hscale = 0.f;
    }
}

// The tile pass U over the tiles of `tiles` (ctr[0] of them, ctr[1] the tile
// ticket): U = 0 the cell tiles, U = kUnitShift the coarse tiles (512-cell
// blocks).
template <int U>
__global__ void __launch_bounds__(ListTile<U>::kThreads, ListTile<U>::kCtas)
    k_lists(DensityArgs a, const uint2 *__restrict__ tiles, uint32_t *ctr) {
    constexpr int T = ListTile<U>::kThreads;
    constexpr int kPer = (kTileCellsMax + T - 1) / T;  // units per thread
    extern __shared__ float4 s_tile_raw[];
    ListShared<U> &S = *reinterpret_cast<ListShared<U> *>(s_tile_raw);
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t ntiles = ctr[0];
    for (;;) {
        __syncthreads();  // the previous tile is done with the staged data
        if (tid == 0) {
            const uint32_t t = atomicAdd(ctr + 1, 1u);
            S.tile = t;
            if (t < ntiles) {
                const uint2 r = tiles[t];
                S.start = max(r.x, (uint32_t)a.lists.first);
                S.end = min(r.y, (uint32_t)a.lists.last);
            }
        }
        __syncthreads();
        if (S.tile >= ntiles) break;
        const uint32_t tstart = S.start, tend = S.end;
        if (tstart >= tend) continue;  // a tile of another slice
        // a tile whose staged box overflows shared memory is taken again as
        // its octets (coarse tiles: its units), one at a time, and an octet that
        // still does once more for lists that reach just as far as its particles'
        // first sweeps (a body under compression, whose h shrinks); what overflows
        // even so is left to the per-particle pass.  (Octets taken cell by cell
        // instead: eight boxes one after another for little less of a box, and
        // often in vain; free run of N = 1e5, density passes of steps 11 and 46
        // 2.2 and 2.6 ms instead of 1.4 and 1.0; N = 1e6, first 26 passes 92 ms
        // instead of 87, while a settled one is 2.06 with it and 2.07 so.)
        constexpr int kSplit = U == 0 ? 3 : 3 * U;
        const bool splittable = (a.skey[tstart] >> kSplit) != (a.skey[tend - 1] >> kSplit);
        int level = 0;  // 0 the tile, 1 its octets, 2 an octet once more
        uint32_t r0 = tstart;
        auto advance = [&](uint32_t to) {
            r0 = to;
            level = min(level, 1);
        };
        while (r0 < tend) {
            __syncthreads();
            if (tid == 0) {
                uint32_t r1 = tend;
                if (level > 0)  // the rest of r0's octet / unit
                    r1 = (U == 0 ? a.octets : a.units)[a.skey[r0] >> kSplit].y + 1u;
                r1 = min(max(r0 + 1u, r1), tend);
                S.narrow = level == 2;
                S.reach = level == 2 ? kFirstReach : kTileStageReach;
                S.end = r1;
                S.next = 0u;
                S.box[0] = S.box[1] = S.box[2] = 0x7fffffff;
                S.box[3] = S.box[4] = S.box[5] = -0x7fffffff;
                S.defer_all = 0;
                S.need = 0;
                S.hmax_bits = 0;
            }
            __syncthreads();
            const uint32_t start = r0, end = S.end;
            // the staged box: union of the list boxes of the pass's particles
            {
                int b[6] = {0x7fffffff, 0x7fffffff, 0x7fffffff, -0x7fffffff, -0x7fffffff, -0x7fffffff};
                bool need = false;
                for (uint32_t p = start + tid; p < end; p += T) {
                    if (a.mode[p] != U) continue;
                    need = true;
                    const float4 me = a.sp4[p];
                    CellBox cb;
                    tile_box(me.x, me.y, me.z, (S.narrow ? a.first_h : a.start_h)[p], cb, S.reach);
                    b[0] = min(b[0], cb.lo0);
                    b[1] = min(b[1], cb.lo1);
                    b[2] = min(b[2], cb.lo2);
                    b[3] = max(b[3], cb.hi0);
                    b[4] = max(b[4], cb.hi1);
                    b[5] = max(b[5], cb.hi2);
                }
                if (__any_sync(0xffffffffu, need)) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        b[k] = __reduce_min_sync(0xffffffffu, b[k]);
                        b[k + 3] = __reduce_max_sync(0xffffffffu, b[k + 3]);
                    }
                    if (lane == 0) {
                        S.need = 1;
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            atomicMin(&S.box[k], b[k]);
                            atomicMax(&S.box[k + 3], b[k + 3]);
                        }
                    }
                }
            }
            __syncthreads();
            if (!S.need) {  // nothing in the range for this pass
                advance(end);
                continue;
            }
            const int us = unit_shift<U>(S.box);
            const int lo0 = S.box[0] >> us, lo1 = S.box[1] >> us, lo2 = S.box[2] >> us;
            const int nx = box_extent(S.box[0], S.box[3], us), ny = box_extent(S.box[1], S.box[4], us),
                      nz = box_extent(S.box[2], S.box[5], us);
            const bool too_many = box_units(nx, ny, nz) > kTileCellsMax;
            const int ncell = too_many ? 0 : nx * ny * nz;
            // unit counts (kPer consecutive units per thread) and their
            // exclusive scan
            uint32_t c_cnt[kPer], c_first[kPer];
            uint32_t tsum = 0u;
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                const int c = kPer * tid + k;
                c_cnt[k] = c_first[k] = 0u;
                if (c < ncell) {
                    const int ix = c / (ny * nz), rem = c - ix * ny * nz, iy = rem / nz, iz = rem - iy * nz;
                    const uint2 r = unit_range(a.cells, a.octets, a.units, us, lo0 + ix, lo1 + iy, lo2 + iz);
                    if (r.x != 0xffffffffu) {
                        c_cnt[k] = r.y - r.x + 1u;
                        c_first[k] = r.x;
                    }
                }
                tsum += c_cnt[k];
            }
            uint32_t inc = tsum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane == 31) S.wsum[tid >> 5] = inc;
            __syncthreads();
            uint32_t wbase = 0u;
            for (int w = 0; w < (tid >> 5); ++w) wbase += S.wsum[w];
            uint32_t run = wbase + inc - tsum;
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                const int c = kPer * tid + k;
                if (c < ncell) S.off[c] = run;
                run += c_cnt[k];
            }
            if (tid == T - 1) {
                S.off[ncell] = run;
                if (too_many || run > (uint32_t)ListTile<U>::kStage) S.defer_all = 1;
            }
            __syncthreads();
            if (S.defer_all) {
                if (level < 2) level = level == 0 && splittable ? 1 : 2;
                else advance(end);  // its particles are left without a list
                continue;
            }
            float hmax = 0.f;
            stage_units(c_cnt, c_first, inc - tsum, inc, lane, [&](uint32_t v, uint32_t g, int) {
                const float h = __ldg(a.start_h + g);
                S.pos[wbase + v] = __ldg(a.sp4 + g);
                S.gidx[wbase + v] = g;
                S.hs[wbase + v] = h;
                hmax = fmaxf(hmax, h);
            });
            const int hbits = __reduce_max_sync(0xffffffffu, __float_as_int(hmax));
            if (lane == 0 && hbits > 0) atomicMax(&S.hmax_bits, hbits);
            __syncthreads();
            // warps take the tile's particles four at a time
            for (;;) {
                uint32_t j = 0u;
                if (lane == 0) j = atomicAdd(&S.next, (uint32_t)kTileGpw);
                j = __shfl_sync(0xffffffffu, j, 0);
                if (start + j >= end) break;
                lists_tile_warp<U>(a, S, start + j, end, lane);
            }
            advance(end);
        }
    }
}

// The density pass over the lists: a warp takes four consecutive sorted
// particles, eight lanes each, in lockstep so it never runs its groups one after
// another.  Particles without a list, and those whose h outgrows theirs, are
// appended to `deferred` (sorted index) with nothing written;
// k_density_deferred takes them from the start.  The iteration is
// density_particle's with the neighbour cache never in use (h < MAX_H
// throughout, so the reference's int max_h stays 0).
// only: kAllModes, or whether the particles of the coarse tiles are taken
// (kUnitShift) or those of all other modes (0).
constexpr int kAllModes = -1;
constexpr int kListThreads = 256;
__global__ void __launch_bounds__(kListThreads, 4)
    k_density_list(DensityArgs a, int only, uint32_t *__restrict__ deferred, uint32_t *dctr) {
    constexpr int L = kTileLanes;
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & (L - 1);
    const int p = a.lists.first + (int)((blockIdx.x * (unsigned)kListThreads + threadIdx.x) / L);
    const uint8_t mode = p < a.lists.last ? a.mode[p] : kModeInactive;
    // the group iterates its particle (uniform within the group)
    bool live = p < a.lists.last && (only == kAllModes || (mode == kUnitShift) == (only == kUnitShift));
    uint32_t ind = 0u;
    float4 me = make_float4(0.f, 0.f, 0.f, 0.f), mv = me;
    float h_plain = 0.5f;
    int n_list = -1;
    if (live) {
        ind = a.cidx[p];
        me = a.sp4[p];
        mv = a.sv4[p];
        h_plain = a.h[ind];
        if (mode == kModeInactive) {
            // density.metal:40-55: EOS only
            if (sub == 0) {
                float2 pc = eos_lookup(a.eos, a.mat[ind], a.rho[ind], a.u[ind]);
                a.P[ind] = pc.x;
                a.c[ind] = pc.y;
                float rho = a.rho[ind], fi = a.f[ind];
                a.sA[p] = make_float4(me.x, me.y, me.z, h_plain);
                a.sB[p] = make_float4(mv.x, mv.y, mv.z, pc.y);
                a.sC[p] = make_float4(me.w, (fi * pc.x / (rho * rho)), rho, a.B[ind]);
            }
            live = false;
        }
    }
    auto defer = [&]() {
        if (sub == 0) {
            deferred[atomicAdd(dctr, 1u)] = (uint32_t)p;
            a.lists.count[p] = kNoList;  // (too short for the acceleration pass too)
        }
        live = false;
    };
    const uint32_t *list = a.lists.entries + (size_t)(p < a.lists.last ? p - a.lists.first : 0) * kTileList;
    float hi = 0.5f, list_r2 = 0.f;
    bool seeded = false;
    if (live) {
        const uint8_t c = a.lists.count[p];
        if (c == kNoList) {
            defer();
        } else {
            n_list = c;
            list_r2 = fabsf(a.lists.reach2[p]);
            hi = tile_start_h(a, ind, h_plain, seeded);
        }
    }
    const float px = me.x, py = me.y, pz = me.z, mi = me.w;
    const int maxn = __reduce_max_sync(kFull, n_list);
    // The sorted index behind list entry i, this particle's own past the list's
    // end: loads without branches, so that many are in flight together.
    const int self = min(p, a.n - 1);
    auto entry = [&](int i) { return i < n_list ? (int)__ldg(list + i) : self; };
    // Distance and mass of the pair of list entries (i, i + L); nothing (a
    // massless neighbour far away) past the list's end.
    auto entry_pair = [&](int i, F2 &r, F2 &m) {
        float rr[2], mm[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float4 q = __ldg(a.sp4 + entry(i + e * L));
            const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
            const bool in = i + e * L < n_list;
            rr[e] = in ? pair_sqrt(dx * dx + dy * dy + dz * dz) : 1e30f;
            mm[e] = in ? q.w : 0.f;
        }
        r = f2(rr[0], rr[1]);
        m = f2(mm[0], mm[1]);
    };
    F2 rp[kRegPairs], mp[kRegPairs];
#pragma unroll
    for (int t = 0; t < kRegPairs; ++t) entry_pair(sub + 2 * t * L, rp[t], mp[t]);
    bool iter = live;
    bool first = true, fell_back = false;
    int sweeps = 0, count = 0;
    float h2x4 = 4.f * hi * hi;
    float h1 = 1.f / hi;
    float w4 = 0.f, eps = 1.f;  // 4 pi h^3 x the density
    while (__any_sync(kFull, iter)) {
        // the cubic spline as (2 - q)+^3 / 4 - (1 - q)+^3
        const F2 nh = f2(-h1);
        F2 acc = f2(0.f);
        auto add = [&](F2 r, F2 m) {
            const F2 t = clamp0(fma2(r, nh, f2(2.f))), u = clamp0(fma2(r, nh, f2(1.f)));
            acc = fma2(m, fma2(f2(-4.f) * u, u * u, t * (t * t)), acc);
        };
#pragma unroll
        for (int t = 0; t < kRegPairs; ++t) add(rp[t], mp[t]);
        for (int i = kRegList + sub; i < maxn; i += 2 * L) {
            F2 r, m;
            entry_pair(i, r, m);
            add(r, m);
        }
        const float wsum = group_sum<L>(sum(acc), kFull);
        if (iter) {
            w4 = wsum;
            const float dens = kernel_norm(h1) * wsum;
            float nh_ = fmin_ref(kResolutionEta * cbrtf(pdiv(mi, dens)), kMaxH);
            nh_ = 0.5f * (hi + nh_);
            eps = fabsf(nh_ - hi) * h1;
            ++sweeps;
            if (first && seeded && eps > kSeedFallback) {
                // the seed disagrees with its own first sweep: start again from
                // the plain guess
                fell_back = true;
                hi = h_plain;
                h1 = 1.f / hi;
                h2x4 = 4.f * hi * hi;
                eps = 1.f;
            } else if (eps > a.eta) {
                // at MAX_H the reference's int max_h would leave 0, and a
                // particle that does not converge ends on another h than its
                // last sweep's: the per-particle pass takes both, and those
                // whose list is too short for the new h
                hi = nh_;
                h1 = 1.f / hi;
                h2x4 = 4.f * hi * hi;
                if (nh_ >= kMaxH || ++count >= kMaxNR || !(h2x4 <= list_r2)) defer();
            }
            first = false;
            iter = live && eps > a.eta;
        }
    }
    // gradient sweep (density.metal:145-213) over the last sweep's neighbours,
    // those within 2 h; with g' = 3 (1 - q)+^2 - 3 (2 - q)+^2 / 4 the spline's
    // derivative, dW/dh = -(3 W + q g') / h (up to the norm), so of it only
    // the sum of q g' is new
    const float vix = mv.x, viy = mv.y, viz = mv.z;
    F2 qg = f2(0.f), vdiv2 = qg, cx2 = qg, cy2 = qg, cz2 = qg;
    int nn = 0;
    const F2 nh = f2(-h1);
#pragma unroll 2
    for (int i = sub; i < maxn; i += 2 * L) {
        // (a neighbour past 2 h, or the list's end: this particle itself)
        float4 q[2], vj[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int gi = entry(i + e * L);
            q[e] = __ldg(a.sp4 + gi);
            vj[e] = __ldg(a.sv4 + gi);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float dx = q[e].x - px, dy = q[e].y - py, dz = q[e].z - pz;
            const bool in = dx * dx + dy * dy + dz * dz <= h2x4 && i + e * L < n_list;
            if (!in) {
                q[e] = me;
                vj[e] = mv;
            }
            nn += in ? 1 : 0;
        }
        const F2 dx = f2(q[0].x, q[1].x) + f2(-px), dy = f2(q[0].y, q[1].y) + f2(-py),
                 dz = f2(q[0].z, q[1].z) + f2(-pz);
        const F2 r2 = fma2(dz, dz, fma2(dy, dy, dx * dx));
        float ra, rb;
        unpack(r2, ra, rb);
        const F2 rinv = f2(ra > 1e-24f ? rsqrt_hw(ra) : 0.f, rb > 1e-24f ? rsqrt_hw(rb) : 0.f);
        const F2 r = r2 * rinv;
        const F2 t = clamp0(fma2(r, nh, f2(2.f))), u = clamp0(fma2(r, nh, f2(1.f)));
        const F2 g = f2(q[0].w, q[1].w) * fma2(f2(3.f) * u, u, f2(-0.75f) * (t * t));
        qg = fma2(g, r * nh, qg);  // (nh is -1/h: minus the sum)
        const F2 gr = g * rinv;
        const F2 gx = gr * dx, gy = gr * dy, gz = gr * dz;
        const F2 vx = f2(vj[0].x, vj[1].x) + f2(-vix), vy = f2(vj[0].y, vj[1].y) + f2(-viy),
                 vz = f2(vj[0].z, vj[1].z) + f2(-viz);
        vdiv2 = fma2(vz, gz, fma2(vy, gy, fma2(vx, gx, vdiv2)));
        cx2 = fma2(vy, gz, fma2(neg(vz), gy, cx2));
        cy2 = fma2(vz, gx, fma2(neg(vx), gz, cy2));
        cz2 = fma2(vx, gy, fma2(neg(vy), gx, cz2));
    }
    nn = group_sum_i<L>(nn, kFull);
    const float norm = kernel_norm(h1);  // 1 / (4 pi h^3)
    const float nqg = group_sum<L>(sum(qg), kFull);
    const float gnorm = 4.f * norm * h1;
    float vdiv = gnorm * group_sum<L>(sum(vdiv2), kFull);
    const float cx = gnorm * group_sum<L>(sum(cx2), kFull);
    const float cy = gnorm * group_sum<L>(sum(cy2), kFull);
    const float cz = gnorm * group_sum<L>(sum(cz2), kFull);
    if (a.stats) {
        const uint32_t mine = live && sub == 0 ? 1u : 0u;
        const uint32_t sw = __reduce_add_sync(kFull, mine * (uint32_t)sweeps);
        const uint32_t fb = __reduce_add_sync(kFull, mine * (fell_back ? 1u : 0u));
        const uint32_t mx = __reduce_max_sync(kFull, mine * (uint32_t)sweeps);
        const uint32_t np = __reduce_add_sync(kFull, mine);
        __shared__ uint32_t s_stats[4];
        if (threadIdx.x < 4) s_stats[threadIdx.x] = 0u;
        __syncthreads();
        if (lane == 0) {
            atomicAdd(&s_stats[0], sw);
            atomicAdd(&s_stats[1], fb);
            atomicMax(&s_stats[2], mx);
            atomicAdd(&s_stats[3], np);
        }
        __syncthreads();
        if (threadIdx.x == 0 && s_stats[3]) {
            atomicAdd(a.stats + 0, s_stats[0]);
            if (s_stats[1]) atomicAdd(a.stats + 1, s_stats[1]);
            atomicMax(a.stats + 2, s_stats[2]);
            atomicAdd(a.stats + 3, s_stats[3]);
        }
    }
    if (!live || sub != 0) return;
    // 3 sum(W) + sum(q g') over sum(4 W): nqg is minus sum(q g')
    const float dens_h = -gnorm * (0.75f * w4 - nqg);
    float dens = norm * w4;
    nn = min(nn, kNeighbourCache);
    if (nn >= kNeighbourCache) dens += dens;  // the reference's full scan adds the density again
    mark_grown(a, (uint32_t)p, hi);
    if (a.nn_out) a.nn_out[ind] = (float)nn;
    vdiv = fabsf(vdiv) / dens;
    float acurl = sqrtf(cx * cx + cy * cy + cz * cz) / dens;
    float fi = 1.f / (1.f + (hi / (3.f * dens)) * dens_h);
    float2 pc = eos_lookup(a.eos, a.mat[ind], dens, a.u[ind]);
    float bal = vdiv / (vdiv + acurl + 1e-4f * (pc.y / hi));
    a.h[ind] = hi;
    a.rho[ind] = dens;
    a.f[ind] = fi;
    a.P[ind] = pc.x;
    a.c[ind] = pc.y;
    a.B[ind] = bal;
    if (!(dens == dens) || !(pc.x == pc.x)) raise_health(a.health, SPH_HEALTH_NAN_DENSITY);
    a.sA[p] = make_float4(px, py, pz, hi);
    a.sB[p] = make_float4(vix, viy, viz, pc.y);
    a.sC[p] = make_float4(mi, (fi * pc.x / (dens * dens)), dens, bal);
}

struct AccelArgs {
    int n;
    const uint32_t *cidx;
    const uint32_t *skey;  // sorted cell keys (tile passes)
    const uint2 *cells;
    const uint2 *octets;   // 8-cell octet ranges and
    const uint2 *units;    // 64-cell unit ranges (coarse tiles)
    uint8_t *cflags;       // per 512-cell block: holds a coarse-tile particle
    int coarse;            // coarse tiles on
    uint8_t *mode;         // [n] the pass that takes each sorted particle (kMode*), written by k_acceleration_plan
    NeighbourLists lists;  // the density pass's
    const float4 *sA, *sB, *sC;
    float4 *acc4;
    float *du, *dhdt;
    int32_t *nat;
    const uint8_t *active;
    int32_t *globals;
    int individual;  // SPH_TIMESTEP_INDIVIDUAL: inactive particles bound the global step
};

// The ticks an inactive particle allows the global step: INT_MAX with the
// reference's test (all particles active anyway); with individual timesteps
// the time left to its next active time, so no step passes it.
__device__ __forceinline__ int inactive_ticks(const AccelArgs &a, uint32_t ind) {
    if (!a.individual) return 0x7fffffff;
    return max(a.nat[ind] - a.globals[0], 1);
}

// The particle's own terms of accelerations.metal:60-141.
struct AccelI {
    float xi, yi, zi, hi, vxi, vyi, vzi, ci, facti, rhoi, Bi, hi1, hi2x4;
};
__device__ __forceinline__ AccelI accel_i(const float4 A, const float4 Bv, const float4 Cv) {
    AccelI I;
    I.xi = A.x;
    I.yi = A.y;
    I.zi = A.z;
    I.hi = A.w;
    I.vxi = Bv.x;
    I.vyi = Bv.y;
    I.vzi = Bv.z;
    I.ci = Bv.w;
    I.facti = Cv.y;
    I.rhoi = Cv.z;
    I.Bi = Cv.w;
    I.hi1 = 1.f / I.hi;
    I.hi2x4 = I.hi * I.hi * 4.f;
    return I;
}
// Running sums of one particle (a slice of its pairs): acceleration, du/dt,
// dh/dt, with Kahan compensations in the mixed-precision form, and the
// largest signal speed.
struct AccelSum {
    float dvx = 0.f, dvy = 0.f, dvz = 0.f, du = 0.f, dh = 0.f;
    float kx = 0.f, ky = 0.f, kz = 0.f, ku = 0.f, kh = 0.f;
    float vsig = 1e-12f;
};
template <bool KAHAN>
__device__ __forceinline__ void accel_add(float &sum, float &comp, float v) {
    if (KAHAN) {
        const float y = v - comp;
        const float t = sum + y;
        comp = (t - sum) - y;
        sum = t;
    } else {
        sum += v;
    }
}
// accelerations.metal:75-124: one accepted pair (Aj = (x, y, z, h),
// Bj = (v, c), Cj = (m, f P / rho^2, rho, B) of the neighbour).
template <bool KAHAN>
__device__ __forceinline__ void accel_pair(const AccelI &I, AccelSum &S, const float4 Aj, const float4 Bj,
                                           const float4 Cj) {
    const float dx = I.xi - Aj.x, dy = I.yi - Aj.y, dz = I.zi - Aj.z;
    const float r2 = dx * dx + dy * dy + dz * dz;
    const float hj = Aj.w;
    const float r = pair_sqrt(r2);
    const float r1 = pair_rinv(r2, r);
    const float mj = Cj.x, factj = Cj.y, rhoj = Cj.z, Balj = Cj.w;
    const float hj1 = pdiv(1.f, hj);
    const float vx = I.vxi - Bj.x, vy = I.vyi - Bj.y, vz = I.vzi - Bj.z;
    const float rhoij = 0.5f * (I.rhoi + rhoj);
    const float vdr = vx * dx + vy * dy + vz * dz;
    const float mu = vdr < 0.f ? vdr * r1 : 0.f;
    const float vsig = I.ci + Bj.w - 3.f * mu;
    S.vsig = fmax_ref(vsig, S.vsig);
    const float Bij = 0.5f * (I.Bi + Balj);
    const float nu = pdiv(-0.5f * kViscosityAlpha * Bij * mu * vsig, rhoij);
    const float rhx = dx * r1, rhy = dy * r1, rhz = dz * r1;
    const float si = kernel_gradw_scale(r, I.hi1), sj = kernel_gradw_scale(r, hj1);
    const float gix = si * rhx, giy = si * rhy, giz = si * rhz;
    const float gjx = sj * rhx, gjy = sj * rhy, gjz = sj * rhz;
    const float gx = 0.5f * (gix + gjx), gy = 0.5f * (giy + gjy), gz = 0.5f * (giz + gjz);
    accel_add<KAHAN>(S.dvx, S.kx, -(mj * (I.facti * gix + factj * gjx + nu * gx)));
    accel_add<KAHAN>(S.dvy, S.ky, -(mj * (I.facti * giy + factj * gjy + nu * gy)));
    accel_add<KAHAN>(S.dvz, S.kz, -(mj * (I.facti * giz + factj * gjz + nu * gz)));
    accel_add<KAHAN>(S.du, S.ku,
                     mj * (I.facti * (vx * gix + vy * giy + vz * giz) + 0.5f * nu * (vx * gx + vy * gy + vz * gz)));
    accel_add<KAHAN>(S.dh, S.kh, pdiv(mj, rhoj) * (vx * gix + vy * giy + vz * giz));
}
// The same for two neighbours per lane in packed arithmetic (product build's
// tiles).  All of a pair's vector terms lie along the pair, so they are the
// scalar factors below times (x_j - x_i) / r:
//   si, sj       gradW(h_i), gradW(h_j) along the pair
//   push         m_j (f_i si + f_j sj + nu (si + sj) / 2) / r
//   w            (v_j - v_i) . (x_j - x_i) / r
struct AccelSum2 {
    F2 x = F2{0}, y = F2{0}, z = F2{0}, du = F2{0}, dh = F2{0};
    F2 kx = F2{0}, ky = F2{0}, kz = F2{0}, ku = F2{0}, kh = F2{0};
    float vsig = 1e-12f;
};
template <bool KAHAN>
__device__ __forceinline__ void accel_add2(F2 &sum, F2 &comp, F2 v) {
    if (KAHAN) {
        const F2 minus = f2(-1.f);
        const F2 y = fma2(comp, minus, v);
        const F2 t = sum + y;
        comp = fma2(y, minus, fma2(sum, minus, t));
        sum = t;
    } else {
        sum = sum + v;
    }
}
// pi h^4 times the spline's gradient along the pair at distance r: the
// derivative of (2 - q)+^3 / 4 - (1 - q)+^3
__device__ __forceinline__ F2 spline_slope(F2 r, F2 minus_h1) {
    const F2 t = clamp0(fma2(r, minus_h1, f2(2.f))), u = clamp0(fma2(r, minus_h1, f2(1.f)));
    return fma2(f2(3.f) * u, u, f2(-0.75f) * (t * t));
}
template <bool KAHAN>
__device__ __forceinline__ void accel_pair2(const AccelI &I, float fac_i, AccelSum2 &S, const float4 (&A)[2],
                                            const float4 (&B)[2], const float4 (&C)[2]) {
    const F2 ex = f2(A[0].x, A[1].x) + f2(-I.xi), ey = f2(A[0].y, A[1].y) + f2(-I.yi),
             ez = f2(A[0].z, A[1].z) + f2(-I.zi);
    const F2 r2 = fma2(ez, ez, fma2(ey, ey, ex * ex));
    const F2 r1 = rsqrt2(r2);
    const F2 r = r2 * r1;
    const F2 vx = f2(B[0].x, B[1].x) + f2(-I.vxi), vy = f2(B[0].y, B[1].y) + f2(-I.vyi),
             vz = f2(B[0].z, B[1].z) + f2(-I.vzi);
    const F2 w = fma2(vz, ez, fma2(vy, ey, vx * ex)) * r1;
    float wa, wb;
    unpack(w, wa, wb);
    const F2 mu = f2(fminf(wa, 0.f), fminf(wb, 0.f));
    const F2 vsig = fma2(f2(-3.f), mu, f2(B[0].w, B[1].w) + f2(I.ci));
    float va, vb;
    unpack(vsig, va, vb);
    S.vsig = fmaxf(S.vsig, fmaxf(va, vb));
    // -alpha B_ij mu vsig / (2 rho_ij), the halves of B_ij and rho_ij cancelled
    const F2 bal = f2(C[0].w, C[1].w) + f2(I.Bi);
    const F2 nu = f2(-0.5f * kViscosityAlpha) * bal * (mu * vsig) *
                  f2(pdiv(1.f, I.rhoi + C[0].z), pdiv(1.f, I.rhoi + C[1].z));
    const F2 nhj = f2(pdiv(-1.f, A[0].w), pdiv(-1.f, A[1].w));
    const F2 hj2 = nhj * nhj;
    const F2 si = f2(fac_i) * spline_slope(r, f2(-I.hi1));
    const F2 sj = (f2(kPi1) * hj2) * hj2 * spline_slope(r, nhj);
    const F2 mean = f2(0.5f) * (si + sj);
    const F2 m = f2(C[0].x, C[1].x);
    const F2 fsi = f2(I.facti) * si;
    const F2 push = m * fma2(nu, mean, fma2(f2(C[0].y, C[1].y), sj, fsi)) * r1;
    accel_add2<KAHAN>(S.x, S.kx, push * ex);
    accel_add2<KAHAN>(S.y, S.ky, push * ey);
    accel_add2<KAHAN>(S.z, S.kz, push * ez);
    accel_add2<KAHAN>(S.du, S.ku, m * w * fma2(f2(0.5f) * nu, mean, fsi));
    accel_add2<KAHAN>(S.dh, S.kh, m * w * si * f2(pdiv(1.f, C[0].z), pdiv(1.f, C[1].z)));
}

// A lane's two halves (with their compensations) as one.
template <bool KAHAN>
__device__ __forceinline__ AccelSum accel_close(const AccelSum2 &S) {
    const F2 minus = f2(-1.f);
    AccelSum r;
    r.dvx = sum(KAHAN ? fma2(S.kx, minus, S.x) : S.x);
    r.dvy = sum(KAHAN ? fma2(S.ky, minus, S.y) : S.y);
    r.dvz = sum(KAHAN ? fma2(S.kz, minus, S.z) : S.z);
    r.du = sum(KAHAN ? fma2(S.ku, minus, S.du) : S.du);
    r.dh = sum(KAHAN ? fma2(S.kh, minus, S.dh) : S.dh);
    r.vsig = S.vsig;
    return r;
}

// The group's sums combined (every lane ends with the same bits).
template <int L, bool KAHAN>
__device__ __forceinline__ void accel_reduce(AccelSum &S, unsigned gm) {
    if (KAHAN) {
        S.dvx -= S.kx;
        S.dvy -= S.ky;
        S.dvz -= S.kz;
        S.du -= S.ku;
        S.dh -= S.kh;
    }
    S.dvx = group_sum<L>(S.dvx, gm);
    S.dvy = group_sum<L>(S.dvy, gm);
    S.dvz = group_sum<L>(S.dvz, gm);
    S.du = group_sum<L>(S.du, gm);
    S.dh = group_sum<L>(S.dh, gm);
    S.vsig = group_max<L>(S.vsig, gm);
}
// accelerations.metal:129-140: the particle's timestep in ticks, DT0 halved
// until it is at most `goal` (kRMax times at most): the halvings are read off
// the goal's exponent, 2^e <= goal < 2^(e + 1).
__device__ __forceinline__ int accel_ticks(const AccelI &I, float vsig) {
    const float goal = 2.0f * kCFL * kGamma * I.hi / vsig;
    static_assert(kDT0 == 32.f, "5 below is log2 DT0");
    const int e = (int)((__float_as_uint(goal) >> 23) & 255u) - 127;
    return (1 << kRMax) >> min(max(5 - e, 0), kRMax);
}
__device__ __forceinline__ void accel_store(const AccelArgs &a, uint32_t ind, const AccelSum &S, int idt) {
    float4 acc = a.acc4[ind];
    acc.x += S.dvx;
    acc.y += S.dvy;
    acc.z += S.dvz;
    a.acc4[ind] = acc;
    a.du[ind] = S.du;
    a.dhdt[ind] = S.dh;
    a.nat[ind] = a.globals[0] + idt;
}

// accelerations.metal:12-141 for one sorted particle per lane group.  The
// walk covers the particle's own box of radius 2 min(h, MAX_SMOOTHING_LENGTH)
// (the reference's box, which also decides which pairs with r < 2 h_j are
// seen, Q8).  The pairs that pass the reference's test are first collected in
// order into the group's list, then evaluated by all lanes of the group
// together, so the long pair computation runs with every lane busy.  Returns
// the particle's timestep in ticks (INT_MAX when inactive).
template <int L, bool KAHAN>
__device__ __forceinline__ int accel_particle(const AccelArgs &a, int index, int sub, unsigned gm, int gbase,
                                              uint32_t *w_off, uint32_t *w_start, uint32_t *list) {
    const uint32_t ind = a.cidx[index];
    if (!a.active[ind]) return inactive_ticks(a, ind);
    const AccelI I = accel_i(a.sA[index], a.sB[index], a.sC[index]);
    AccelSum S;
    const float4 *sA = a.sA, *sB = a.sB, *sC = a.sC;
    auto drain = [&](int cnt) {
        __syncwarp(gm);
        for (int i = sub; i < cnt; i += L) {
            const uint32_t k = list[i];
            accel_pair<KAHAN>(I, S, __ldg(sA + k), __ldg(sB + k), __ldg(sC + k));
        }
        __syncwarp(gm);
        return true;
    };
    const int rest = group_collect<L>(
        I.xi, I.yi, I.zi, fmin_ref(I.hi, kMaxH), 3.402823466e+38f, a.cells, sub, gm, gbase, w_off, w_start, list,
        kListMax,
        [&](uint32_t k) {
            const float4 Aj = __ldg(sA + k);
            const float dx = I.xi - Aj.x, dy = I.yi - Aj.y, dz = I.zi - Aj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            const float hj2x4 = Aj.w * Aj.w * 4.f;
            return !((r2 > I.hi2x4 && r2 > hj2x4) || r2 < 1e-12f);
        },
        drain);
    drain(rest);
    accel_reduce<L, KAHAN>(S, gm);
    const int idt = accel_ticks(I, S.vsig);
    if (sub == 0) accel_store(a, ind, S, idt);
    return idt;
}

// Block-wide minimum of the timesteps, then one atomic per block that lowers
// the global one.
__device__ __forceinline__ void block_min_dt(int idt, int32_t *dt) {
    __shared__ int wmin[32];
    const int lane = threadIdx.x & 31;
    for (int o = 16; o > 0; o >>= 1) idt = min(idt, __shfl_xor_sync(0xffffffffu, idt, o));
    if (lane == 0) wmin[threadIdx.x >> 5] = idt;
    __syncthreads();
    if (threadIdx.x < 32) {
        int v = (threadIdx.x < ((blockDim.x + 31) >> 5)) ? wmin[threadIdx.x] : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (threadIdx.x == 0 && v < *(volatile int32_t *)dt) atomicMin(dt, v);
    }
}

#ifdef SPH_PARITY
template <int L, bool KAHAN>
__global__ void __launch_bounds__(parts_per_block<L>() * L) k_acceleration(AccelArgs a) {
    extern __shared__ uint32_t s_lists[];
    __shared__ uint32_t s_off[parts_per_block<L>() * L], s_start[parts_per_block<L>() * L];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, sub = lane & (L - 1), gbase = lane & ~(L - 1);
    const int index = t / L;
    int idt = 0x7fffffff;
    if (index < a.n)
        idt = accel_particle<L, KAHAN>(a, index, sub, group_mask<L>(lane), gbase, s_off + (threadIdx.x & ~31),
                                       s_start + (threadIdx.x & ~31),
                                       s_lists + (size_t)(threadIdx.x / L) * kListMax);
    block_min_dt(idt, a.globals + 1);
}
#endif

// The particles the tile pass handed on (sorted indices idx[0, *count)).
template <int L, bool KAHAN>
__global__ void __launch_bounds__(parts_per_block<L>() * L)
    k_acceleration_deferred(AccelArgs a, const uint32_t *__restrict__ idx, const uint32_t *__restrict__ count) {
    extern __shared__ uint32_t s_lists[];
    __shared__ uint32_t s_off[parts_per_block<L>() * L], s_start[parts_per_block<L>() * L];
    const int lane = threadIdx.x & 31, sub = lane & (L - 1), gbase = lane & ~(L - 1);
    const uint32_t cnt = *count;
    constexpr int per_block = parts_per_block<L>();
    int idt = 0x7fffffff;
    for (uint32_t base = blockIdx.x * per_block; base < cnt; base += gridDim.x * per_block) {
        const uint32_t j = base + threadIdx.x / L;
        if (j < cnt)
            idt = min(idt, accel_particle<L, KAHAN>(a, (int)idx[j], sub, group_mask<L>(lane), gbase,
                                                    s_off + (threadIdx.x & ~31), s_start + (threadIdx.x & ~31),
                                                    s_lists + (size_t)(threadIdx.x / L) * kListMax));
    }
    block_min_dt(idt, a.globals + 1);
}

// ---- acceleration over cell tiles (product build) ---------------------------
//
// The tiles of the density pass (k_density_plan), staged the same way with the
// sA records (x, y, z, h) of the union of the tile particles' boxes of radius
// 2 min(h, MAX_H) -- the reference's box, exact (cell_box) -- plus each staged
// particle's cell within the staged box.  Warps take four particles at a time:
// the transposed list build walks the rows of the four boxes as one flat
// sequence and keeps a pair when r <= 2 h_i, or when r <= 2 h_j and the
// neighbour's cell lies in the particle's box (the reference sees such a pair
// only there, Q8); then the pair arithmetic runs over the lists with every
// lane busy, reading the neighbour's sB / sC records by its sorted index.
// Particles whose box reaches more than kTileReach cells past their own cell,
// whose list overflows, and every particle of a tile whose staged box exceeds
// the budget go to k_acceleration_deferred.
constexpr int kTileThreads = 384;
constexpr int kTileGroups = kTileThreads / kTileLanes;  // particles in flight per CTA
constexpr int kTileAccList = 256;                       // list entries per particle
constexpr int kTileAccStage = 3072;                     // staged particles per tile
constexpr int kTileCellsPerThread = (kTileCellsMax + kTileThreads - 1) / kTileThreads;

struct TileAccShared {
    float4 pos[kTileAccStage];          // staged sA (x, y, z, h)
    uint32_t gidx[kTileAccStage];       // staged sorted index
    uint32_t scell[kTileAccStage];      // staged cell, box-relative (pack_cell)
    uint32_t off[kTileCellsMax + 1];
    uint16_t list[kTileGroups][kTileAccList];
    int box[6];
    uint32_t wsum[kTileThreads / 32];
    uint32_t start, end, tile, next;
    int defer_all;
    int need;                           // some particle of the range needs the warp pass
    int dtmin;
    int hmax_bits;                      // largest staged h (float bits; h > 0)
};

// The reference's box of an acceleration particle (cells) and the pass that
// takes it: 0 the cell tiles (reach within kTileReach cells of its own),
// kUnitShift the coarse tiles (within kTileReach units), -1 the per-particle
// pass (h at MAX_H, or coarse tiles off).
__device__ __forceinline__ int accel_mode(float px, float py, float pz, float h, CellBox &b, int coarse) {
    b = cell_box(px, py, pz, fmin_ref(h, kMaxH));
    if (!(h < kMaxH)) return -1;
    const int ox = (int)floorf(__fdiv_rn(px, kCellWidth)), oy = (int)floorf(__fdiv_rn(py, kCellWidth)),
              oz = (int)floorf(__fdiv_rn(pz, kCellWidth));
    if (within_reach<0>(ox, oy, oz, b)) return 0;
    if (coarse && within_reach<kUnitShift>(ox, oy, oz, b)) return kUnitShift;
    return -1;
}

// Three cell coordinates below kBoxCellsMax in one word, each followed by a
// guard bit: in_box subtracts all three at once, and a guard bit that a
// subtraction borrows marks a coordinate past the bound.
constexpr int kBoxCellsMax = 512;
constexpr uint32_t kGuards = (1u << 9) | (1u << 19) | (1u << 29);
__device__ __forceinline__ uint32_t pack_cell(int x, int y, int z) {
    return (uint32_t)x | ((uint32_t)y << 10) | ((uint32_t)z << 20);
}
__device__ __forceinline__ bool in_box(uint32_t c, uint32_t lo, uint32_t hi) {
    return (((c | kGuards) - lo) & ((hi | kGuards) - c) & kGuards) == kGuards;
}

// One warp: the acceleration pass of sorted particles p0 .. p0 + 3 of the
// staged tile (lane group g takes p0 + g) whose pass is U (the staged box
// counts U-units; the group boxes and staged cells stay in cells, relative to
// the box's first cell).  Returns the warp's smallest timestep in ticks
// (INT_MAX when none).
template <bool KAHAN, int U>
__device__ __forceinline__ int accel_tile_warp(const AccelArgs &a, TileAccShared &S, uint32_t p0, uint32_t end,
                                               int lane, int wslot, uint32_t *deferred, uint32_t *dctr) {
    constexpr int L = kTileLanes;
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int kBig = 0x3fffffff;
    const int g = lane / L, sub = lane & (L - 1);
    uint16_t *list = S.list[wslot * kTileGpw + g];
    const uint32_t p = p0 + (uint32_t)g;
    bool live = p < end;
    uint32_t ind = 0u;
    int idt_inactive = 0x7fffffff;
    const uint8_t mode = live ? a.mode[p] : kModeInactive;
    if (live && mode != U && (U != 0 || mode < kModeWalk)) live = false;  // another pass takes it
    if (live) {
        ind = a.cidx[p];
        if (mode == kModeInactive) {
            idt_inactive = inactive_ticks(a, ind);
            live = false;
        }
    }
    float4 A = make_float4(0.f, 0.f, 0.f, 1.f), Bv = A, Cv = A;
    if (live) {
        A = a.sA[p];
        Bv = a.sB[p];
        Cv = a.sC[p];
    }
    const AccelI I = accel_i(A, Bv, Cv);
    // the staged box in its units
    const int us = unit_shift<U>(S.box);
    const float uw = kCellWidth * (float)(1 << us), uiw = (1.f / kCellWidth) / (float)(1 << us);
    const int lo0 = S.box[0] >> us, lo1 = S.box[1] >> us, lo2 = S.box[2] >> us;
    const int ny = (S.box[4] >> us) - lo1 + 1, nz = (S.box[5] >> us) - lo2 + 1;
    CellBox b;
    bool want = false;
    if (live) {
        if (mode != U || S.defer_all) {
            if (sub == 0) deferred[atomicAdd(dctr, 1u)] = p;
            live = false;
        } else {
            b = cell_box(I.xi, I.yi, I.zi, fmin_ref(I.hi, kMaxH));
            want = true;
        }
    }
    if (!want) {
        b.lo0 = b.lo1 = b.lo2 = kBig;
        b.hi0 = b.hi1 = b.hi2 = -kBig;
    }
    uint32_t blo = kGuards, bhi = 0u;  // the group's box, relative to the staged box
    if (want) {
        blo = pack_cell(b.lo0 - (lo0 << us), b.lo1 - (lo1 << us), b.lo2 - (lo2 << us));
        bhi = pack_cell(b.hi0 - (lo0 << us), b.hi1 - (lo1 << us), b.hi2 - (lo2 << us));
    }
    const int u0 = __reduce_min_sync(kFull, b.lo0) >> us, u1 = __reduce_min_sync(kFull, b.lo1) >> us,
              u2 = __reduce_min_sync(kFull, b.lo2) >> us;
    const int v0 = __reduce_max_sync(kFull, b.hi0) >> us, v1 = __reduce_max_sync(kFull, b.hi1) >> us,
              v2 = __reduce_max_sync(kFull, b.hi2) >> us;
    if (u0 > v0) return __reduce_min_sync(kFull, idt_inactive);  // no active particle takes the tile path
    __syncwarp();
    // every accepted pair lies within 2 max(h_i, largest staged h) of the particle
    const float hm = fmaxf(I.hi, __int_as_float(S.hmax_bits));
    const Reach4 reach(I.xi, I.yi, I.zi, want ? 4.f * hm * hm : -1.f);
    F2 nx[kTileGpw / 2], ny2[kTileGpw / 2], nz2[kTileGpw / 2];  // minus the positions, two particles each
    float qr[kTileGpw];
    uint32_t klo[kTileGpw], khi[kTileGpw];
#pragma unroll
    for (int k = 0; k < kTileGpw; ++k) {
        qr[k] = __shfl_sync(kFull, want ? I.hi2x4 : -1.f, k * L);
        klo[k] = __shfl_sync(kFull, blo, k * L);
        khi[k] = __shfl_sync(kFull, bhi, k * L);
    }
#pragma unroll
    for (int k = 0; k < kTileGpw / 2; ++k) {
        nx[k] = f2(-__shfl_sync(kFull, I.xi, 2 * k * L), -__shfl_sync(kFull, I.xi, (2 * k + 1) * L));
        ny2[k] = f2(-__shfl_sync(kFull, I.yi, 2 * k * L), -__shfl_sync(kFull, I.yi, (2 * k + 1) * L));
        nz2[k] = f2(-__shfl_sync(kFull, I.zi, 2 * k * L), -__shfl_sync(kFull, I.zi, (2 * k + 1) * L));
    }
    uint16_t (*const lists)[kTileAccList] = &S.list[wslot * kTileGpw];
    int cnt[kTileGpw] = {};
    const unsigned below = (1u << lane) - 1u;
    const int nyu = v1 - u1 + 1;
    const int rows = (v0 - u0 + 1) * nyu;
    for (int rb = 0; rb < rows; rb += 32) {
        const int r = rb + lane;
        uint32_t len = 0u, s0 = 0u;
        if (r < rows) {
            // the row's z range that an accepted pair of the four can have
            const int x = u0 + r / nyu, y = u1 + r % nyu;
            int zl, zh;
            if (reach.row(x, y, uw, uiw, zl, zh)) {
                zl = max(zl, u2);
                zh = min(zh, v2);
                if (zl <= zh) {
                    const int c0 = ((x - lo0) * ny + (y - lo1)) * nz;
                    s0 = S.off[c0 + (zl - lo2)];
                    len = S.off[c0 + (zh - lo2) + 1] - s0;
                }
            }
        }
        uint32_t pre = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, pre, o);
            if (lane >= o) pre += t;
        }
        const uint32_t excl = pre - len;
        const uint32_t total = __shfl_sync(kFull, pre, 31);
        s0 -= excl;  // staged slot of flat index v in this row: s0 + v
        for (uint32_t vb = 0; vb < total; vb += 32u) {
            const uint32_t v = vb + (uint32_t)lane;
            int j = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t e = __shfl_sync(kFull, excl, j + step);
                if (e <= v) j += step;
            }
            const uint32_t s = __shfl_sync(kFull, s0, j) + v;
            float4 q = make_float4(3e38f, 3e38f, 3e38f, 0.f);
            uint32_t sc = 0u;
            if (v < total) {
                q = S.pos[s];
                sc = S.scell[s];
            }
            const float hj2x4 = q.w * q.w * 4.f;
            const F2 qx = f2(q.x), qy = f2(q.y), qz = f2(q.z);
            float d[kTileGpw];
#pragma unroll
            for (int k = 0; k < kTileGpw / 2; ++k) {
                const F2 dx = qx + nx[k], dy = qy + ny2[k], dz = qz + nz2[k];
                unpack(fma2(dz, dz, fma2(dy, dy, dx * dx)), d[2 * k], d[2 * k + 1]);
            }
#pragma unroll
            for (int k = 0; k < kTileGpw; ++k) {
                // r <= 2 h_i, or r <= 2 h_j with the neighbour's cell in the
                // particle's box (empty for a group that takes no part)
                const bool hit = d[k] >= 1e-12f && (d[k] <= qr[k] || (d[k] <= hj2x4 && in_box(sc, klo[k], khi[k])));
                const unsigned bal = __ballot_sync(kFull, hit);
                const int at = cnt[k] + __popc(bal & below);
                if (hit && at < kTileAccList) lists[k][at] = (uint16_t)s;
                cnt[k] += __popc(bal);
            }
        }
    }
    __syncwarp();
    int n_list = 0;
#pragma unroll
    for (int k = 0; k < kTileGpw; ++k)
        if (g == k) n_list = cnt[k];
    if (live && n_list > kTileAccList) {
        if (sub == 0) deferred[atomicAdd(dctr, 1u)] = p;
        live = false;
    }
    const int maxn = __reduce_max_sync(kFull, live ? n_list : 0);
    AccelSum2 S2;
    const float hi2 = I.hi1 * I.hi1, fac_i = kPi1 * hi2 * hi2;
    for (int i = sub; i < maxn; i += 2 * L) {
        // (past the list's end: no mass, no relative motion, far away)
        const float4 none = make_float4(I.xi + 1e15f, I.yi, I.zi, 1.f);
        float4 Aj[2] = {none, none}, Bj[2], Cj[2];
        Bj[0] = Bj[1] = make_float4(I.vxi, I.vyi, I.vzi, -1e30f);
        Cj[0] = Cj[1] = make_float4(0.f, 0.f, 1.f, 0.f);
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (live && i + e * L < n_list) {
                const uint32_t s = list[i + e * L];
                const uint32_t gj = S.gidx[s];
                Aj[e] = S.pos[s];
                Bj[e] = __ldg(a.sB + gj);
                Cj[e] = __ldg(a.sC + gj);
            }
        accel_pair2<KAHAN>(I, fac_i, S2, Aj, Bj, Cj);
    }
    AccelSum Sm = accel_close<KAHAN>(S2);
    accel_reduce<L, false>(Sm, kFull);
    int idt = idt_inactive;
    if (live) {
        idt = accel_ticks(I, Sm.vsig);
        if (sub == 0) accel_store(a, ind, Sm, idt);
    }
    return __reduce_min_sync(kFull, idt);
}

__global__ void __launch_bounds__(256) k_acceleration_plan(AccelArgs a, uint2 *tiles, uint32_t *ctr,
                                                           uint32_t block_max, uint32_t half_max, uint32_t big_max) {
    tile_plan(a.n, a.skey, a.cells, a.cflags, a.mode, tiles, ctr, block_max, half_max, big_max, [&](int p) -> uint8_t {
        const float4 A = a.sA[p];
        if (!a.active[a.cidx[p]]) return kModeInactive;
        CellBox b;
        const int m = accel_mode(A.x, A.y, A.z, A.w, b, a.coarse);
        if (m < 0) return kModeWalk;
        // the list is complete when no neighbour the box can hold has outgrown it
        // (a NaN h counts as larger than any; a list without the neighbours' own
        // reach has a negative one)
        if (a.lists.entries && a.lists.count[p] != kNoList) {
            int grown = 0;
            for (int x = b.lo0 >> kUnitShift; x <= b.hi0 >> kUnitShift; ++x)
                for (int y = b.lo1 >> kUnitShift; y <= b.hi1 >> kUnitShift; ++y)
                    for (int z = b.lo2 >> kUnitShift; z <= b.hi2 >> kUnitShift; ++z) {
                        const int mask = (kCellsPerDim >> kUnitShift) - 1;
                        grown = max(grown, __ldg(a.lists.grown + morton3((uint32_t)(x & mask), (uint32_t)(y & mask),
                                                                         (uint32_t)(z & mask))));
                    }
            const float hg = __int_as_float(grown);
            if (4.f * hg * hg <= 0.9999f * a.lists.reach2[p]) return kModeList;
        }
        return (uint8_t)m;
    });
}

// The acceleration tile pass U over `tiles` (ctr[0] of them, ctr[1] the
// ticket), staged and taken as in k_lists; deferred particles are counted in
// *dctr.
template <bool KAHAN, int U>
__global__ void __launch_bounds__(kTileThreads, 2)
    k_acceleration_tile(AccelArgs a, const uint2 *__restrict__ tiles, uint32_t *ctr, uint32_t *__restrict__ deferred,
                        uint32_t *dctr) {
    extern __shared__ float4 s_tile_raw[];
    TileAccShared &S = *reinterpret_cast<TileAccShared *>(s_tile_raw);
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) S.dtmin = 0x7fffffff;
    const uint32_t ntiles = ctr[0];
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            const uint32_t t = atomicAdd(ctr + 1, 1u);
            S.tile = t;
            if (t < ntiles) {
                const uint2 r = tiles[t];
                S.start = r.x;
                S.end = r.y;
            }
        }
        __syncthreads();
        if (S.tile >= ntiles) break;
        const uint32_t tstart = S.start, tend = S.end;
        // a tile whose staged box overflows shared memory is taken again as
        // its octets (coarse tiles: its units), one at a time; one that still
        // overflows is handed to the per-particle pass
        constexpr int kSplit = U == 0 ? 3 : 3 * U;
        const bool splittable = (a.skey[tstart] >> kSplit) != (a.skey[tend - 1] >> kSplit);
        bool whole = true;
        uint32_t r0 = tstart;
        while (r0 < tend) {
            __syncthreads();
            if (tid == 0) {
                uint32_t r1 = tend;
                if (!whole) {  // the rest of r0's octet / unit
                    const uint32_t o = a.skey[r0] >> kSplit;
                    r1 = r0 + 1u;
                    if (U == 0) {
                        for (int j = 0; j < 8; ++j) {
                            const uint2 r = a.cells[o * 8u + (uint32_t)j];
                            if (r.x != 0xffffffffu) r1 = max(r1, r.y + 1u);
                        }
                    } else {
                        r1 = max(r1, a.units[o].y + 1u);
                    }
                }
                S.end = r1;
                S.next = 0u;
                S.box[0] = S.box[1] = S.box[2] = 0x7fffffff;
                S.box[3] = S.box[4] = S.box[5] = -0x7fffffff;
                S.defer_all = 0;
                S.need = 0;
                S.hmax_bits = 0;
            }
            __syncthreads();
            const uint32_t start = r0, end = S.end;
            {
                int b[6] = {0x7fffffff, 0x7fffffff, 0x7fffffff, -0x7fffffff, -0x7fffffff, -0x7fffffff};
                // the warp pass is needed for this pass's particles and, in the
                // cell-tile pass, for the inactive (their next active time bounds
                // the step) and deferred ones
                bool need = false;
                for (uint32_t p = start + tid; p < end; p += kTileThreads) {
                    const uint8_t m = a.mode[p];
                    need |= m == U || (U == 0 && m >= kModeWalk);
                    if (m != U) continue;
                    const float4 A = a.sA[p];
                    const CellBox cb = cell_box(A.x, A.y, A.z, fmin_ref(A.w, kMaxH));
                    b[0] = min(b[0], cb.lo0);
                    b[1] = min(b[1], cb.lo1);
                    b[2] = min(b[2], cb.lo2);
                    b[3] = max(b[3], cb.hi0);
                    b[4] = max(b[4], cb.hi1);
                    b[5] = max(b[5], cb.hi2);
                }
    #pragma unroll
                for (int k = 0; k < 3; ++k) {
                    b[k] = __reduce_min_sync(0xffffffffu, b[k]);
                    b[k + 3] = __reduce_max_sync(0xffffffffu, b[k + 3]);
                }
                if (__any_sync(0xffffffffu, need) && lane == 0) S.need = 1;
                if (lane == 0) {
    #pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        atomicMin(&S.box[k], b[k]);
                        atomicMax(&S.box[k + 3], b[k + 3]);
                    }
                }
            }
            __syncthreads();
            if (!S.need) {  // nothing in the range for this pass
                r0 = end;
                continue;
            }
            const bool any = S.box[0] <= S.box[3];
            const int us = unit_shift<U>(S.box);
            const int lo0 = S.box[0] >> us, lo1 = S.box[1] >> us, lo2 = S.box[2] >> us;
            const int nx = any ? box_extent(S.box[0], S.box[3], us) : 0, ny = any ? box_extent(S.box[1], S.box[4], us) : 0,
                      nz = any ? box_extent(S.box[2], S.box[5], us) : 0;
            int ncell = 0;
            if (any) {
                static_assert(kCellsPerDim <= kBoxCellsMax, "a box that is staged has cells within pack_cell's range");
                if (box_units(nx, ny, nz) > kTileCellsMax) {
                    if (tid == 0) S.defer_all = 1;
                } else {
                    ncell = nx * ny * nz;
                }
            }
            uint32_t c_cnt[kTileCellsPerThread], c_first[kTileCellsPerThread];
            uint32_t tsum = 0u;
    #pragma unroll
            for (int k = 0; k < kTileCellsPerThread; ++k) {
                const int c = kTileCellsPerThread * tid + k;
                c_cnt[k] = c_first[k] = 0u;
                if (c < ncell) {
                    const int ix = c / (ny * nz), rem = c - ix * ny * nz, iy = rem / nz, iz = rem - iy * nz;
                    const uint2 r = unit_range(a.cells, a.octets, a.units, us, lo0 + ix, lo1 + iy, lo2 + iz);
                    if (r.x != 0xffffffffu) {
                        c_cnt[k] = r.y - r.x + 1u;
                        c_first[k] = r.x;
                    }
                }
                tsum += c_cnt[k];
            }
            uint32_t inc = tsum;
    #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane == 31) S.wsum[tid >> 5] = inc;
            __syncthreads();
            uint32_t wbase = 0u;
            for (int w = 0; w < (tid >> 5); ++w) wbase += S.wsum[w];
            uint32_t run = wbase + inc - tsum;
    #pragma unroll
            for (int k = 0; k < kTileCellsPerThread; ++k) {
                const int c = kTileCellsPerThread * tid + k;
                if (c < ncell) S.off[c] = run;
                run += c_cnt[k];
            }
            if (tid == kTileThreads - 1) {
                S.off[ncell] = run;
                if (run > (uint32_t)kTileAccStage) S.defer_all = 1;
            }
            __syncthreads();
            if (S.defer_all && whole && splittable) {
                whole = false;
                continue;
            }
            float hmax = 0.f;
            if (!S.defer_all) {
                stage_units(c_cnt, c_first, inc - tsum, inc, lane, [&](uint32_t v, uint32_t g, int c) {
                    const float4 q = __ldg(a.sA + g);
                    c += kTileCellsPerThread * (tid - lane);
                    int ix = c / (ny * nz), rem = c - ix * ny * nz, iy = rem / nz, iz = rem - iy * nz;
                    if (U > 0) {
                        // the particle's cell within its unit: the low bits of its key
                        const uint32_t key = a.skey[g];
                        int dx = 0, dy = 0, dz = 0;
#pragma unroll
                        for (int bit = 0; bit < kUnitShift; ++bit) {
                            dx |= (int)((key >> (3 * bit)) & 1u) << bit;
                            dy |= (int)((key >> (3 * bit + 1)) & 1u) << bit;
                            dz |= (int)((key >> (3 * bit + 2)) & 1u) << bit;
                        }
                        const int low = (1 << us) - 1;
                        ix = (ix << us) | (dx & low);
                        iy = (iy << us) | (dy & low);
                        iz = (iz << us) | (dz & low);
                    }
                    S.pos[wbase + v] = q;
                    S.gidx[wbase + v] = g;
                    S.scell[wbase + v] = pack_cell(ix, iy, iz);
                    hmax = fmaxf(hmax, q.w);
                });
            }
            {
                float v = hmax;
    #pragma unroll
                for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
                if (lane == 0 && v > 0.f) atomicMax(&S.hmax_bits, __float_as_int(v));
            }
            __syncthreads();
            int wmin = 0x7fffffff;
            for (bool more = true; more;) {
                uint32_t j = 0u;
                if (lane == 0) j = atomicAdd(&S.next, (uint32_t)kTileGpw);
                j = __shfl_sync(0xffffffffu, j, 0);
                more = start + j < end;
                if (!more) break;
                wmin = min(wmin, accel_tile_warp<KAHAN, U>(a, S, start + j, end, lane, tid >> 5, deferred, dctr));
            }
            if (lane == 0 && wmin != 0x7fffffff) atomicMin(&S.dtmin, wmin);
            r0 = end;
        }
    }
    if (tid == 0 && S.dtmin != 0x7fffffff) atomicMin(a.globals + 1, S.dtmin);
}

// The particles whose list the density pass left (kModeList): eight lanes
// each, two neighbours per lane and step, all neighbour records read by sorted
// index (they are neighbours in that order too, so most come from L1).  Same
// pairs and arithmetic as the tiles; what is saved is the search, which was
// 70 % of a tile's time.  Measured, acceleration pass at N = 1e6: 1.61 -> 0.86 ms
// (24 warps per SM; with 32 and spilled sums 0.93).
template <bool KAHAN>
__global__ void __launch_bounds__(kListThreads, 3) k_acceleration_list(AccelArgs a) {
    constexpr int L = kTileLanes;
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & (L - 1);
    const int p = (int)((blockIdx.x * (unsigned)kListThreads + threadIdx.x) / L);
    const bool live = p < a.n && a.mode[p] == kModeList;
    int idt = 0x7fffffff;
    if (__any_sync(kFull, live)) {
        float4 A = make_float4(0.f, 0.f, 0.f, 1.f), Bv = A, Cv = A;
        int n_list = 0;
        if (live) {
            A = a.sA[p];
            Bv = a.sB[p];
            Cv = a.sC[p];
            n_list = a.lists.count[p];
        }
        const AccelI I = accel_i(A, Bv, Cv);
        CellBox box = cell_box(I.xi, I.yi, I.zi, fmin_ref(I.hi, kMaxH));
        const uint32_t *list = a.lists.entries + (size_t)(live ? p : 0) * kTileList;
        const float hi2 = I.hi1 * I.hi1, fac_i = kPi1 * hi2 * hi2;
        const int maxn = __reduce_max_sync(kFull, n_list);
        AccelSum2 S2;
        // the sorted index behind list entry i, this particle's own past the end
        const int self = min(p, a.n - 1);
        auto entry = [&](int i) { return i < n_list ? (int)__ldg(list + i) : self; };
        int g[2] = {entry(sub), entry(sub + L)};
        float4 Aj[2] = {__ldg(a.sA + g[0]), __ldg(a.sA + g[1])};
#pragma unroll 1
        for (int i = sub; i < maxn; i += 2 * L) {
            // the next step's neighbours are on their way while this one's count
            const int gn[2] = {entry(i + 2 * L), entry(i + 3 * L)};
            float4 Bj[2], Cj[2], An[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                Bj[e] = __ldg(a.sB + g[e]);
                Cj[e] = __ldg(a.sC + g[e]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) An[e] = __ldg(a.sA + gn[e]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float dx = Aj[e].x - I.xi, dy = Aj[e].y - I.yi, dz = Aj[e].z - I.zi;
                const float d = dx * dx + dy * dy + dz * dz;
                bool hit = d >= 1e-12f && d <= I.hi2x4;
                if (!hit && d >= 1e-12f && d <= Aj[e].w * Aj[e].w * 4.f) {
                    // seen only through the neighbour's h: only when its
                    // cell lies in the particle's box
                    const int cx = (int)floorf(__fdiv_rn(Aj[e].x, kCellWidth)),
                              cy = (int)floorf(__fdiv_rn(Aj[e].y, kCellWidth)),
                              cz = (int)floorf(__fdiv_rn(Aj[e].z, kCellWidth));
                    hit = cx >= box.lo0 && cx <= box.hi0 && cy >= box.lo1 && cy <= box.hi1 && cz >= box.lo2 &&
                          cz <= box.hi2;
                }
                if (!hit || i + e * L >= n_list) {
                    // no pair: no mass, no relative motion, far away
                    Aj[e] = make_float4(I.xi + 1e15f, I.yi, I.zi, 1.f);
                    Bj[e] = make_float4(I.vxi, I.vyi, I.vzi, -1e30f);
                    Cj[e] = make_float4(0.f, 0.f, 1.f, 0.f);
                }
            }
            accel_pair2<KAHAN>(I, fac_i, S2, Aj, Bj, Cj);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                g[e] = gn[e];
                Aj[e] = An[e];
            }
        }
        AccelSum Sm = accel_close<KAHAN>(S2);
        accel_reduce<L, false>(Sm, kFull);
        if (live) {
            idt = accel_ticks(I, Sm.vsig);
            if (sub == 0) accel_store(a, a.cidx[p], Sm, idt);
        }
    }
    idt = __reduce_min_sync(kFull, idt);
    if (lane == 0 && idt < *(volatile int32_t *)(a.globals + 1)) atomicMin(a.globals + 1, idt);
}

struct StepArgs {
    int n;
    float4 *pos4, *vel4;
    const float4 *acc4;
    float *rho, *u, *h;
    const float *du, *dhdt;
    int32_t *globals;
    double4 *pos64;  // mixed-precision form: FP64 master positions
    double *dglob;   // mixed-precision form: [0] global time in seconds
};

// step.metal:12-46.  Every thread reads dt before thread 0 advances the
// global time in a separate word, as in the reference.  MIXED: the drift is
// added to FP64 positions, and the float positions are their roundings; the
// global time is also kept in FP64 seconds.
template <bool MIXED>
__global__ void k_step(StepArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const int32_t ticks = a.globals[1];
    const float dt = kDtMin1 * (float)ticks;
    if (i == 0) {
        a.globals[0] += ticks;
        if (MIXED) a.dglob[0] += (double)kDtMin1 * (double)ticks;
    }
    float4 v = a.vel4[i];
    const float4 ac = a.acc4[i];
    const float hi = a.h[i];
    const float h1 = 1.f / hi;
    const float dh = a.dhdt[i];
    a.h[i] = fmin_ref(hi * expf(h1 * dh * dt), kMaxH);
    a.rho[i] *= expf(-3.f * h1 * dh * dt);
    a.vel4[i] = make_float4(v.x + dt * ac.x, v.y + dt * ac.y, v.z + dt * ac.z, v.w);
    a.u[i] += dt * a.du[i];
    float4 p = a.pos4[i];
    const float dx = dt * v.x + 0.5f * ac.x * dt * dt;
    const float dy = dt * v.y + 0.5f * ac.y * dt * dt;
    const float dz = dt * v.z + 0.5f * ac.z * dt * dt;
    if (MIXED) {
        double4 q = a.pos64[i];
        q.x += (double)dx;
        q.y += (double)dy;
        q.z += (double)dz;
        a.pos64[i] = q;
        p.x = (float)q.x;
        p.y = (float)q.y;
        p.z = (float)q.z;
    } else {
        p.x += dx;
        p.y += dy;
        p.z += dz;
    }
    a.pos4[i] = p;
}

__global__ void k_pos_to64(int n, const float4 *__restrict__ pos4, double4 *__restrict__ pos64) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos4[i];
    pos64[i] = make_double4((double)p.x, (double)p.y, (double)p.z, 0.0);
}

// FP64 conservation sums per block: mass, kinetic, internal and potential
// energy, momentum, angular momentum about the origin (FP64 positions when
// present); one record of kDiag doubles per block, summed in block order by
// k_diag_total so the result does not depend on scheduling.
constexpr int kDiagThreads = 256;
__global__ void __launch_bounds__(kDiagThreads) k_diag_block(int n, const float4 *__restrict__ pos4,
                                                                const double4 *__restrict__ pos64,
                                                                const float4 *__restrict__ vel4,
                                                                const float *__restrict__ u,
                                                                const float *__restrict__ phi, double *out) {
    __shared__ double red[kDiag][kDiagThreads / 32];
    double v[kDiag];
#pragma unroll
    for (int k = 0; k < kDiag; ++k) v[k] = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = pos4[i];
        const double m = (double)p.w;
        double x = p.x, y = p.y, z = p.z;
        if (pos64) {
            const double4 q = pos64[i];
            x = q.x;
            y = q.y;
            z = q.z;
        }
        const float4 w = vel4[i];
        const double vx = w.x, vy = w.y, vz = w.z;
        v[0] += m;
        v[1] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
        v[2] += m * (double)u[i];
        v[3] += 0.5 * m * (double)phi[i];
        v[4] += m * vx;
        v[5] += m * vy;
        v[6] += m * vz;
        v[7] += m * (y * vz - z * vy);
        v[8] += m * (z * vx - x * vz);
        v[9] += m * (x * vy - y * vx);
    }
#pragma unroll
    for (int k = 0; k < kDiag; ++k) {
        double x = v[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = x;
    }
    __syncthreads();
    if (threadIdx.x < kDiag) {
        double t = 0.0;
        for (int w = 0; w < kDiagThreads / 32; ++w) t += red[threadIdx.x][w];
        out[(size_t)blockIdx.x * kDiag + threadIdx.x] = t;
    }
}

__global__ void k_diag_total(int blocks, double *partials, double *total) {
    const int k = threadIdx.x;
    if (k >= kDiag) return;
    double t = 0.0;
    for (int b = 0; b < blocks; ++b) t += partials[(size_t)b * kDiag + k];
    total[k] = t;
}

// render.metal:49-66
__global__ void k_snapshot(int n, const float4 *__restrict__ pos4, const int32_t *__restrict__ mat, int32_t *img) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float R_E = 6.3710f;
    float4 p = pos4[i];
    float ux = p.x, uy = p.y;
    ux -= 250.f;
    uy -= 250.f;
    const float s = kSnapshotRes / (20.f * R_E);
    ux *= s;
    uy *= s;
    if (ux < 0.f || uy < 0.f || ux > (float)kSnapshotRes || uy > (float)kSnapshotRes) return;
    int px = (int)ux, py = (int)uy;
    long pixel = (long)px + (long)(kSnapshotRes - 1 - py) * kSnapshotRes;
    // uv == SNAPSHOT_RESOLUTION exactly would index one past the image in the
    // reference; those splats are dropped here
    if (pixel < 0 || pixel >= (long)kSnapshotRes * kSnapshotRes || px >= kSnapshotRes) return;
    atomicMax(img + pixel, mat[i]);
}

// Dynamic shared memory of the walks' lists.
template <int L>
constexpr size_t list_smem() {
    return sizeof(uint32_t) * parts_per_block<L>() * kListMax;
}
#ifdef SPH_PARITY
// Above 48 KiB: the per-device opt-in, set once per device.
void list_smem_opt_in() {
    constexpr int smem = (int)list_smem<kParityLanes>();
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(k_density<kParityLanes>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(k_acceleration<kParityLanes, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(k_acceleration<kParityLanes, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        done[dev] = true;
    }
}
#endif

// Shared memory of the tile kernels (above 48 KiB: the per-device opt-in) and
// the device's SM count, set up once per device.
int tile_smem_opt_in() {
    static int sms[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!sms[dev]) {
        cudaFuncSetAttribute(k_lists<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ListShared<0>));
        cudaFuncSetAttribute(k_lists<kUnitShift>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(ListShared<kUnitShift>));
        cudaFuncSetAttribute(k_acceleration_tile<false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(TileAccShared));
        cudaFuncSetAttribute(k_acceleration_tile<true, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(TileAccShared));
        cudaFuncSetAttribute(k_acceleration_tile<false, kUnitShift>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(TileAccShared));
        cudaFuncSetAttribute(k_acceleration_tile<true, kUnitShift>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(TileAccShared));
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        sms[dev] = v > 0 ? v : 148;
    }
    return sms[dev];
}

// Persistent CTAs of the tile passes: as many as are resident, but no more
// than one per ~48 particles (a tile holds ~100-300), so a small context -- an
// ensemble instance -- leaves the rest of the device to the others.
unsigned tile_grid(int n, int resident) {
    const int want = (n + 47) / 48;
    return (unsigned)std::max(1, std::min(resident, want));
}

}  // namespace

size_t neighbour_list_entries(int n) { return (size_t)n * kTileList; }

sph_status launch_density(sph_ctx *ctx, cudaStream_t st) {
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    const uint32_t *cidx = ctx->cell_sort.vals[ctx->cell_final];
    k_gather<<<(n + 255) / 256, 256, 0, st>>>(n, cidx, ctx->pos4, ctx->vel4, ctx->sp4, ctx->sv4);
    DensityArgs a;
    a.n = n;
    a.cidx = cidx;
    a.skey = ctx->cell_sort.keys[ctx->cell_final];
    a.cells = ctx->cell_range;
    a.octets = ctx->octets;
    a.units = ctx->units;
    a.cflags = ctx->coarse_flags;
    a.coarse = ctx->tile_coarse;
    a.mode = ctx->tile_mode;
    a.first_h = ctx->tile_first_h;
    a.start_h = ctx->tile_h;
    a.lists = NeighbourLists{ctx->nlist, 0, n, ctx->nlist_count, ctx->nlist_reach2, ctx->grown};
    a.sp4 = ctx->sp4;
    a.sv4 = ctx->sv4;
    a.h = ctx->h;
    a.rho = ctx->rho;
    a.f = ctx->f;
    a.P = ctx->P;
    a.c = ctx->c;
    a.B = ctx->B;
    a.u = ctx->u;
    a.mat = ctx->mat;
    a.active = ctx->active;
    a.sA = ctx->sA;
    a.sB = ctx->sB;
    a.sC = ctx->sC;
    a.globals = ctx->globals;
    a.health = ctx->health;
    a.eos = ctx->eos;
    a.eta = ctx->form.h_tolerance > 0.f ? ctx->form.h_tolerance : kDensityEta;
    a.seed = nullptr;
    a.nn_out = ctx->hs.nn;
    a.stats = ctx->hs.stats;
    sph_status s = SPH_OK;
    // the learned seed's online refresh, unless a full step ran it ahead
    if (hseed_online_due(ctx) && !ctx->hs.trained_ahead) s = launch_hseed_online(ctx, st);
    if (s != SPH_OK) return s;
    if (ctx->hs.stats) cudaMemsetAsync(ctx->hs.stats, 0, sizeof(uint32_t) * 4, st);
    if (ctx->hs.capture) s = launch_hseed_capture(ctx, st);
    if (s == SPH_OK && ctx->form.h_seed == SPH_HSEED_LEARNED) {
        s = launch_hseed_infer(ctx, st);
        a.seed = ctx->hs.seed;
    }
    if (s != SPH_OK) return s;
    a.nn_out = ctx->hs.nn;
    a.stats = ctx->hs.stats;
#ifdef SPH_PARITY
    constexpr int parts = parts_per_block<kParityLanes>();
    list_smem_opt_in();
    k_density<kParityLanes><<<(unsigned)((n + parts - 1) / parts), parts * kParityLanes, list_smem<kParityLanes>(),
                              st>>>(a);
#else
    // the lists over cell tiles, then over the coarse tiles of the flagged
    // blocks (the tile list is reused); the iteration; the per-particle pass
    // over what it deferred
    const int sms = tile_smem_opt_in();
    uint32_t *ctr = ctx->tile_ctr;
    cudaMemsetAsync(ctr, 0, sizeof(uint32_t) * 8, st);
    cudaMemsetAsync(ctx->grown, 0, sizeof(int) * kNumUnits, st);
    k_density_plan<<<(n + 255) / 256, 256, 0, st>>>(a, ctx->tiles, ctr, ctx->tile_block_max, ctx->tile_half_max,
                                                    ctx->tile_big_max);
    auto search = [&](auto unit, uint32_t *c) {
        constexpr int U = decltype(unit)::value;
        k_lists<U><<<tile_grid(n, sms * ListTile<U>::kCtas), ListTile<U>::kThreads, sizeof(ListShared<U>), st>>>(
            a, ctx->tiles, c);
    };
    auto iterate = [&](int only) {
        const unsigned grid =
            (unsigned)(((int64_t)(a.lists.last - a.lists.first) * kTileLanes + kListThreads - 1) / kListThreads);
        k_density_list<<<grid, kListThreads, 0, st>>>(a, only, ctx->deferred, ctr + 2);
    };
    auto coarse_starts = [&]() {
        k_coarse_starts<<<(n + 255) / 256, 256, 0, st>>>(n, a.skey, ctx->units, ctx->coarse_flags, ctx->tiles,
                                                         ctr + 4);
    };
    using Cells = std::integral_constant<int, 0>;
    using Units = std::integral_constant<int, kUnitShift>;
    const int room = ctx->nlist ? std::min(ctx->list_room, n) : 0;
    if (room == n) {
        search(Cells{}, ctr);
        if (a.coarse) {
            coarse_starts();
            search(Units{}, ctr + 4);
        }
        iterate(kAllModes);
    } else if (room == 0) {
        // (every particle is left to the walk; the coarse tiles' flags stay for
        // the acceleration pass, which sets the same and more)
        iterate(kAllModes);
    } else {
        // lists of a slice of the sorted order at a time; the tile list holds
        // one kind of tiles, so first all slices of the one, then of the other
        auto slices = [&](auto unit, uint32_t *c) {
            for (int64_t first = 0; first < n; first += room) {
                a.lists.first = (int)first;
                a.lists.last = (int)std::min<int64_t>(n, first + room);
                if (first > 0) cudaMemsetAsync(c + 1, 0, sizeof(uint32_t), st);
                search(unit, c);
                iterate(decltype(unit)::value);
            }
        };
        slices(Cells{}, ctr);
        if (a.coarse) {
            coarse_starts();
            slices(Units{}, ctr + 4);
        }
    }
    k_density_deferred<kWalkLanes>
        <<<tile_grid(n, sms * 2) * 4, parts_per_block<kWalkLanes>() * kWalkLanes, list_smem<kWalkLanes>(), st>>>(
            a, ctx->deferred, ctr + 2);
#endif
    if (ctx->hs.capture) s = launch_hseed_targets(ctx, st);
    if (s != SPH_OK) return s;
    return cuda_status(cudaGetLastError(), "density");
}

sph_status launch_acceleration(sph_ctx *ctx, cudaStream_t st) {
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    AccelArgs a;
    a.n = n;
    a.cidx = ctx->cell_sort.vals[ctx->cell_final];
    a.skey = ctx->cell_sort.keys[ctx->cell_final];
    a.cells = ctx->cell_range;
    a.octets = ctx->octets;
    a.units = ctx->units;
    a.cflags = ctx->coarse_flags;
    a.coarse = ctx->tile_coarse;
    a.mode = ctx->tile_mode;
    const bool whole = ctx->nlist && ctx->list_room >= n;  // every particle's list is there
    a.lists = NeighbourLists{whole ? ctx->nlist : nullptr, 0, n, ctx->nlist_count, ctx->nlist_reach2, ctx->grown};
    a.sA = ctx->sA;
    a.sB = ctx->sB;
    a.sC = ctx->sC;
    a.acc4 = ctx->acc4;
    a.du = ctx->du;
    a.dhdt = ctx->dhdt;
    a.nat = ctx->nat;
    a.active = ctx->active;
    a.globals = ctx->globals;
    a.individual = ctx->form.timestep == SPH_TIMESTEP_INDIVIDUAL;
    const bool kahan = ctx->form.precision == SPH_PRECISION_MIXED;
#ifdef SPH_PARITY
    constexpr int parts = parts_per_block<kParityLanes>();
    constexpr size_t smem = list_smem<kParityLanes>();
    const unsigned blocks = (unsigned)((n + parts - 1) / parts);
    list_smem_opt_in();
    if (kahan)
        k_acceleration<kParityLanes, true><<<blocks, parts * kParityLanes, smem, st>>>(a);
    else
        k_acceleration<kParityLanes, false><<<blocks, parts * kParityLanes, smem, st>>>(a);
#else
    constexpr size_t smem = list_smem<kWalkLanes>();
    // the density pass's tiles, rebuilt so the pass also stands alone; its own
    // counters (tile_ctr[8..15]); then the coarse tiles and the deferred
    const int sms = tile_smem_opt_in();
    uint32_t *ctr = ctx->tile_ctr + 8;
    cudaMemsetAsync(ctr, 0, sizeof(uint32_t) * 8, st);
    k_acceleration_plan<<<(n + 255) / 256, 256, 0, st>>>(a, ctx->tiles, ctr, ctx->tile_block_max,
                                                         ctx->tile_half_max, ctx->tile_big_max);
    const unsigned tgrid = tile_grid(n, sms * 2);
    const size_t tsm = sizeof(TileAccShared);
    if (whole) {
        const unsigned lgrid = (unsigned)(((int64_t)n * kTileLanes + kListThreads - 1) / kListThreads);
        if (kahan) k_acceleration_list<true><<<lgrid, kListThreads, 0, st>>>(a);
        else k_acceleration_list<false><<<lgrid, kListThreads, 0, st>>>(a);
    }
    if (kahan)
        k_acceleration_tile<true, 0><<<tgrid, kTileThreads, tsm, st>>>(a, ctx->tiles, ctr, ctx->deferred, ctr + 2);
    else
        k_acceleration_tile<false, 0><<<tgrid, kTileThreads, tsm, st>>>(a, ctx->tiles, ctr, ctx->deferred, ctr + 2);
    if (a.coarse) {
        k_coarse_starts<<<(n + 255) / 256, 256, 0, st>>>(n, a.skey, ctx->units, ctx->coarse_flags, ctx->tiles,
                                                         ctr + 4);
        if (kahan)
            k_acceleration_tile<true, kUnitShift>
                <<<tgrid, kTileThreads, tsm, st>>>(a, ctx->tiles, ctr + 4, ctx->deferred, ctr + 2);
        else
            k_acceleration_tile<false, kUnitShift>
                <<<tgrid, kTileThreads, tsm, st>>>(a, ctx->tiles, ctr + 4, ctx->deferred, ctr + 2);
    }
    if (kahan)
        k_acceleration_deferred<kWalkLanes, true>
            <<<tgrid * 4, parts_per_block<kWalkLanes>() * kWalkLanes, smem, st>>>(a, ctx->deferred, ctr + 2);
    else
        k_acceleration_deferred<kWalkLanes, false>
            <<<tgrid * 4, parts_per_block<kWalkLanes>() * kWalkLanes, smem, st>>>(a, ctx->deferred, ctr + 2);
#endif
    return cuda_status(cudaGetLastError(), "acceleration");
}

sph_status launch_step(sph_ctx *ctx, cudaStream_t st) {
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    StepArgs a;
    a.n = n;
    a.pos4 = ctx->pos4;
    a.vel4 = ctx->vel4;
    a.acc4 = ctx->acc4;
    a.rho = ctx->rho;
    a.u = ctx->u;
    a.h = ctx->h;
    a.du = ctx->du;
    a.dhdt = ctx->dhdt;
    a.globals = ctx->globals;
    a.pos64 = ctx->pos64;
    a.dglob = ctx->dglob;
    if (ctx->form.precision == SPH_PRECISION_MIXED)
        k_step<true><<<(n + 255) / 256, 256, 0, st>>>(a);
    else
        k_step<false><<<(n + 255) / 256, 256, 0, st>>>(a);
    return cuda_status(cudaGetLastError(), "step");
}

sph_status launch_pos_to64(sph_ctx *ctx, cudaStream_t st) {
    if (ctx->n > 0 && ctx->pos64) k_pos_to64<<<(ctx->n + 255) / 256, 256, 0, st>>>(ctx->n, ctx->pos4, ctx->pos64);
    return cuda_status(cudaGetLastError(), "positions to FP64");
}

// ctx->diag: [kDiagBlocks * kDiag] partials, then kDiag totals
sph_status launch_diag_sums(sph_ctx *ctx, cudaStream_t st) {
    double *tot = ctx->diag + (size_t)kDiagBlocks * kDiag;
    k_diag_block<<<kDiagBlocks, kDiagThreads, 0, st>>>(ctx->n, ctx->pos4,
                                                       ctx->form.precision == SPH_PRECISION_MIXED ? ctx->pos64 : nullptr,
                                                       ctx->vel4, ctx->u, ctx->phi, ctx->diag);
    k_diag_total<<<1, 32, 0, st>>>(kDiagBlocks, ctx->diag, tot);
    return cuda_status(cudaGetLastError(), "diagnostics");
}

sph_status launch_snapshot(sph_ctx *ctx, cudaStream_t st) {
    const int n = ctx->n;
    cudaMemsetAsync(ctx->snapshot, 0, sizeof(int32_t) * kSnapshotRes * kSnapshotRes, st);
    if (n > 0) k_snapshot<<<(n + 255) / 256, 256, 0, st>>>(n, ctx->pos4, ctx->mat, ctx->snapshot);
    return cuda_status(cudaGetLastError(), "snapshot");
}

}  // namespace sph
