// sph_gravity_theta.cu -- the opening-angle gravity form and the FP64 direct
// sum it is measured against.  Neither has a counterpart in the reference,
// whose gravity (Compute.cpp:328-377, sph_gravity.cu here) uses an adaptive
// acceptance test without an opening angle, force-accepts failing leaves and
// keeps integer-truncated softening coefficients (kernels.h:93,97).
//
// Tree: the GPU Morton octree (sph_tree.cu), whose leaves hold contiguous
// runs of the particles in key order.  Up pass (sph_up.cuh, one launch): per
// node the mass, centre of mass, the second moments Q_jk = sum m r_j r_k about
// the centre of mass, and the radius of the smallest sphere about the centre
// of mass that holds the node's box.
//
// Evaluation is a group walk: a warp takes 32 consecutive particles in key
// order (a compact group) and traverses the tree from the root, 32 nodes at a
// time from a queue.  A node is accepted for the whole group when
//     r_node < theta * d   and   d > 2 eps,
// d being the distance from its centre of mass to the group's bounding box
// (so every particle of the group sees it under an angle below theta and
// outside the softening support); accepted nodes are evaluated at each
// particle (M2P: monopole + quadrupole, potential and acceleration), rejected
// leaves are summed particle by particle (P2P with the cubic-spline softened
// kernel and its exact coefficients), rejected branches put their children on
// the queue.  Accepted nodes and rejected leaves are staged in shared memory
// and evaluated in batches with every lane busy; each batch's partial sums
// are added into Kahan-compensated per-particle accumulators.  The walk
// writes acc = G a, |a| (the reference's gravNorm) and the potential G phi.
#include <cuda_runtime.h>

#include "sph_f32x2.cuh"
#include "sph_internal.h"
#include "sph_up.cuh"

namespace sph {

namespace {

// Layout of a theta-form node record (kPoleQ float4 per node):
//   q0 (com.xyz, radius)  q1 (M, Qxx, Qxy, Qxz)  q2 (Qyy, Qyz, Qzz, 0)
//   q3 (bbox min, 0)      q4 (bbox max, 1)

__device__ __forceinline__ float corner_radius(float cx, float cy, float cz, float mnx, float mny, float mnz,
                                               float mxx, float mxy, float mxz) {
    const float dx = fmaxf(cx - mnx, mxx - cx), dy = fmaxf(cy - mny, mxy - cy), dz = fmaxf(cz - mnz, mxz - cz);
    return sqrtf(dx * dx + dy * dy + dz * dz);
}

struct ThetaUpArgs {
    const int32_t *T;
    const int32_t *list_slot;
    int32_t *parent_slot;
    float4 *poles;
    const float4 *pos4;
    uint8_t *active;
    const int32_t *nat;
    const int32_t *globals;
    int individual;  // SPH_TIMESTEP_INDIVIDUAL: activity from the next active times, synced per leaf
};

__device__ void p2m_theta(const ThetaUpArgs &a, int tp, int dp) {
    const int32_t *T = a.T;
    const int np = T[tp];
    const int s = tp + 2;
    // sums relative to the first particle: no cancellation at large |x|
    const float4 x0 = a.pos4[T[s]];
    float m = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
    float mnx = x0.x, mny = x0.y, mnz = x0.z, mxx = x0.x, mxy = x0.y, mxz = x0.z;
    // individual timesteps: the leaf is active when one of its particles is
    // due, and then all of them are (README.md:62-64); otherwise all are
    bool act = true;
    if (a.individual) {
        const int gt = a.globals[0];
        act = false;
        for (int i = 0; i < np && !act; ++i) act = gt >= a.nat[T[s + i]];
    }
    for (int i = 0; i < np; ++i) a.active[T[s + i]] = act ? 1 : 0;
    // (loads only, so that several particles' loads are in flight together)
#pragma unroll 4
    for (int i = 0; i < np; ++i) {
        const float4 q = a.pos4[T[s + i]];
        m += q.w;
        sx += q.w * (q.x - x0.x);
        sy += q.w * (q.y - x0.y);
        sz += q.w * (q.z - x0.z);
        mnx = fminf(mnx, q.x);
        mny = fminf(mny, q.y);
        mnz = fminf(mnz, q.z);
        mxx = fmaxf(mxx, q.x);
        mxy = fmaxf(mxy, q.y);
        mxz = fmaxf(mxz, q.z);
    }
    const float ox = sx / m, oy = sy / m, oz = sz / m;  // com - x0
    float qxx = 0.f, qxy = 0.f, qxz = 0.f, qyy = 0.f, qyz = 0.f, qzz = 0.f;
#pragma unroll 4
    for (int i = 0; i < np; ++i) {
        const float4 q = a.pos4[T[s + i]];
        const float rx = (q.x - x0.x) - ox, ry = (q.y - x0.y) - oy, rz = (q.z - x0.z) - oz;
        qxx += q.w * rx * rx;
        qxy += q.w * rx * ry;
        qxz += q.w * rx * rz;
        qyy += q.w * ry * ry;
        qyz += q.w * ry * rz;
        qzz += q.w * rz * rz;
    }
    const float cx = x0.x + ox, cy = x0.y + oy, cz = x0.z + oz;
    float4 *pr = a.poles + (size_t)dp * kPoleQ;
    pr[0] = make_float4(cx, cy, cz, corner_radius(cx, cy, cz, mnx, mny, mnz, mxx, mxy, mxz));
    pr[1] = make_float4(m, qxx, qxy, qxz);
    pr[2] = make_float4(qyy, qyz, qzz, 0.f);
    pr[3] = make_float4(mnx, mny, mnz, 0.f);
    pr[4] = make_float4(mxx, mxy, mxz, act ? 1.f : 0.f);
    pr[5] = make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ void m2m_theta(const ThetaUpArgs &a, int tp, int dp) {
    const int32_t *T = a.T;
    const int my_slot = a.list_slot[dp];
    int first = -1;
    float4 c0f = make_float4(0.f, 0.f, 0.f, 0.f);
    float m = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
    float mnx = 3.402823466e+38f, mny = mnx, mnz = mnx, mxx = -mnx, mxy = -mnx, mxz = -mnx;
    // all slots' loads at once (an empty slot reads the node's own record): a
    // branch waits for memory three times and not once per child
    int child[8], child_dp[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) child[k] = T[tp + 2 + k];
#pragma unroll
    for (int k = 0; k < 8; ++k) child_dp[k] = child[k] != -1 ? T[child[k] + 1] : dp;
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (child[k] != -1) a.parent_slot[child_dp[k]] = my_slot;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float4 *cp = a.poles + (size_t)child_dp[k] * kPoleQ;
        const float4 q0 = cp[0], q1 = cp[1], q3 = cp[3], q4 = cp[4];
        if (child[k] == -1) continue;
        if (first < 0) {
            first = k;
            c0f = q0;
        }
        m += q1.x;
        sx += q1.x * (q0.x - c0f.x);
        sy += q1.x * (q0.y - c0f.y);
        sz += q1.x * (q0.z - c0f.z);
        mnx = fminf(mnx, q3.x);
        mny = fminf(mny, q3.y);
        mnz = fminf(mnz, q3.z);
        mxx = fmaxf(mxx, q4.x);
        mxy = fmaxf(mxy, q4.y);
        mxz = fmaxf(mxz, q4.z);
    }
    const float ox = sx / m, oy = sy / m, oz = sz / m;
    float qxx = 0.f, qxy = 0.f, qxz = 0.f, qyy = 0.f, qyz = 0.f, qzz = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float4 *cp = a.poles + (size_t)child_dp[k] * kPoleQ;
        const float4 q0 = cp[0], q1 = cp[1], q2 = cp[2];
        if (child[k] == -1) continue;
        const float rx = (q0.x - c0f.x) - ox, ry = (q0.y - c0f.y) - oy, rz = (q0.z - c0f.z) - oz;
        const float mc = q1.x;
        qxx += q1.y + mc * rx * rx;
        qxy += q1.z + mc * rx * ry;
        qxz += q1.w + mc * rx * rz;
        qyy += q2.x + mc * ry * ry;
        qyz += q2.y + mc * ry * rz;
        qzz += q2.z + mc * rz * rz;
    }
    // individual timesteps: a branch is active when a child is; a branch
    // whose children are all leaves activates every leaf and particle under
    // it when one leaf is active (README.md:64)
    bool act = true;
    if (a.individual) {
        act = false;
        bool all_leaves = true;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c = child[k];
            if (c == -1) continue;
            if (a.poles[(size_t)child_dp[k] * kPoleQ + 4].w != 0.f) act = true;
            if (T[c] == 0) all_leaves = false;
        }
        if (act && all_leaves) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c = child[k];
                if (c == -1) continue;
                a.poles[(size_t)child_dp[k] * kPoleQ + 4].w = 1.f;
                for (int j = 0; j < T[c]; ++j) a.active[T[c + 2 + j]] = 1;
            }
        }
    }
    const float cx = c0f.x + ox, cy = c0f.y + oy, cz = c0f.z + oz;
    float4 *pr = a.poles + (size_t)dp * kPoleQ;
    pr[0] = make_float4(cx, cy, cz, corner_radius(cx, cy, cz, mnx, mny, mnz, mxx, mxy, mxz));
    pr[1] = make_float4(m, qxx, qxy, qxz);
    pr[2] = make_float4(qyy, qyz, qzz, 0.f);
    pr[3] = make_float4(mnx, mny, mnz, 0.f);
    pr[4] = make_float4(mxx, mxy, mxz, act ? 1.f : 0.f);
    pr[5] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// (the walk needs the GPU-built tree, so the up pass is always the climb)
__global__ void __launch_bounds__(128) k_up_theta(ThetaUpArgs a, UpNodes u) {
    up_climb(u, [&](int tp, int dp) { p2m_theta(a, tp, dp); }, [&](int tp, int dp) { m2m_theta(a, tp, dp); });
}

// Cubic-spline softened pair kernel with its exact coefficients (the
// reference's kernels.h:87-102 truncates them): force factor f(r) with
// a = -m f(r) R / r, and potential phi(r) (both -> Newtonian for r >= 2 eps).
__device__ __forceinline__ void soft_pair(float r, float &fr, float &pot) {
    const float h = kGravSoft;
    const float h1 = 1.f / h;
    const float q = r * h1;
    if (q >= 2.f) {
        const float r1 = 1.f / r;
        fr = r1 * r1;
        pot = -r1;
    } else if (q > 1.f) {
        const float q2 = q * q;
        fr = (h1 * h1) * ((8.f / 3.f) * q - 3.f * q2 + 1.2f * q2 * q - (1.f / 6.f) * q2 * q2 -
                          1.f / (15.f * q2));
        pot = h1 * ((4.f / 3.f) * q2 - q2 * q + 0.3f * q2 * q2 - (1.f / 30.f) * q2 * q2 * q - 1.6f +
                    1.f / (15.f * q));
    } else {
        const float q2 = q * q;
        fr = (h1 * h1) * ((4.f / 3.f) * q - 1.2f * q2 * q + 0.5f * q2 * q2);
        pot = h1 * ((2.f / 3.f) * q2 - 0.3f * q2 * q2 + 0.1f * q2 * q2 * q - 1.4f);
    }
}

__device__ __forceinline__ float warp_reduce_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_reduce_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ float warp_reduce_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void kahan_add(float &s, float &c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// ---- the group walk ----------------------------------------------------------
constexpr int kWalkWarps = 4;    // warps per block
constexpr int kCellCap = 64;     // accepted nodes staged per warp before evaluation
constexpr int kLeafCap = 64;     // rejected leaves staged per warp before evaluation
constexpr int kStackInts = 8192; // per warp, in global memory (depth-first: <= depth x 256 in use)

__global__ void k_gather_key_order(int n, const uint32_t *__restrict__ order, const float4 *__restrict__ pos4,
                                   float4 *__restrict__ kp4) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) kp4[i] = pos4[order[i]];
}

struct WalkArgs {
    const int32_t *T;
    const float4 *poles;
    const int2 *node_range;
    const float4 *kp4;        // positions and masses in key order
    const uint32_t *order;    // key order -> particle id
    int n, ngroups;
    float theta2;
    float4 *acc4;
    float *gnorm, *phi;
    int32_t *queues;
    uint32_t *counter;
    uint32_t *health;
    const uint8_t *active;  // individual timesteps: only active particles are walked for and written
};

// Staged nodes and particles lie in shared memory as pairs, component by
// component, so that a lane evaluates two of them per step in packed FP32
// arithmetic (sph_f32x2.cuh).  The walk was bound by issue slots (78 % of them
// busy, the FMA pipe 55 %).  A node's components: minus its centre of mass,
// M, and minus its traceless second moments 3 Q - tr Q (xx xy xz yy yz zz),
// whose sign lets every step below be a multiply-add; a particle's: minus its
// position, and m.  Each evaluation stands in the kernel once: two copies did
// not fit the instruction cache and took back what the packing gave.  Measured,
// gravity pass of a 1e6-particle Plummer sphere: 9.86 -> 7.08 ms.
constexpr int kCellVals = 10;
struct CellPair {
    float c[kCellVals][2];
};
struct PartPair {
    float c[4][2];
};

__device__ __forceinline__ F2 at2(const float (&c)[2]) { return F2{*reinterpret_cast<const uint64_t *>(c)}; }

__device__ __forceinline__ void stage_cell(CellPair *cells, int at, float4 com_r, float4 p1, float4 p2) {
    const float tr = p1.y + p2.x + p2.z;  // p1 = (M, Qxx, Qxy, Qxz), p2 = (Qyy, Qyz, Qzz, -)
    const float v[kCellVals] = {-com_r.x,        -com_r.y,    -com_r.z,    p1.x,        tr - 3.f * p1.y,
                                -3.f * p1.z,     -3.f * p1.w, tr - 3.f * p2.x, -3.f * p2.y, tr - 3.f * p2.z};
#pragma unroll
    for (int k = 0; k < kCellVals; ++k) cells[at >> 1].c[k][at & 1] = v[k];
}

// Acceleration (and potential) of the staged nodes at x, per unit G, added to
// s (with S = 3 Q - tr Q: potential -M / r - R.S.R / (2 r^5)).  An odd count's
// last pair is filled up with a massless copy of its node.
__device__ __forceinline__ void eval_cells(const CellPair *cell, int ncell, float4 x, float &sx, float &sy, float &sz,
                                           float &sp) {
    const F2 px = f2(x.x), py = f2(x.y), pz = f2(x.z);
    const F2 half = f2(-0.5f), five_halves = f2(-2.5f);
    F2 ax = f2(0.f), ay = ax, az = ax, ap = ax;  // minus the sums
    const int pairs = (ncell + 1) >> 1;
    for (int j = 0; j < pairs; ++j) {
        const CellPair &c = cell[j];
        const F2 Rx = px + at2(c.c[0]), Ry = py + at2(c.c[1]), Rz = pz + at2(c.c[2]);
        const F2 r2 = fma2(Rz, Rz, fma2(Ry, Ry, Rx * Rx));
        const F2 rinv = rsqrt2(r2);
        const F2 rinv2 = rinv * rinv;
        const F2 rinv3 = rinv * rinv2;
        const F2 rinv5 = rinv3 * rinv2;
        const F2 M = at2(c.c[3]);
        const F2 xx = at2(c.c[4]), xy = at2(c.c[5]), xz = at2(c.c[6]);
        const F2 yy = at2(c.c[7]), yz = at2(c.c[8]), zz = at2(c.c[9]);
        const F2 SRx = fma2(xz, Rz, fma2(xy, Ry, xx * Rx));  // minus S R
        const F2 SRy = fma2(yz, Rz, fma2(yy, Ry, xy * Rx));
        const F2 SRz = fma2(zz, Rz, fma2(yz, Ry, xz * Rx));
        const F2 q5 = fma2(Rz, SRz, fma2(Ry, SRy, Rx * SRx)) * rinv5;
        ap = fma2(half, q5, fma2(M, rinv, ap));
        const F2 radial = fma2(five_halves * q5, rinv2, M * rinv3);
        ax = fma2(rinv5, SRx, fma2(radial, Rx, ax));
        ay = fma2(rinv5, SRy, fma2(radial, Ry, ay));
        az = fma2(rinv5, SRz, fma2(radial, Rz, az));
    }
    sx -= sum(ax);
    sy -= sum(ay);
    sz -= sum(az);
    sp -= sum(ap);
}

// Force factor s (acceleration s R) and potential of one pair at any r, for
// the pairs that reach into the softening: few, so out of line, where they do
// not crowd the instruction cache of the far pairs.
__device__ __noinline__ float2 near_pair(float r2, float m) {
    if (!(r2 > 0.f)) return make_float2(0.f, 0.f);
    const float r = sqrtf(r2);
    float fr, pot;
    soft_pair(r, fr, pot);
    return make_float2(-m * fr / r, m * pot);
}

// Softened pair sums of the staged particles at x, per unit G, added to s
// (an odd count's last pair is filled up with a massless copy).
__device__ __forceinline__ void eval_parts(const PartPair *part, int np, float4 x, float &sx, float &sy, float &sz,
                                           float &sp) {
    const float soft2x4 = 4.f * kGravSoft * kGravSoft;
    const F2 px = f2(x.x), py = f2(x.y), pz = f2(x.z);
    F2 ax = f2(0.f), ay = ax, az = ax, ap = ax;  // minus the sums of the pairs outside the softening
    const int pairs = (np + 1) >> 1;
#pragma unroll 2
    for (int j = 0; j < pairs; ++j) {
        const PartPair &q = part[j];
        const F2 rx = px + at2(q.c[0]), ry = py + at2(q.c[1]), rz = pz + at2(q.c[2]);
        const F2 r2 = fma2(rz, rz, fma2(ry, ry, rx * rx));
        float r2a, r2b;
        unpack(r2, r2a, r2b);
        if (fminf(r2a, r2b) >= soft2x4) {
            const F2 rinv = f2(rsqrt_hw(r2a), rsqrt_hw(r2b));
            const F2 mr = at2(q.c[3]) * rinv;
            const F2 s = mr * rinv * rinv;
            ax = fma2(s, rx, ax);
            ay = fma2(s, ry, ay);
            az = fma2(s, rz, az);
            ap = ap + mr;
        } else {
            float xa, xb, ya, yb, za, zb;
            unpack(rx, xa, xb);
            unpack(ry, ya, yb);
            unpack(rz, za, zb);
            const float2 a = near_pair(r2a, q.c[3][0]), b = near_pair(r2b, q.c[3][1]);
            sx += a.x * xa + b.x * xb;
            sy += a.x * ya + b.x * yb;
            sz += a.x * za + b.x * zb;
            sp += a.y + b.y;
        }
    }
    sx -= sum(ax);
    sy -= sum(ay);
    sz -= sum(az);
    sp -= sum(ap);
}

// (6 blocks per SM: with the registers of 8 the sums spill, 7.48 instead of
// 7.08 ms at the size above)
template <bool ACC>
__global__ void __launch_bounds__(32 * kWalkWarps, 6) k_walk(WalkArgs a) {
    __shared__ __align__(16) CellPair s_cell[kWalkWarps][kCellCap / 2];
    __shared__ int2 s_leaf[kWalkWarps][kLeafCap];
    __shared__ int s_loff[kWalkWarps][kLeafCap];
    __shared__ __align__(16) PartPair s_part[kWalkWarps][16];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned full = 0xffffffffu;
    const unsigned lt = (1u << lane) - 1u;
    int32_t *stk = a.queues + (size_t)(blockIdx.x * kWalkWarps + w) * kStackInts;
    const int32_t *T = a.T;
    const float soft2x4 = 4.f * kGravSoft * kGravSoft;
    while (true) {
        int g = 0;
        if (lane == 0) g = (int)atomicAdd(a.counter, 1u);
        g = __shfl_sync(full, g, 0);
        if (g >= a.ngroups) break;
        const int i = g * 32 + lane;
        const bool valid = i < a.n;
        // individual timesteps: only active particles get gravity, and a
        // group without one is skipped (the down-pass culling of README.md:64)
        const bool act = valid && (!a.active || a.active[a.order[i]]);
        if (!__any_sync(full, act)) continue;
        const float4 xi = a.kp4[valid ? i : g * 32];
        float ax = 0.f, ay = 0.f, az = 0.f, ph = 0.f, cax = 0.f, cay = 0.f, caz = 0.f, cph = 0.f;
        int ncell = 0, nleaf = 0;
        // the box the walk tests nodes against, and whether this lane's
        // particle belongs to the particles being walked for
        float bx0, by0, bz0, bx1, by1, bz1;
        bool mine = true;
        auto flush_cells = [&]() {
            __syncwarp();
            if ((ncell & 1) && lane < kCellVals)
                s_cell[w][ncell >> 1].c[lane][1] = lane < 3 ? s_cell[w][ncell >> 1].c[lane][0] : 0.f;
            __syncwarp();
            float sx = 0.f, sy = 0.f, sz = 0.f, sp = 0.f;
            eval_cells(s_cell[w], ncell, xi, sx, sy, sz, sp);
            if (mine) {
                kahan_add(ax, cax, sx);
                kahan_add(ay, cay, sy);
                kahan_add(az, caz, sz);
                kahan_add(ph, cph, sp);
            }
            ncell = 0;
            __syncwarp();
        };
        auto flush_leaves = [&]() {
            __syncwarp();
            // number the staged leaves' particles consecutively
            const int c0 = (lane < nleaf) ? s_leaf[w][lane].y : 0;
            const int c1 = (lane + 32 < nleaf) ? s_leaf[w][lane + 32].y : 0;
            int inc0 = c0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(full, inc0, o);
                if (lane >= o) inc0 += y;
            }
            const int tot0 = __shfl_sync(full, inc0, 31);
            int inc1 = c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(full, inc1, o);
                if (lane >= o) inc1 += y;
            }
            const int tot = tot0 + __shfl_sync(full, inc1, 31);
            if (lane < nleaf) s_loff[w][lane] = inc0 - c0;
            if (lane + 32 < nleaf) s_loff[w][lane + 32] = tot0 + inc1 - c1;
            __syncwarp();
            float sx = 0.f, sy = 0.f, sz = 0.f, sp = 0.f;
            for (int j0 = 0; j0 < tot; j0 += 32) {
                const int j = j0 + lane;
                if (j < tot) {
                    int q = 0;  // the last leaf whose first particle number is <= j
#pragma unroll
                    for (int step = kLeafCap / 2; step > 0; step >>= 1)
                        if (q + step < nleaf && s_loff[w][q + step] <= j) q += step;
                    float4 p = a.kp4[s_leaf[w][q].x + (j - s_loff[w][q])];
                    // a position that is no number (a run that blew up) would make
                    // every target's sums none: left out here, once for 32 targets
                    if (!(fabsf(p.x + p.y + p.z) < 1e30f)) p = make_float4(1e18f, 1e18f, 1e18f, 0.f);
                    PartPair &to = s_part[w][lane >> 1];
                    to.c[0][lane & 1] = -p.x;
                    to.c[1][lane & 1] = -p.y;
                    to.c[2][lane & 1] = -p.z;
                    to.c[3][lane & 1] = p.w;
                    if (j == tot - 1 && !(lane & 1)) {
                        to.c[0][1] = -p.x;
                        to.c[1][1] = -p.y;
                        to.c[2][1] = -p.z;
                        to.c[3][1] = 0.f;
                    }
                }
                __syncwarp();
                eval_parts(s_part[w], min(32, tot - j0), xi, sx, sy, sz, sp);
                __syncwarp();
            }
            if (mine) {
                kahan_add(ax, cax, sx);
                kahan_add(ay, cay, sy);
                kahan_add(az, caz, sz);
                kahan_add(ph, cph, sp);
            }
            nleaf = 0;
        };
        auto walk = [&]() {
            // depth-first: each round pops up to 32 nodes off the top of the
            // stack and pushes the children of the rejected branches
            if (lane == 0) stk[0] = 0;  // the root
            __syncwarp();
            int size = 1;
            // (the evaluations stand here once: with a copy before the staging
            // and one after the loop, the warps' instruction fetches missed)
            for (;;) {
                const bool end = size == 0;
                if (ncell + 32 > kCellCap || (end && ncell > 0)) flush_cells();
                if (nleaf + 32 > kLeafCap || (end && nleaf > 0)) flush_leaves();
                if (end) break;
                const int take = min(size, 32);
                size -= take;
                const bool v = lane < take;
                const int tp = v ? stk[size + lane] : 0;
                __syncwarp();
                const int dp = T[tp + 1];
                const int cnt = T[tp];
                const float4 *pr = a.poles + (size_t)dp * kPoleQ;
                const float4 c0 = pr[0];
                const float dx = fmaxf(fmaxf(bx0 - c0.x, c0.x - bx1), 0.f);
                const float dy = fmaxf(fmaxf(by0 - c0.y, c0.y - by1), 0.f);
                const float dz = fmaxf(fmaxf(bz0 - c0.z, c0.z - bz1), 0.f);
                const float d2 = dx * dx + dy * dy + dz * dz;
                bool acc = v && c0.w * c0.w < a.theta2 * d2 && d2 > soft2x4;
                const bool rleaf = v && !acc && cnt != 0;
                bool rbr = v && !acc && cnt == 0;
                int nch = 0;
                if (rbr)
                    for (int c = 0; c < 8; ++c) nch += (T[tp + 2 + c] != -1) ? 1 : 0;
                int inc = nch;
    #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(full, inc, o);
                    if (lane >= o) inc += y;
                }
                const int tot = __shfl_sync(full, inc, 31);
                if (size + tot > kStackInts) {
                    // no room (deeper than the stack allows): the rejected branches
                    // are taken as accepted nodes, flagged in the health word
                    if (lane == 0) raise_health(a.health, SPH_HEALTH_LIST_CAPACITY);
                    acc = acc || rbr;
                    rbr = false;
                } else {
                    if (rbr) {
                        // reversed, so that the first child is popped first
                        int o = size + inc - 1;
                        for (int c = 0; c < 8; ++c) {
                            const int ch = T[tp + 2 + c];
                            if (ch != -1) stk[o--] = ch;
                        }
                    }
                    size += tot;
                }
                // accepted nodes: stage their records
                const unsigned ma = __ballot_sync(full, acc);
                if (acc) {
                    const int o = ncell + __popc(ma & lt);
                    stage_cell(s_cell[w], o, c0, pr[1], pr[2]);
                }
                ncell += __popc(ma);
                // rejected leaves: stage their particle ranges
                const unsigned ml = __ballot_sync(full, rleaf);
                if (rleaf) s_leaf[w][nleaf + __popc(ml & lt)] = a.node_range[dp];
                nleaf += __popc(ml);
                __syncwarp();
            }
        };
        // A group that straddles a jump of the key order (two distant clusters
        // of particles) is cut there: consecutive particles farther apart
        // than 6x the group's typical step (the mean of the steps no longer
        // than twice the mean step) start a new segment, and every segment is
        // walked against its own box.  Almost every group is one segment.
        {
            const float4 xn = make_float4(__shfl_down_sync(full, xi.x, 1), __shfl_down_sync(full, xi.y, 1),
                                          __shfl_down_sync(full, xi.z, 1), 0.f);
            const bool has_next = lane < 31;
            const float ddx = xn.x - xi.x, ddy = xn.y - xi.y, ddz = xn.z - xi.z;
            const float step = has_next ? sqrtf(ddx * ddx + ddy * ddy + ddz * ddz) : 0.f;
            const float mean1 = warp_reduce_sum(step) * (1.f / 31.f);
            const bool small = has_next && step <= 2.f * mean1;
            const float n2 = warp_reduce_sum(small ? 1.f : 0.f);
            const float mean2 = warp_reduce_sum(small ? step : 0.f) / fmaxf(n2, 1.f);
            const bool cut = has_next && step > 6.f * mean2 && step > 0.f;
            // segment of this lane = number of cuts before it
            const unsigned cuts = __ballot_sync(full, cut);
            const int seg = __popc(cuts & lt);
            const int nseg = __popc(cuts) + 1;
            for (int q = 0; q < nseg; ++q) {
                mine = seg == q;
                const float big = 3.402823466e+38f;
                bx0 = warp_reduce_min(mine ? xi.x : big);
                by0 = warp_reduce_min(mine ? xi.y : big);
                bz0 = warp_reduce_min(mine ? xi.z : big);
                bx1 = warp_reduce_max(mine ? xi.x : -big);
                by1 = warp_reduce_max(mine ? xi.y : -big);
                bz1 = warp_reduce_max(mine ? xi.z : -big);
                walk();
            }
        }
        if (act) {
            const uint32_t id = a.order[i];
            if (ACC) {
                const float4 old = a.acc4[id];
                a.acc4[id] = make_float4(kG * ax, kG * ay, kG * az, old.w);
                a.gnorm[id] = sqrtf(ax * ax + ay * ay + az * az);
            }
            a.phi[id] = kG * ph;
        }
        __syncwarp();
    }
}
// FP64 direct sum over all particles at the given targets, with the exact
// softened kernel: out[4 t] = (ax, ay, az, phi) including G.  One block per
// target; positions are the float32 working positions promoted to double.
__global__ void __launch_bounds__(256) k_direct_f64(const float4 *__restrict__ pos4, int n,
                                                    const int32_t *__restrict__ targets, int nt,
                                                    double *__restrict__ out) {
    __shared__ double red[4][8];
    const int t = blockIdx.x;
    if (t >= nt) return;
    const int ip = targets[t];
    const float4 xi = pos4[ip];
    const double xx = xi.x, xy = xi.y, xz = xi.z;
    const double h = (double)kGravSoft, h1 = 1.0 / h;
    double ax = 0.0, ay = 0.0, az = 0.0, ph = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        if (j == ip) continue;
        const float4 xj = pos4[j];
        const double rx = xx - (double)xj.x, ry = xy - (double)xj.y, rz = xz - (double)xj.z;
        const double r2 = rx * rx + ry * ry + rz * rz;
        if (r2 == 0.0) continue;
        const double r = sqrt(r2);
        const double q = r * h1;
        double fr, pot;
        if (q >= 2.0) {
            fr = 1.0 / r2;
            pot = -1.0 / r;
        } else if (q > 1.0) {
            const double q2 = q * q;
            fr = h1 * h1 * ((8.0 / 3.0) * q - 3.0 * q2 + 1.2 * q2 * q - (1.0 / 6.0) * q2 * q2 - 1.0 / (15.0 * q2));
            pot = h1 * ((4.0 / 3.0) * q2 - q2 * q + 0.3 * q2 * q2 - (1.0 / 30.0) * q2 * q2 * q - 1.6 +
                        1.0 / (15.0 * q));
        } else {
            const double q2 = q * q;
            fr = h1 * h1 * ((4.0 / 3.0) * q - 1.2 * q2 * q + 0.5 * q2 * q2);
            pot = h1 * ((2.0 / 3.0) * q2 - 0.3 * q2 * q2 + 0.1 * q2 * q2 * q - 1.4);
        }
        const double m = (double)xj.w;
        const double s = -m * fr / r;
        ax += s * rx;
        ay += s * ry;
        az += s * rz;
        ph += m * pot;
    }
    double v[4] = {ax, ay, az, ph};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        double x = v[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = x;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
        out[4 * (size_t)t + threadIdx.x] = (double)kG * s;
    }
}

}  // namespace

static sph_status theta_pass(sph_ctx *ctx, float theta, bool acc, cudaStream_t st, cudaEvent_t up_done) {
    Tree &tr = ctx->tree;
    TreeBuild &tb = ctx->tb;
    if (!tr.valid || ctx->n <= 0) return SPH_OK;
    if (ctx->params.tree_source != SPH_TREE_GPU || !tb.order) {
        set_error("the theta gravity form walks the GPU-built tree (tree_source SPH_TREE_GPU)");
        return SPH_ERR_UNSUPPORTED;
    }
    const int n = ctx->n;
    ThetaUpArgs u;
    u.T = tr.tree;
    u.list_slot = tr.list_slot;
    u.parent_slot = tr.parent_slot;
    u.poles = tr.poles;
    u.pos4 = ctx->pos4;
    u.active = ctx->active;
    u.nat = ctx->nat;
    u.globals = ctx->globals;
    // activity follows the next active times only when the accelerations are
    // computed (the potential for the diagnostics covers every particle)
    u.individual = acc && ctx->form.timestep == SPH_TIMESTEP_INDIVIDUAL;
    k_up_theta<<<up_blocks(tr, 128), 128, 0, st>>>(u, up_nodes(tr));
    if (up_done) cudaEventRecord(up_done, st);
    // resident warps of the walk, each with its two node queues
    static int max_blocks_per_sm = 0;
    if (max_blocks_per_sm == 0) {
        int b0 = 0, b1 = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_walk<true>, 32 * kWalkWarps, 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_walk<false>, 32 * kWalkWarps, 0);
        max_blocks_per_sm = b0 < b1 ? b0 : b1;
        if (max_blocks_per_sm < 1) max_blocks_per_sm = 1;
    }
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    const int ngroups = (n + 31) / 32;
    int blocks = sms * max_blocks_per_sm;
    if (blocks * kWalkWarps > ngroups) blocks = (ngroups + kWalkWarps - 1) / kWalkWarps;
    const int64_t qints = (int64_t)blocks * kWalkWarps * kStackInts;
    if (qints > tb.walk_queue_ints) {
        cudaFree(tb.walk_queues);
        tb.walk_queues = nullptr;
        tb.walk_queue_ints = 0;
        cudaError_t e = cudaMalloc(&tb.walk_queues, sizeof(int32_t) * qints);
        if (e != cudaSuccess) return cuda_status(e, "gravity (theta) walk queues");
        tb.walk_queue_ints = qints;
    }
    if (!tb.walk_counter) {
        cudaError_t e = cudaMalloc(&tb.walk_counter, sizeof(uint32_t));
        if (e != cudaSuccess) return cuda_status(e, "gravity (theta) walk counter");
    }
    if (!tb.kp4) {
        cudaError_t e = cudaMalloc(&tb.kp4, sizeof(float4) * (size_t)n);
        if (e != cudaSuccess) return cuda_status(e, "gravity (theta) positions");
    }
    float4 *kp4 = tb.kp4;
    k_gather_key_order<<<(n + 255) / 256, 256, 0, st>>>(n, tb.order, ctx->pos4, kp4);
    cudaMemsetAsync(tb.walk_counter, 0, sizeof(uint32_t), st);
    WalkArgs w;
    w.T = tr.tree;
    w.poles = tr.poles;
    w.node_range = tr.node_range;
    w.kp4 = kp4;
    w.order = tb.order;
    w.n = n;
    w.ngroups = ngroups;
    w.theta2 = theta * theta;
    w.acc4 = ctx->acc4;
    w.gnorm = ctx->gnorm;
    w.phi = ctx->phi;
    w.queues = tb.walk_queues;
    w.counter = tb.walk_counter;
    w.health = ctx->health;
    w.active = u.individual ? ctx->active : nullptr;
    if (acc)
        k_walk<true><<<blocks, 32 * kWalkWarps, 0, st>>>(w);
    else
        k_walk<false><<<blocks, 32 * kWalkWarps, 0, st>>>(w);
    return cuda_status(cudaGetLastError(), "gravity (theta)");
}

sph_status launch_gravity_theta(sph_ctx *ctx, cudaStream_t st, cudaEvent_t up_done) {
    return theta_pass(ctx, ctx->form.theta, true, st, up_done);
}

sph_status launch_potential_theta(sph_ctx *ctx, float theta, cudaStream_t st) {
    return theta_pass(ctx, theta, false, st, nullptr);
}

sph_status launch_direct_f64(sph_ctx *ctx, const int32_t *d_targets, int nt, double *d_out, cudaStream_t st) {
    if (nt <= 0) return SPH_OK;
    k_direct_f64<<<nt, 256, 0, st>>>(ctx->pos4, ctx->n, d_targets, nt, d_out);
    return cuda_status(cudaGetLastError(), "direct f64");
}

}  // namespace sph
