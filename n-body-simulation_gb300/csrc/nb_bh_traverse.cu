// nb_bh_traverse.cu -- Barnes-Hut accelerations over the DFS-ordered octree
// (replaces BarnesHutAlgorithm::computeAccelerations, BarnesHutAlgorithm.cpp:280-401).
//
// Nodes are stored in the order the reference's stack pops them (DFS pre-order, children in
// visit order 2,0,3,1,6,4,7,5), each with a skip link to the first node after its subtree.
// "Accept" (or skip) continues at the skip link and "open" continues at the next node, so a
// traversal needs no stack at all and visits nodes in exactly the reference's order.
//
//  * per-body rule (NB_OPEN_THETA), default schedule (bh_theta_fix_kernel, NB_F64 with fixed-point
//    monopoles (nb_fix.cuh), and bh_theta_team_kernel, the same with several lanes per body for
//    small systems; bh_theta_lane_kernel, NB_F64_IEEE; bh_theta_df_kernel, double-float): each lane
//    walks its own body's DFS sequence, deciding each
//    cell with an FP32 pre-test whose rounding margin is proven and the reference's FP64
//    expression only inside that margin; find-then-compute, so the FP64 monopoles of all lanes
//    that found one run together. Warps take groups of 32 bodies close together in the tree, after
//    the first traversal of a tree sorted within windows of 512 by the length of their last
//    walk, so that the lanes of a warp finish together.
//  * per-body rule, lockstep schedule (bh_theta_f64_kernel, nb_bh_set_schedule(1)): the 32 lanes
//    of a warp hold 32 bodies adjacent in tree order, each with its own position in the DFS
//    sequence. Every iteration the warp takes the smallest position (__reduce_min_sync) and the
//    lanes sitting on it evaluate that node -- one broadcast load -- and advance by their own
//    decision.
//    Either way each body sees the reference's sequence of accepted nodes in the reference's
//    order.
//  * group rule (NB_OPEN_THETA_GROUP): the warp walks one sequence; a cell is opened when any
//    lane's rule opens it, otherwise all lanes accept it -- no divergence.
#include <algorithm>

#include "nb_bh.cuh"

namespace {

constexpr int TR_THREADS = 128;

enum Mode { IEEE64 = 0, FAST64 = 1, F32 = 2 };

template <int MODE>
struct Arith;

template <>
struct Arith<IEEE64> {
    __device__ static double sub(double a, double b) { return __dsub_rn(a, b); }
    __device__ static double norm2(double a, double b, double c) {
        return __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c));
    }
    __device__ static double rsqrt(double v) { return __ddiv_rn(1.0, __dsqrt_rn(v)); }
    __device__ static double mul(double a, double b) { return __dmul_rn(a, b); }
    __device__ static double add(double a, double b) { return __dadd_rn(a, b); }
    // acc += m * (d * inv), rounded as the reference writes it
    __device__ static double accum(double acc, double m, double d, double inv) {
        return __dadd_rn(acc, __dmul_rn(m, __dmul_rn(d, inv)));
    }
    __device__ static void monopole_xyz(double m, double dx, double dy, double dz, double eps2,
                                        double& ax, double& ay, double& az) {
        monopole(m, dx, dy, dz, norm2(dx, dy, dz), eps2, ax, ay, az);
    }
    // the reference's monopole: den = d2 + eps2, inv = 1/sqrt(den^3), acc += m * (d * inv)
    __device__ static void monopole(double m, double dx, double dy, double dz, double d2,
                                    double eps2, double& ax, double& ay, double& az) {
        double den = __dadd_rn(d2, eps2);
        den = __dmul_rn(__dmul_rn(den, den), den);
        const double inv = rsqrt(den);
        ax = accum(ax, m, dx, inv);
        ay = accum(ay, m, dy, inv);
        az = accum(az, m, dz, inv);
    }
};

template <>
struct Arith<FAST64> {
    __device__ static double sub(double a, double b) { return a - b; }
    __device__ static double norm2(double a, double b, double c) { return fma(a, a, fma(b, b, c * c)); }
    __device__ static double rsqrt(double v) { return nb_rsqrt_f64(v); }
    __device__ static double mul(double a, double b) { return a * b; }
    __device__ static double add(double a, double b) { return a + b; }
};

using nbfix::FixRec;

// 32-byte loads (one instruction of the load pipe instead of two). READ_ONLY: of memory that nothing
// writes while the kernel runs; otherwise (dependent launches) volatile, as the wait before them.
template <bool READ_ONLY = true>
__device__ __forceinline__ NodeRec32 load_rec32(const NodeRec32* p) {
    NodeRec32 r;
    if constexpr (READ_ONLY)
        asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(r.cx), "=f"(r.cy), "=f"(r.cz), "=f"(r.gm), "=f"(r.edge2), "=r"(r.skip),
              "=r"(r.body), "=r"(r.level)
            : "l"(p));
    else
        asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(r.cx), "=f"(r.cy), "=f"(r.cz), "=f"(r.gm), "=f"(r.edge2), "=r"(r.skip),
                       "=r"(r.body), "=r"(r.level)
                     : "l"(p)
                     : "memory");
    return r;
}
template <bool READ_ONLY = true>
__device__ __forceinline__ FixRec load_fix(const nbfix::FixHi* hi, const uint4* lo, uint32_t k) {
    FixRec r;
    if constexpr (READ_ONLY)
        asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=r"(r.x2), "=r"(r.y2), "=r"(r.z2), "=r"(r.mh), "=r"(r.x1), "=r"(r.y1), "=r"(r.z1),
              "=r"(r.e)
            : "l"(hi + k));
    else
        asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r.x2), "=r"(r.y2), "=r"(r.z2), "=r"(r.mh), "=r"(r.x1), "=r"(r.y1),
                       "=r"(r.z1), "=r"(r.e)
                     : "l"(hi + k)
                     : "memory");
    const uint4 l = lo[k];
    r.x0 = l.x;
    r.y0 = l.y;
    r.z0 = l.z;
    r.ml = l.w;
    return r;
}

// A body in the fixed point of the node records (nb_fix.cuh); sh_max < 0: FP64 pairs only.
struct FixBody {
    nbfix::Fix3 p;
    int sh_max;
};
template <int MODE>
__device__ __forceinline__ FixBody fix_body(double px, double py, double pz, int K,
                                            const nbfix::Eps2Table& e2) {
    FixBody b{};
    if constexpr (MODE == FAST64) b.sh_max = nbfix::split3(px, py, pz, K, b.p) ? e2.sh_max : -1;
    return b;
}

// Adds the monopole of node k to a body's sums: NB_F64's arithmetic, in every schedule.
__device__ __forceinline__ void fix_monopole(const FixRec& f, const NodeRec64* __restrict__ rec64,
                                             uint32_t k, const FixBody& b, int K,
                                             const nbfix::Eps2Table& e2,
                                             const double* __restrict__ x,
                                             const double* __restrict__ y,
                                             const double* __restrict__ z, uint32_t me,
                                             double eps2, double& acx, double& acy, double& acz) {
    double w, dx, dy, dz;
    if (b.sh_max < 0 || !nbfix::term(f, b.p, K, e2, b.sh_max, w, dx, dy, dz)) {
        const NodeRec64 q = rec64[k];
        if (q.mass == 0) return;
        dx = q.cx - x[me];
        dy = q.cy - y[me];
        dz = q.cz - z[me];
        w = nb_m_rinv3_f64(q.mass, fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
    }
    acx = fma(w, dx, acx);
    acy = fma(w, dy, acy);
    acz = fma(w, dz, acz);
}

// Per-body reference rule, FP64 (IEEE64 bit-identical to the host evaluation; FAST64: NB_F64's
// arithmetic, with the TEAM partial sums of the default schedule's lanes in turn).
template <int MODE, int TEAM>
__global__ void __launch_bounds__(TR_THREADS)
bh_theta_f64_kernel(const NodeRec64* __restrict__ rec, const nbfix::FixHi* __restrict__ fix_hi,
                    const uint4* __restrict__ fix_lo,
                    const uint32_t* __restrict__ info,
                    const uint32_t* __restrict__ ids, const double* __restrict__ x,
                    const double* __restrict__ y, const double* __restrict__ z,
                    const double* __restrict__ box, uint32_t n,
                    double theta, double eps2, double G, double* __restrict__ ax,
                    double* __restrict__ ay, double* __restrict__ az) {
    using A = Arith<MODE>;
    __shared__ nbfix::Eps2Table e2;
    const int K = (int)box[10];
    if (MODE == FAST64) {
        nbfix::fill_eps2(e2, eps2, K);
        __syncthreads();
    }
    const uint32_t p = blockIdx.x * TR_THREADS + threadIdx.x;
    const bool valid = p < n;
    const uint32_t nn = info[0];
    const uint32_t me = valid ? ids[p] : NB_NONE;
    double px = 0, py = 0, pz = 0;
    if (valid) {
        px = x[me];
        py = y[me];
        pz = z[me];
    }
    const FixBody me_fix = fix_body<MODE>(px, py, pz, K, e2);
    double acx[TEAM] = {}, acy[TEAM] = {}, acz[TEAM] = {};
    uint32_t ord = 0;
    uint32_t kl = valid ? 0u : nn;
    for (;;) {
        const uint32_t k = __reduce_min_sync(0xffffffffu, kl);
        if (k >= nn) break;
        if (kl != k) continue;
        const NodeRec64 r = rec[k];
        if (r.mass != 0 && r.body != me) {  // BarnesHutAlgorithm.cpp:349
            const double dx = A::sub(r.cx, px), dy = A::sub(r.cy, py), dz = A::sub(r.cz, pz);
            const double d2 = A::norm2(dx, dy, dz);
            const double cur = A::mul(r.edge, A::rsqrt(d2));  // :355-357
            if (cur < theta || r.body != NB_NONE) {           // :359
                if constexpr (MODE == FAST64) {
                    const uint32_t c = ord++ & (uint32_t)(TEAM - 1);
                    fix_monopole(load_fix(fix_hi, fix_lo, k), rec, k, me_fix, K, e2, x, y, z, me,
                                 eps2, acx[c], acy[c], acz[c]);
                } else {
                    A::monopole(r.mass, dx, dy, dz, d2, eps2, acx[0], acy[0], acz[0]);
                }
                kl = r.skip;
            } else {
                kl = k + 1;
            }
        } else {
            kl = r.skip;
        }
    }
#pragma unroll
    for (int o = TEAM / 2; o > 0; o >>= 1)
        for (int c = 0; c < o; ++c) {
            acx[c] += acx[c + o];
            acy[c] += acy[c + o];
            acz[c] += acz[c + o];
        }
    if (valid) {
        ax[me] = A::mul(acx[0], G);
        ay[me] = A::mul(acy[0], G);
        az[me] = A::mul(acz[0], G);
    }
}

// The part of the opening test's margin that no distance reduces: theta^2 * 4 (2^-24 E)^2.
__device__ __forceinline__ float margin_floor(float th2, float edge) {
    const float u = 2.0f * 5.9604645e-8f * edge;
    return th2 * (u * u);
}

// Per-body reference rule, FP64, each lane walking its own DFS sequence (no union walk).
// The opening test is decided in FP32 on the anchored FP32 records whenever the FP32 error
// bound proves the answer; only undecided cells evaluate the reference's FP64 expression.
// FP32 error bound of d^2 with positions rounded relative to the box centre (|c-a|, |p-a| <=
// E/2 per axis, u = 2^-24): |d2f - d2| <= u d^2 (2*sqrt(3) E/d + 5) + 3 u^2 E^2; the test below
// widens it by 4x (the last term to 4 u^2 E^2: it decides only where d2f is far below u^2 E^2, when
// one axis resolves less than the others) and adds the roundings of edge^2 and theta^2*d2f.
// Accumulation order per body is the reference's DFS order, so MODE IEEE64 stays bit-identical.
// Warps take groups of 32 sorted positions; with `order` != nullptr the bodies of the positions
// come from it (the previous walk's lengths regrouped within windows, regroup_kernel) instead of
// from ids. Each body's accepted-cell count goes to walk_len[body].
__global__ void __launch_bounds__(TR_THREADS)
bh_theta_lane_kernel(const NodeRec32* __restrict__ rec32, const NodeRec64* __restrict__ rec64,
                     const uint32_t* __restrict__ info, const uint32_t* __restrict__ ids,
                     const double* __restrict__ x, const double* __restrict__ y,
                     const double* __restrict__ z, const double* __restrict__ box, uint32_t n,
                     double theta, double eps2, double G, double* __restrict__ ax,
                     double* __restrict__ ay, double* __restrict__ az,
                     uint32_t* __restrict__ next_group, const uint32_t* __restrict__ order,
                     uint32_t* __restrict__ walk_len) {
    using A = Arith<IEEE64>;
    const uint32_t n_groups = (n + 31) / 32;
    const int lane = threadIdx.x & 31;
    // persistent warps: each takes the next 32 bodies until none are left, so no warp waits for
    // its block's slowest warp and the last wave's tail is one group long
    for (;;) {
        uint32_t grp = 0;
        if (lane == 0) grp = atomicAdd(next_group, 1u);
        grp = __shfl_sync(0xffffffffu, grp, 0);
        if (grp >= n_groups) break;
        const uint32_t p = grp * 32 + lane;
        const bool valid = p < n;  // lanes past the end stay (they take part in the warp votes)
        const uint32_t nn = info[0];
        const uint32_t me = valid ? (order != nullptr ? order[p] : ids[p]) : NB_NONE;
        uint32_t accepted = 0;
        const double px = valid ? x[me] : 0.0, py = valid ? y[me] : 0.0, pz = valid ? z[me] : 0.0;
        const double E = box[6];
        const double ox = box[0] + E / 2, oy = box[1] + E / 2, oz = box[2] + E / 2;
        const float pxf = (float)(px - ox), pyf = (float)(py - oy), pzf = (float)(pz - oz);
        const float th2 = (float)(theta * theta);
        const float u4 = 4.0f * 5.9604645e-8f;  // 4 * 2^-24
        const float Ef = (float)E, floor2 = margin_floor(th2, Ef);
        double acx = 0, acy = 0, acz = 0;
        uint32_t k = valid ? 0u : nn;
        // Find, then compute: every lane walks (FP32 tests, divergent but off the FP64 pipe) to its
        // next accepted cell, then the lanes evaluate their FP64 monopoles together, so the FP64
        // work runs with all unfinished lanes instead of the few that accept in the same iteration.
        for (;;) {
            bool found = false;
            uint32_t next = 0;
            while (k < nn) {
                const NodeRec32 r = rec32[k];
                if (r.body == me) {
                    k = r.skip;
                    continue;
                }
                bool accept = r.body != NB_NONE;
                if (!accept) {
                    const float dxf = r.cx - pxf, dyf = r.cy - pyf, dzf = r.cz - pzf;
                    const float d2f = fmaf(dxf, dxf, fmaf(dyf, dyf, dzf * dzf));
                    const float t = th2 * d2f;
                    const float rel = u4 * (3.5f * Ef * nb_rsqrt_f32(d2f) + 8.0f);
                    const float margin = fmaf(t, rel, fmaf(u4, r.edge2, floor2));
                    if (r.edge2 > t + margin) {
                        accept = false;  // certainly opened
                    } else if (r.edge2 < t - margin) {
                        accept = true;   // certainly accepted
                    } else {             // undecided: the reference's FP64 expression
                        const NodeRec64 q = rec64[k];
                        const double dx = A::sub(q.cx, px), dy = A::sub(q.cy, py),
                                     dz = A::sub(q.cz, pz);
                        accept = A::mul(q.edge, A::rsqrt(A::norm2(dx, dy, dz))) < theta;
                    }
                }
                if (accept) {
                    found = true;
                    next = r.skip;
                    break;
                }
                k = k + 1;
            }
            if (!__any_sync(0xffffffffu, found)) break;
            if (found) {
                ++accepted;
                const NodeRec64 q = rec64[k];
                if (q.mass != 0) {
                    const double dx = A::sub(q.cx, px), dy = A::sub(q.cy, py), dz = A::sub(q.cz, pz);
                    A::monopole_xyz(q.mass, dx, dy, dz, eps2, acx, acy, acz);
                }
                k = next;
            }
        }
        if (valid) {
            ax[me] = A::mul(acx, G);
            ay[me] = A::mul(acy, G);
            az[me] = A::mul(acz, G);
            walk_len[me] = accepted;
        }
    }
}

// Opening parameter as a kernel argument: its FP32 square stays in the constant bank.
struct Theta {
    double value;
    float sq;
    explicit Theta(double theta) : value(theta), sq((float)(theta * theta)) {}
};
struct Pretest {
    float px, py, pz, edge, floor2;  // body relative to the box centre, box edge, margin_floor
};
// Decision of the reference's opening rule for node `idx` seen from a body: true = accepted (a
// leaf, or certainly below theta), by the FP32 test where its margin allows (see
// bh_theta_lane_kernel), else by the FP64 expression.
__device__ __forceinline__ bool accepts(const NodeRec32& r, const Pretest& b,
                                        const NodeRec64* __restrict__ rec64, uint32_t idx,
                                        const double* __restrict__ x,
                                        const double* __restrict__ y,
                                        const double* __restrict__ z, uint32_t me, Theta theta) {
    using A = Arith<FAST64>;
    const float u4 = 4.0f * 5.9604645e-8f;  // 4 * 2^-24
    const float dx = r.cx - b.px, dy = r.cy - b.py, dz = r.cz - b.pz;
    const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float t = theta.sq * d2;
    const float rel = u4 * (3.5f * b.edge * nb_rsqrt_f32(d2) + 8.0f);
    const float margin = fmaf(t, rel, fmaf(u4, r.edge2, b.floor2));
    if (r.body != NB_NONE || r.edge2 < t - margin) return true;
    if (r.edge2 > t + margin) return false;
    const NodeRec64 q = rec64[idx];
    const double ex = A::sub(q.cx, x[me]), ey = A::sub(q.cy, y[me]), ez = A::sub(q.cz, z[me]);
    return A::mul(q.edge, A::rsqrt(A::norm2(ex, ey, ez))) < theta.value;
}

__device__ __forceinline__ Pretest pretest_of(const double* __restrict__ box, double px, double py,
                                              double pz, Theta theta) {
    const double E = box[6];
    return Pretest{(float)(px - (box[0] + E / 2)), (float)(py - (box[1] + E / 2)),
                   (float)(pz - (box[2] + E / 2)), (float)E, margin_floor(theta.sq, (float)E)};
}

// The next group of 32 bodies for a persistent warp, n_groups when none is left (one lane calls it).
// With the groups' costs from the last walks they are handed out in WALK_CLASSES passes over tree
// order, the costliest class first, so that the walks that start last are short ones: at 131,101
// bodies (Plummer; 1.1 groups per resident warp) a step takes 1.32 ms instead of 1.43, NB_DF64 at
// 262,144 2.77 instead of 2.91, 1,048,576 bodies 12.98 instead of 13.01; with 2 classes 1.40 and
// 2.92, with 4 1.33 and 2.80. The order does not change the results.
constexpr uint32_t WALK_CLASSES = 8;

__device__ __forceinline__ uint32_t next_walk(uint32_t* __restrict__ next_group, uint32_t n_groups,
                                              const uint32_t* __restrict__ cost,
                                              const unsigned long long* __restrict__ cost_sum) {
    if (cost == nullptr) return min(atomicAdd(next_group, 1u), n_groups);
    for (;;) {
        const uint32_t c = atomicAdd(next_group, 1u), pass = c / n_groups;
        if (pass >= WALK_CLASSES) return n_groups;
        const uint32_t g = c - pass * n_groups;
        // 8 cost / mean, its class: 11 and more, 10, ..., 5, less
        const unsigned long long q = 8ull * cost[g] * n_groups / max(*cost_sum, 1ull);
        if (11u - (uint32_t)min(max(q, 4ull), 11ull) == pass) return g;
    }
}

// Per-body reference rule, NB_F64: one lane per body. Each lane walks its body's DFS sequence and
// lists up to FIX_LIST accepted cells, then the warp evaluates its lanes' lists together, the next
// cell's record loaded while the current one is computed.
//  Bound: the load pipe (75% of its wavefronts: every lane reads its own 32-byte walk record per
//  visited and 48-byte fixed-point record per accepted cell) and issue (61% of cycles). The
//  monopole is ~137 instructions with 3 FP64 ones (nb_fix.cuh) against 16 FP64 operations before,
//  whose pipe was 82% busy; 256-bit loads halve the load instructions (14.6 -> 13.45 ms), the
//  lists (against one accepted cell at a time) keep 30.9 of 32 lanes active (17.2 -> 14.6 ms with
//  the record prefetch). Step at 1,048,576 bodies (disc, theta = 0.5): 35.5 -> 13.2 ms. 24 warps
//  per SM: 20 measured 4%, 28 2.5% and 32 4% slower; lists of 8 2% slower.
constexpr int FIX_LIST = 16;
constexpr int FIX_BLOCKS_PER_SM = 6;

__global__ void __launch_bounds__(TR_THREADS, FIX_BLOCKS_PER_SM)
bh_theta_fix_kernel(const NodeRec32* __restrict__ rec32, const NodeRec64* __restrict__ rec64,
                    const nbfix::FixHi* __restrict__ fix_hi, const uint4* __restrict__ fix_lo,
                    const uint32_t* __restrict__ info, const uint32_t* __restrict__ ids,
                    const double* __restrict__ x, const double* __restrict__ y,
                    const double* __restrict__ z, const double* __restrict__ box, uint32_t n,
                    Theta theta, double eps2, double G, double* __restrict__ ax,
                    double* __restrict__ ay, double* __restrict__ az,
                    uint32_t* __restrict__ next_group, const uint32_t* __restrict__ order,
                    uint32_t* __restrict__ walk_len, const uint32_t* __restrict__ cost,
                    const unsigned long long* __restrict__ cost_sum) {
    __shared__ nbfix::Eps2Table e2;
    __shared__ uint32_t list[FIX_LIST][TR_THREADS];
    const int K = (int)box[10];
    nbfix::fill_eps2(e2, eps2, K);
    __syncthreads();
    const uint32_t n_groups = (n + 31) / 32, nn = info[0];
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    for (;;) {  // persistent warps, as bh_theta_lane_kernel
        uint32_t grp = 0;
        if (lane == 0) grp = next_walk(next_group, n_groups, cost, cost_sum);
        grp = __shfl_sync(0xffffffffu, grp, 0);
        if (grp >= n_groups) break;
        const uint32_t p = grp * 32 + lane;
        const bool valid = p < n;
        const uint32_t me = valid ? (order != nullptr ? order[p] : ids[p]) : 0u;
        Pretest pre;
        FixBody body;
        {
            const double px = x[me], py = y[me], pz = z[me];
            pre = pretest_of(box, px, py, pz, theta);
            body = fix_body<FAST64>(px, py, pz, K, e2);
        }
        // bit 31 keeps the body's mark of rounded coordinates (a register less through the walk)
        uint32_t accepted = body.p.rounded << 31, k = valid ? 0u : nn;
        double acx = 0, acy = 0, acz = 0;
        for (;;) {
            int cnt = 0;
            while (cnt < FIX_LIST && k < nn) {
                const NodeRec32 r = load_rec32(rec32 + k);
                const bool accept = accepts(r, pre, rec64, k, x, y, z, me, theta);
                if (accept && r.body != me) {
                    list[cnt][tid] = k;
                    ++cnt;
                }
                k = accept ? r.skip : k + 1;
            }
            accepted += cnt;
            const int most = __reduce_max_sync(0xffffffffu, cnt);
            if (most == 0) break;
            FixRec next = load_fix(fix_hi, fix_lo, cnt > 0 ? list[0][tid] : 0u);
            for (int i = 0; i < most; ++i) {
                const FixRec f = next;
                body.p.rounded = accepted >> 31;
                if (i + 1 < cnt) next = load_fix(fix_hi, fix_lo, list[i + 1][tid]);
                if (i < cnt)
                    fix_monopole(f, rec64, list[i][tid], body, K, e2, x, y, z, me, eps2, acx, acy,
                                 acz);
            }
        }
        if (valid) {
            ax[me] = acx * G;
            ay[me] = acy * G;
            az[me] = acz * G;
            walk_len[me] = accepted & 0x7fffffffu;
        }
    }
}

// Per-body reference rule, NB_F64, T lanes per body, for systems too small to fill the chip with
// one lane per body. A body's lanes test T consecutive nodes of its DFS sequence at once (aligned
// windows: one coalesced load). Within a window a node is visited exactly when no accepted node
// before it covers it (an accepted node's subtree ends at its skip link, and whatever covers an
// unvisited node covers its subtree too), which a prefix maximum of the accepted nodes' skip links
// decides. The accepted cells go to the body's list in DFS order; cell number c belongs to lane
// c mod T, and the lanes' sums are added pairwise at the end.
//  Bound: the latency of a walk of dependent windows and of ~accepted / T monopoles by one warp.
//  Traversal at theta = 0.5 (disc), one lane per body -> T lanes: 777 bodies 135 -> 31 us (T = 32),
//  4,000 273 -> 77 us (16), 16,411 471 -> 300 us (4), 32,768 625 -> 540 us (2).
//  Registers for 20 warps per SM (24 warps: 3% slower at 16,411 bodies).
constexpr int TEAM_BLOCKS_PER_SM = 5;

template <int T>
__global__ void __launch_bounds__(TR_THREADS, TEAM_BLOCKS_PER_SM)
bh_theta_team_kernel(const NodeRec32* rec32, const NodeRec64* rec64,
                     const nbfix::FixHi* fix_hi, const uint4* fix_lo,
                     const uint32_t* info, const uint32_t* ids,
                     const double* x, const double* y,
                     const double* z, const double* box, uint32_t n,
                     Theta theta, double eps2, double G, double* __restrict__ ax,
                     double* __restrict__ ay, double* __restrict__ az,
                     uint32_t* __restrict__ walk_len) {
    nb_grid_wait();
    constexpr int B = 32 / T;                     // bodies per warp
    constexpr int CAP = T * 8 > 64 ? T * 8 : 64;  // listed cells per body and round
    constexpr int WARPS = TR_THREADS / 32;
    __shared__ nbfix::Eps2Table e2;
    __shared__ uint32_t lists[WARPS][B][CAP];
    const int K = (int)box[10];
    nbfix::fill_eps2(e2, eps2, K);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, seg = lane / T, j = lane % T;
    const uint32_t seg_mask = T == 32 ? 0xffffffffu : (1u << (T & 31)) - 1u;
    uint32_t* list = lists[warp][seg];
    const uint32_t p = (blockIdx.x * WARPS + warp) * B + seg, nn = info[0];
    const bool valid = p < n;
    const uint32_t me = valid ? ids[p] : 0u;
    Pretest pre;
    FixBody body;
    {
        const double px = x[me], py = y[me], pz = z[me];
        pre = pretest_of(box, px, py, pz, theta);
        body = fix_body<FAST64>(px, py, pz, K, e2);
    }
    double acx = 0, acy = 0, acz = 0;
    uint32_t k = valid ? 0u : nn;  // the same in a body's lanes, like cnt and ord
    int ord = 0;                   // cells accepted in earlier rounds
    for (;;) {
        int cnt = 0;
        for (;;) {
            const bool active = k < nn && cnt <= CAP - T;
            if (!__any_sync(0xffffffffu, active)) break;
            const uint32_t base = k & ~(uint32_t)(T - 1), idx = base + j;
            bool take = false;
            uint32_t end = 0;  // inclusive prefix maximum of the accepted nodes' skip links
            if (active && idx >= k && idx < nn) {
                const NodeRec32 r = load_rec32<false>(rec32 + idx);
                const bool accept = accepts(r, pre, rec64, idx, x, y, z, me, theta);
                take = accept && r.body != me;
                if (accept) end = r.skip;
            }
#pragma unroll
            for (int o = 1; o < T; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, end, o, T);
                if (j >= o) end = max(end, v);
            }
            uint32_t before = __shfl_up_sync(0xffffffffu, end, 1, T);
            if (j == 0) before = 0;
            take = take && before <= idx;
            const uint32_t taken = (__ballot_sync(0xffffffffu, take) >> (seg * T)) & seg_mask;
            if (take) list[cnt + __popc(taken & ((1u << j) - 1u))] = idx;
            end = __shfl_sync(0xffffffffu, end, T - 1, T);
            if (active) k = max(base + T, end);
            cnt += __popc(taken);
        }
        const int most = __reduce_max_sync(0xffffffffu, cnt);
        if (most == 0) break;
        __syncwarp();
        int i = (j - ord) & (T - 1);
        FixRec next = load_fix<false>(fix_hi, fix_lo, i < cnt ? list[i] : 0u);
        for (int c = 0; c < most; c += T, i += T) {
            const FixRec f = next;
            if (i + T < cnt) next = load_fix<false>(fix_hi, fix_lo, list[i + T]);
            if (i < cnt)
                fix_monopole(f, rec64, list[i], body, K, e2, x, y, z, me, eps2, acx, acy, acz);
        }
        ord += cnt;
        __syncwarp();
    }
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) {
        acx += __shfl_xor_sync(0xffffffffu, acx, o);
        acy += __shfl_xor_sync(0xffffffffu, acy, o);
        acz += __shfl_xor_sync(0xffffffffu, acz, o);
    }
    if (valid && j == 0) {
        ax[me] = acx * G;
        ay[me] = acy * G;
        az[me] = acz * G;
        walk_len[me] = ord;
    }
}

// Walk order of the next per-body traversal: within each window of RG_WINDOW sorted positions
// (bodies close together in the tree), the bodies by decreasing length of their last walk (ties
// by position), so that the 32 lanes of a warp walk sequences of similar length and fewer lanes
// sit idle while the FP64 monopoles of the others run (a warp instruction costs the FP64 pipe the
// same however few lanes are active). Bitonic sort of (length, position) keys in shared memory.
constexpr int RG_WINDOW = 512;

__global__ void __launch_bounds__(RG_WINDOW)
regroup_kernel(const uint32_t* __restrict__ ids, const uint32_t* __restrict__ walk_len, uint32_t n,
               uint32_t* __restrict__ order, uint32_t* __restrict__ cost,
               unsigned long long* __restrict__ cost_sum) {
    __shared__ unsigned long long key[RG_WINDOW];
    const uint32_t i = threadIdx.x, p = blockIdx.x * RG_WINDOW + i;
    // ascending keys: longest walk first, then position; positions past n sort last
    key[i] = p < n ? ((unsigned long long)(~walk_len[ids[p]]) << 32) | i : ~0ull;
    __syncthreads();
    for (uint32_t k = 2; k <= RG_WINDOW; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const uint32_t q = i ^ j;
            if (q > i) {
                const unsigned long long a = key[i], b = key[q];
                if (((i & k) == 0) == (a > b)) {
                    key[i] = b;
                    key[q] = a;
                }
            }
            __syncthreads();
        }
    }
    if (p < n) order[p] = ids[blockIdx.x * RG_WINDOW + (uint32_t)(key[i] & 0xffffffffu)];
    if (i < RG_WINDOW / 32) {  // the groups' costs: their longest walks, and the sum of all groups'
        const uint32_t first = blockIdx.x * RG_WINDOW + i * 32;
        const uint32_t c = first < n ? ~(uint32_t)(key[i * 32] >> 32) : 0u;
        if (first < n) cost[first / 32] = c;
        const uint32_t sum = __reduce_add_sync((1u << (RG_WINDOW / 32)) - 1u, c);
        if (i == 0) atomicAdd(cost_sum, (unsigned long long)sum);
    }
}

// Per-body reference rule with FP64-accurate double-float monopoles (NB_DF64, systems of one lane
// per body; smaller ones take bh_theta_team_kernel's fixed point, which is faster there and more
// accurate). The walk, the decisions and the lists are those of bh_theta_fix_kernel, so each body
// accepts exactly the reference's cells; the accepted monopoles are evaluated in double-float
// arithmetic on the FP32 pipe (~2^-48 relative per operation). Centres and the body are exact
// triple-floats relative to the box centre (rec32 and df_terms), so the separation is accurate to
// ~2^-48 of itself. rsqrt: hardware estimate y0 plus the third-order step
// y = y0 (1 + e/2 + 3e^2/8), e = 1 - r^2 y0^2 evaluated with error-free products. The sums are
// Neumaier-compensated (hi + running lo), converted to FP64 at the end and scaled by G / G_build.
//  Bound: the load pipe and issue, as bh_theta_fix_kernel. Lists, record prefetch and 256-bit loads
//  against one cell at a time inside the divergent walk: 262,144 bodies 3.18 -> 2.63 ms, 1,048,576
//  11.9 -> 11.0 ms (disc, theta = 0.5); 20 warps per SM (32: 3 to 12% slower). Same bits as before.
struct DfBody {
    float hx, hy, hz, mx, my, mz, lx, ly, lz;  // minus the box centre, exactly
    float e2h, e2l;                            // eps^2
    float ahx, ahy, ahz, alx, aly, alz;        // compensated sums
};

__device__ __forceinline__ void df_monopole(const float4 c, const DfTerms& t, DfBody& b) {
    if (c.w == 0.f && t.gl == 0.f) return;
    const nb_df dx = tf_diff(c.x, t.mx, t.lx, b.hx, b.mx, b.lx);
    const nb_df dy = tf_diff(c.y, t.my, t.ly, b.hy, b.my, b.ly);
    const nb_df dz = tf_diff(c.z, t.mz, t.lz, b.hz, b.mz, b.lz);
    // r^2 + eps^2
    const nb_df sx = df_sqr(dx), sy = df_sqr(dy), sz = df_sqr(dz);
    nb_df u = df_two_sum(sx.h, sy.h);
    u.l += sx.l + sy.l;
    nb_df v = df_two_sum(u.h, sz.h);
    v.l += u.l + sz.l;
    nb_df w2 = df_two_sum(v.h, b.e2h);  // eps^2 may be as large as r^2
    w2.l += v.l + b.e2l;
    const nb_df r2 = df_two_sum(w2.h, w2.l);
    // 1/r
    const float y0 = nb_rsqrt_f32(r2.h);
    const float q = y0 * y0, qe = fmaf(y0, y0, -q);  // y0^2 = q + qe exactly
    const float th = r2.h * q;
    float te = fmaf(r2.h, q, -th);
    te = fmaf(r2.h, qe, te);
    te = fmaf(r2.l, q, te);
    const float e = (1.0f - th) - te;  // 1 - th is exact (th is within 2^-21 of 1)
    const nb_df inv = df_fast_two_sum(y0, y0 * (e * fmaf(0.375f, e, 0.5f)));
    // G m / r^3
    const nb_df w = df_mul(nb_df{c.w, t.gl}, df_mul(df_sqr(inv), inv));
    // compensated sums
    const nb_df tx = df_mul(dx, w), ty = df_mul(dy, w), tz = df_mul(dz, w);
    nb_df s = df_two_sum(b.ahx, tx.h);
    b.ahx = s.h;
    b.alx += s.l + tx.l;
    s = df_two_sum(b.ahy, ty.h);
    b.ahy = s.h;
    b.aly += s.l + ty.l;
    s = df_two_sum(b.ahz, tz.h);
    b.ahz = s.h;
    b.alz += s.l + tz.l;
}

__device__ __forceinline__ DfTerms load_df(const DfTerms* __restrict__ p) {
    DfTerms t;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(t.mx), "=f"(t.my), "=f"(t.mz), "=f"(t.gl), "=f"(t.lx), "=f"(t.ly), "=f"(t.lz),
          "=f"(t.pad)
        : "l"(p));
    return t;
}

constexpr int DF_BLOCKS_PER_SM = 5;

__global__ void __launch_bounds__(TR_THREADS, DF_BLOCKS_PER_SM)
bh_theta_df_kernel(const NodeRec32* __restrict__ rec32, const DfTerms* __restrict__ df_terms,
                   const NodeRec64* __restrict__ rec64, const uint32_t* __restrict__ info,
                   const uint32_t* __restrict__ ids, const double* __restrict__ x,
                   const double* __restrict__ y, const double* __restrict__ z,
                   const double* __restrict__ box, uint32_t n, Theta theta, double eps2,
                   double gscale, double* __restrict__ ax, double* __restrict__ ay,
                   double* __restrict__ az, uint32_t* __restrict__ next_group,
                   const uint32_t* __restrict__ order, uint32_t* __restrict__ walk_len,
                   const uint32_t* __restrict__ cost,
                   const unsigned long long* __restrict__ cost_sum) {
    __shared__ uint32_t list[FIX_LIST][TR_THREADS];
    const uint32_t n_groups = (n + 31) / 32, nn = info[0];
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    for (;;) {  // persistent warps, as bh_theta_lane_kernel
        uint32_t grp = 0;
        if (lane == 0) grp = next_walk(next_group, n_groups, cost, cost_sum);
        grp = __shfl_sync(0xffffffffu, grp, 0);
        if (grp >= n_groups) break;
        const uint32_t p = grp * 32 + lane;
        const bool valid = p < n;
        const uint32_t me = valid ? (order != nullptr ? order[p] : ids[p]) : 0u;
        Pretest pre;
        DfBody b{};
        {
            const double px = x[me], py = y[me], pz = z[me], E = box[6];
            pre = pretest_of(box, px, py, pz, theta);
            tf_split_diff(px, box[0] + E / 2, b.hx, b.mx, b.lx);
            tf_split_diff(py, box[1] + E / 2, b.hy, b.my, b.ly);
            tf_split_diff(pz, box[2] + E / 2, b.hz, b.mz, b.lz);
            b.e2h = (float)eps2;
            b.e2l = (float)(eps2 - (double)b.e2h);
        }
        uint32_t accepted = 0, k = valid ? 0u : nn;
        for (;;) {
            int cnt = 0;
            while (cnt < FIX_LIST && k < nn) {
                const NodeRec32 r = load_rec32(rec32 + k);
                const bool accept = accepts(r, pre, rec64, k, x, y, z, me, theta);
                if (accept && r.body != me) {
                    list[cnt][tid] = k;
                    ++cnt;
                }
                k = accept ? r.skip : k + 1;
            }
            accepted += cnt;
            const int most = __reduce_max_sync(0xffffffffu, cnt);
            if (most == 0) break;
            uint32_t at = cnt > 0 ? list[0][tid] : 0u;
            float4 next_c = *reinterpret_cast<const float4*>(rec32 + at);
            DfTerms next_t = load_df(df_terms + at);
            for (int i = 0; i < most; ++i) {
                const float4 c = next_c;
                const DfTerms t = next_t;
                if (i + 1 < cnt) {
                    at = list[i + 1][tid];
                    next_c = *reinterpret_cast<const float4*>(rec32 + at);
                    next_t = load_df(df_terms + at);
                }
                if (i < cnt) df_monopole(c, t, b);
            }
        }
        if (valid) {
            walk_len[me] = accepted;
            ax[me] = ((double)b.ahx + (double)b.alx) * gscale;
            ay[me] = ((double)b.ahy + (double)b.aly) * gscale;
            az[me] = ((double)b.ahz + (double)b.alz) * gscale;
        }
    }
}

// Per-body reference rule with FP32 pair math and compensated accumulation.
__global__ void __launch_bounds__(TR_THREADS)
bh_theta_f32_kernel(const NodeRec32* __restrict__ rec, const uint32_t* __restrict__ info,
                    const uint32_t* __restrict__ ids, const double* __restrict__ x,
                    const double* __restrict__ y, const double* __restrict__ z,
                    const double* __restrict__ box, uint32_t n, float theta, float eps2,
                    double* __restrict__ ax, double* __restrict__ ay, double* __restrict__ az) {
    const uint32_t p = blockIdx.x * TR_THREADS + threadIdx.x;
    const bool valid = p < n;
    const uint32_t nn = info[0];
    const uint32_t me = valid ? ids[p] : NB_NONE;
    const double ox = box[0] + box[6] / 2, oy = box[1] + box[6] / 2, oz = box[2] + box[6] / 2;
    float px = 0, py = 0, pz = 0;
    if (valid) {
        px = (float)(x[me] - ox);
        py = (float)(y[me] - oy);
        pz = (float)(z[me] - oz);
    }
    float hx = 0, hy = 0, hz = 0, lx = 0, ly = 0, lz = 0;
    uint32_t kl = valid ? 0u : nn;
    const float theta2 = theta * theta;
    for (;;) {
        const uint32_t k = __reduce_min_sync(0xffffffffu, kl);
        if (k >= nn) break;
        if (kl != k) continue;
        const NodeRec32 r = rec[k];
        if (r.gm != 0 && r.body != me) {
            const float dx = r.cx - px, dy = r.cy - py, dz = r.cz - pz;
            const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (r.body != NB_NONE || r.edge2 < theta2 * d2) {
                const float inv = nb_rsqrt_f32(d2 + eps2);
                const float s = r.gm * inv * inv * inv;
                // TwoSum of each term into (h, l)
                const float tx = dx * s, ty = dy * s, tz = dz * s;
                float sh = hx + tx, bp = sh - hx;
                lx += (hx - (sh - bp)) + (tx - bp);
                hx = sh;
                sh = hy + ty;
                bp = sh - hy;
                ly += (hy - (sh - bp)) + (ty - bp);
                hy = sh;
                sh = hz + tz;
                bp = sh - hz;
                lz += (hz - (sh - bp)) + (tz - bp);
                hz = sh;
                kl = r.skip;
            } else {
                kl = k + 1;
            }
        } else {
            kl = r.skip;
        }
    }
    if (valid) {
        ax[me] = (double)hx + (double)lx;
        ay[me] = (double)hy + (double)ly;
        az[me] = (double)hz + (double)lz;
    }
}

// Group rule, FP64.
__global__ void __launch_bounds__(TR_THREADS)
bh_group_f64_kernel(const NodeRec64* __restrict__ rec, const uint32_t* __restrict__ info,
                    const uint32_t* __restrict__ ids, const double* __restrict__ x,
                    const double* __restrict__ y, const double* __restrict__ z, uint32_t n,
                    double theta, double eps2, double G, double* __restrict__ ax,
                    double* __restrict__ ay, double* __restrict__ az) {
    const uint32_t p = blockIdx.x * TR_THREADS + threadIdx.x;
    const bool valid = p < n;
    const uint32_t nn = info[0];
    const uint32_t me = valid ? ids[p] : NB_NONE;
    double px = 0, py = 0, pz = 0;
    if (valid) {
        px = x[me];
        py = y[me];
        pz = z[me];
    }
    const double theta2 = theta * theta;
    double acx = 0, acy = 0, acz = 0;
    uint32_t k = 0;
    while (k < nn) {
        const NodeRec64 r = rec[k];
        const double dx = r.cx - px, dy = r.cy - py, dz = r.cz - pz;
        const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
        const bool open = valid && r.body == NB_NONE && r.mass != 0 && r.edge * r.edge >= theta2 * d2;
        if (__any_sync(0xffffffffu, open)) {
            k = k + 1;
            continue;
        }
        if (valid && r.body != me && r.mass != 0) {
            const double s = nb_m_rinv3_f64(r.mass, d2 + eps2);
            acx = fma(s, dx, acx);
            acy = fma(s, dy, acy);
            acz = fma(s, dz, acz);
        }
        k = r.skip;
    }
    if (valid) {
        ax[me] = acx * G;
        ay[me] = acy * G;
        az[me] = acz * G;
    }
}

// Group rule, FP32 pair math; tile sums of 32 accepted cells folded into (hi, lo) by TwoSum.
__global__ void __launch_bounds__(TR_THREADS)
bh_group_f32_kernel(const NodeRec32* __restrict__ rec, const uint32_t* __restrict__ info,
                    const uint32_t* __restrict__ ids, const double* __restrict__ x,
                    const double* __restrict__ y, const double* __restrict__ z,
                    const double* __restrict__ box, uint32_t n, float theta, float eps2,
                    double* __restrict__ ax, double* __restrict__ ay, double* __restrict__ az) {
    const uint32_t p = blockIdx.x * TR_THREADS + threadIdx.x;
    const bool valid = p < n;
    const uint32_t nn = info[0];
    const uint32_t me = valid ? ids[p] : NB_NONE;
    const double ox = box[0] + box[6] / 2, oy = box[1] + box[6] / 2, oz = box[2] + box[6] / 2;
    float px = 0, py = 0, pz = 0;
    if (valid) {
        px = (float)(x[me] - ox);
        py = (float)(y[me] - oy);
        pz = (float)(z[me] - oz);
    }
    const float theta2 = theta * theta;
    float tx = 0, ty = 0, tz = 0, hx = 0, hy = 0, hz = 0, lx = 0, ly = 0, lz = 0;
    int batch = 0;
    uint32_t k = 0;
    while (k < nn) {
        const NodeRec32 r = rec[k];
        const float dx = r.cx - px, dy = r.cy - py, dz = r.cz - pz;
        const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const bool open = valid && r.body == NB_NONE && r.edge2 >= theta2 * d2;
        if (__any_sync(0xffffffffu, open)) {
            k = k + 1;
            continue;
        }
        if (valid && r.body != me) {
            const float inv = nb_rsqrt_f32(d2 + eps2);
            const float s = r.gm * inv * inv * inv;
            tx = fmaf(dx, s, tx);
            ty = fmaf(dy, s, ty);
            tz = fmaf(dz, s, tz);
        }
        if (++batch == 32) {
            batch = 0;
            float sh = hx + tx, bp = sh - hx;
            lx += (hx - (sh - bp)) + (tx - bp);
            hx = sh;
            sh = hy + ty;
            bp = sh - hy;
            ly += (hy - (sh - bp)) + (ty - bp);
            hy = sh;
            sh = hz + tz;
            bp = sh - hz;
            lz += (hz - (sh - bp)) + (tz - bp);
            hz = sh;
            tx = ty = tz = 0;
        }
        k = r.skip;
    }
    if (valid) {
        ax[me] = ((double)hx + (double)lx) + (double)tx;
        ay[me] = ((double)hy + (double)ly) + (double)ty;
        az[me] = ((double)hz + (double)lz) + (double)tz;
    }
}

// Work model: per body, the number of cells accepted (interactions) and opened under the
// per-body rule (FP64 decisions); totals accumulated into out[0] (accepted), out[1] (opened).
__global__ void __launch_bounds__(TR_THREADS)
bh_count_kernel(const NodeRec64* __restrict__ rec, const uint32_t* __restrict__ info,
                const uint32_t* __restrict__ ids, const double* __restrict__ x,
                const double* __restrict__ y, const double* __restrict__ z, uint32_t n,
                double theta, int group, unsigned long long* __restrict__ out) {
    const uint32_t p = blockIdx.x * TR_THREADS + threadIdx.x;
    const bool valid = p < n;
    const uint32_t nn = info[0];
    const uint32_t me = valid ? ids[p] : NB_NONE;
    double px = 0, py = 0, pz = 0;
    if (valid) {
        px = x[me];
        py = y[me];
        pz = z[me];
    }
    unsigned long long acc = 0, opened = 0;
    uint32_t kl = valid ? 0u : nn;
    const double theta2 = theta * theta;
    for (;;) {
        const uint32_t k = group ? (valid ? kl : nn) : kl;
        const uint32_t kk = group ? __reduce_min_sync(0xffffffffu, k) : __reduce_min_sync(0xffffffffu, kl);
        if (kk >= nn) break;
        const NodeRec64 r = rec[kk];
        const double dx = r.cx - px, dy = r.cy - py, dz = r.cz - pz;
        const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
        const bool wants_open = valid && r.mass != 0 && r.body == NB_NONE &&
                                r.edge * r.edge >= theta2 * d2;
        if (group) {
            if (__any_sync(0xffffffffu, wants_open)) {
                if (valid) opened += 1;
                kl = kk + 1;
            } else {
                if (valid && r.body != me && r.mass != 0) acc += 1;
                kl = r.skip;
            }
        } else if (kl == kk) {
            if (r.mass == 0 || r.body == me) {
                kl = r.skip;
            } else if (wants_open) {
                opened += 1;
                kl = kk + 1;
            } else {
                acc += 1;
                kl = r.skip;
            }
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        acc += __shfl_down_sync(0xffffffffu, acc, off);
        opened += __shfl_down_sync(0xffffffffu, opened, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&out[0], acc);
        atomicAdd(&out[1], opened);
    }
}

// Schedule of the per-body FP64 traversal: 0 = per-lane walks (default), 1 = the warp's union
// walk (bh_theta_f64_kernel). Both produce identical results; the switch exists for comparison.
int g_lockstep = 0;

// Resident blocks per SM of the persistent kernels (queried once, before any stream capture uses
// them): the IEEE lane kernel, the fixed-point and the double-float kernel.
int g_lane_per_sm[3] = {0, 0, 0};

nb_status lane_per_sm(nb_precision prec, int* out) {
    const int which = prec == NB_F64_IEEE ? 0 : (prec == NB_F64 ? 1 : 2);
    int& ps = g_lane_per_sm[which];
    if (ps == 0) {
        auto query = [&](auto kernel) {
            return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, kernel, TR_THREADS, 0);
        };
        NB_CUDA_TRY(which == 0 ? query(bh_theta_lane_kernel)
                               : (which == 1 ? query(bh_theta_fix_kernel)
                                             : query(bh_theta_df_kernel)));
        if (ps < 1) ps = 1;
    }
    *out = ps;
    return NB_OK;
}

// Lanes per body of the NB_F64 traversal: the largest power of two that keeps the launch within
// TEAM_LANES_PER_SM lanes per SM. Beyond one wave of resident warps (768 lanes per SM) every extra
// lane only adds walk work; measured on the 152-SM part the fastest T is 32 up to 2,000 bodies, 16
// at 4,000, 8 at 8,000, 4 at 16,411, 2 at 32,768 and 1 at 65,536 (disc theta 0.5 and 1.05,
// Plummer 0.7), next to which half or twice the T is 2 to 25% slower.
constexpr long long TEAM_LANES_PER_SM = 480;

int team_lanes(const nb_ctx* ctx, uint32_t n) {
    int t = 32;
    while (t > 1 && (long long)n * t > TEAM_LANES_PER_SM * ctx->sm_count) t >>= 1;
    return t;
}

unsigned long long* walk_sum(const nb_bh_tree* t) {  // zeroed with the group counter, work[1]
    return reinterpret_cast<unsigned long long*>(t->work + 4);
}

// The walk lengths of the last per-body traversal of the same bodies order this one's groups
// (*order = the regrouped bodies), else tree order (*order = nullptr). The results do not depend
// on the order: each body sums its own sequence.
nb_status walk_order(const nb_bh_tree* t, cudaStream_t s, const uint32_t** order) {
    *order = nullptr;
    if (t->walk_n != t->n) return NB_OK;
    regroup_kernel<<<nb::ceil_div(t->n, RG_WINDOW), RG_WINDOW, 0, s>>>(t->ids, t->walk_len, t->n,
                                                                       t->walk_ids, t->walk_cost,
                                                                       walk_sum(t));
    NB_TRY(nb::check_launch("regroup_kernel"));
    *order = t->walk_ids;
    return NB_OK;
}

// Persistent launch of bh_theta_lane_kernel: resident blocks only, groups from work[1], at most
// LANE_BLOCKS_PER_SM blocks per SM. With all 40 resident warps of an SM contending for its FP64
// pipe, the warps that lose the arbitration keep their first group for the whole launch and
// finish it alone at the end; 20 warps keep the pipe as busy with a shorter tail (1% faster at
// 1,048,576 bodies than 40, 0.2% faster than 24 or 16).
constexpr int LANE_BLOCKS_PER_SM = 5;

nb_status launch_lane(nb_ctx* ctx, const nb_bh_tree* t, nb_precision prec, const double* x,
                      const double* y, const double* z, double* ax, double* ay, double* az,
                      double G, double eps2, cudaStream_t s) {
    int ps = 0;
    NB_TRY(lane_per_sm(prec, &ps));
    if (prec == NB_F64_IEEE) ps = std::min(ps, LANE_BLOCKS_PER_SM);
    int grid = nb::ceil_div(t->n, TR_THREADS);
    if (grid > ctx->sm_count * ps) grid = ctx->sm_count * ps;
    NB_CUDA_TRY(cudaMemsetAsync(t->work + 1, 0, 5 * sizeof(uint32_t), s));
    const uint32_t* order = nullptr;
    NB_TRY(walk_order(t, s, &order));
    if (prec == NB_F64_IEEE)
        bh_theta_lane_kernel<<<grid, TR_THREADS, 0, s>>>(
            t->rec32, t->rec64, t->info, t->ids, x, y, z, t->box, t->n, t->params.theta, eps2, G,
            ax, ay, az, t->work + 1, order, t->walk_len);
    else if (prec == NB_F64)
        bh_theta_fix_kernel<<<grid, TR_THREADS, 0, s>>>(
            t->rec32, t->rec64, t->fix_hi, t->fix_lo, t->info, t->ids, x, y, z, t->box, t->n,
            Theta(t->params.theta), eps2, G, ax, ay, az, t->work + 1, order, t->walk_len,
            order ? t->walk_cost : nullptr, walk_sum(t));
    else
        bh_theta_df_kernel<<<grid, TR_THREADS, 0, s>>>(
            t->rec32, t->df_terms, t->rec64, t->info, t->ids, x, y, z, t->box, t->n,
            Theta(t->params.theta), eps2, G / t->G, ax, ay, az, t->work + 1, order, t->walk_len,
            order ? t->walk_cost : nullptr, walk_sum(t));
    NB_TRY(nb::check_launch("Barnes-Hut lane kernel"));
    t->walk_n = t->n;
    return NB_OK;
}

// NB_F64 and NB_DF64 under the per-body rule: teams of lanes for small systems (in tree order:
// neighbouring bodies share their windows' loads), one lane per body otherwise.
nb_status launch_f64(nb_ctx* ctx, const nb_bh_tree* t, nb_precision prec, const double* x,
                     const double* y, const double* z, double* ax, double* ay, double* az,
                     double G, double eps2, cudaStream_t s) {
    const int team = team_lanes(ctx, t->n);
    if (team == 1) return launch_lane(ctx, t, prec, x, y, z, ax, ay, az, G, eps2, s);
    const int grid = nb::ceil_div((long long)t->n * team, TR_THREADS);
    auto go = [&](auto kernel) {
        return nb::launch_after(kernel, grid, TR_THREADS, 0, s, t->rec32, t->rec64, t->fix_hi,
                                t->fix_lo, t->info, t->ids, x, y, z, t->box, t->n,
                                Theta(t->params.theta), eps2, G, ax, ay, az, t->walk_len);
    };
    switch (team) {
        case 2: NB_CUDA_TRY(go(bh_theta_team_kernel<2>)); break;
        case 4: NB_CUDA_TRY(go(bh_theta_team_kernel<4>)); break;
        case 8: NB_CUDA_TRY(go(bh_theta_team_kernel<8>)); break;
        case 16: NB_CUDA_TRY(go(bh_theta_team_kernel<16>)); break;
        default: NB_CUDA_TRY(go(bh_theta_team_kernel<32>)); break;
    }
    t->walk_n = t->n;
    return NB_OK;
}

// NB_F64 and NB_F64_IEEE in lockstep (nb_bh_set_schedule).
nb_status launch_lockstep(nb_ctx* ctx, const nb_bh_tree* t, nb_precision prec, const double* x,
                          const double* y, const double* z, double* ax, double* ay, double* az,
                          double G, double eps2, cudaStream_t s) {
    auto go = [&](auto kernel) {
        kernel<<<nb::ceil_div(t->n, TR_THREADS), TR_THREADS, 0, s>>>(
            t->rec64, t->fix_hi, t->fix_lo, t->info, t->ids, x, y, z, t->box, t->n, t->params.theta,
            eps2, G, ax, ay, az);
        return nb::check_launch("bh_theta_f64_kernel");
    };
    if (prec == NB_F64_IEEE) return go(bh_theta_f64_kernel<IEEE64, 1>);
    switch (team_lanes(ctx, t->n)) {
        case 1: return go(bh_theta_f64_kernel<FAST64, 1>);
        case 2: return go(bh_theta_f64_kernel<FAST64, 2>);
        case 4: return go(bh_theta_f64_kernel<FAST64, 4>);
        case 8: return go(bh_theta_f64_kernel<FAST64, 8>);
        case 16: return go(bh_theta_f64_kernel<FAST64, 16>);
        default: return go(bh_theta_f64_kernel<FAST64, 32>);
    }
}

}  // namespace

namespace nb {
nb_status launch_learned(nb_ctx* ctx, const nb_bh_tree* t, const double* x, const double* y,
                         const double* z, double* ax, double* ay, double* az, double eps2,
                         unsigned long long* counters, cudaStream_t s);
nb_status learned_per_sm(int* out);
}

extern "C" {

nb_status nb_bh_set_schedule(int lockstep) {
    g_lockstep = lockstep ? 1 : 0;
    return NB_OK;
}

nb_status nb_bh_accel(nb_ctx* ctx, const nb_bh_tree* t, const double* x, const double* y,
                      const double* z, double* ax, double* ay, double* az, double G, double eps2,
                      nb_opening opening, nb_precision prec, nb_stream_t stream_) {
    NB_CHECK_CTX(ctx);
    if (!t) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_accel: null tree");
    if (!t->built) return nb::set_error(NB_ERR_NOT_BUILT, "nb_bh_accel: tree not built");
    if (!x || !y || !z || !ax || !ay || !az)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_accel: null array");
    cudaStream_t s = (cudaStream_t)stream_;
    const uint32_t n = t->n;
    const int grid = nb::ceil_div(n, TR_THREADS);
    const double theta = t->params.theta;
    if (opening == NB_OPEN_THETA) {
        switch (prec) {
            case NB_F64_IEEE:
                NB_TRY(nb_need_records(t, NB_REC_FP64, "nb_bh_accel"));
                if (g_lockstep)
                    return launch_lockstep(ctx, t, prec, x, y, z, ax, ay, az, G, eps2, s);
                return launch_lane(ctx, t, prec, x, y, z, ax, ay, az, G, eps2, s);
            case NB_F64:
                NB_TRY(nb_need_records(t, NB_REC_FP64, "nb_bh_accel"));
                if (g_lockstep)
                    return launch_lockstep(ctx, t, prec, x, y, z, ax, ay, az, G, eps2, s);
                return launch_f64(ctx, t, prec, x, y, z, ax, ay, az, G, eps2, s);
            case NB_DF64:
                NB_TRY(nb_need_records(t, NB_REC_FP64 | NB_REC_DF, "nb_bh_accel"));
                if (t->G == 0)
                    return nb::set_error(NB_ERR_INVALID_ARG,
                                         "nb_bh_accel: NB_DF64 needs a build with G != 0");
                return launch_f64(ctx, t, prec, x, y, z, ax, ay, az, G, eps2, s);
            case NB_F32C:
                if (G != t->G)
                    return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_accel: G differs from the build's");
                bh_theta_f32_kernel<<<grid, TR_THREADS, 0, s>>>(t->rec32, t->info, t->ids, x, y, z,
                                                                t->box, n, (float)theta,
                                                                (float)eps2, ax, ay, az);
                return nb::check_launch("bh_theta_f32_kernel");
            default:
                break;
        }
    } else if (opening == NB_OPEN_THETA_GROUP) {
        switch (prec) {
            case NB_F64_IEEE:
            case NB_F64:
                NB_TRY(nb_need_records(t, NB_REC_FP64, "nb_bh_accel"));
                bh_group_f64_kernel<<<grid, TR_THREADS, 0, s>>>(t->rec64, t->info, t->ids, x, y, z,
                                                                n, theta, eps2, G, ax, ay, az);
                return nb::check_launch("bh_group_f64_kernel");
            case NB_F32C:
                if (G != t->G)
                    return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_accel: G differs from the build's");
                bh_group_f32_kernel<<<grid, TR_THREADS, 0, s>>>(t->rec32, t->info, t->ids, x, y, z,
                                                                t->box, n, (float)theta,
                                                                (float)eps2, ax, ay, az);
                return nb::check_launch("bh_group_f32_kernel");
            default:
                break;
        }
    } else if (opening == NB_OPEN_LEARNED) {
        if (prec != NB_F32C)
            return nb::set_error(NB_ERR_UNSUPPORTED, "nb_bh_accel: NB_OPEN_LEARNED runs in NB_F32C");
        if (G != t->G)
            return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_accel: G differs from the build's");
        NB_TRY(nb_need_records(t, NB_REC_LEARNED, "nb_bh_accel"));
        return nb::launch_learned(ctx, t, x, y, z, ax, ay, az, eps2, nullptr, s);
    }
    return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_accel: unknown opening %d / precision %d",
                         (int)opening, (int)prec);
}

nb_status nb_bh_count_interactions(nb_ctx* ctx, const nb_bh_tree* t, const double* x,
                                   const double* y, const double* z, nb_opening opening,
                                   unsigned long long* out_dev, nb_stream_t stream_) {
    NB_CHECK_CTX(ctx);
    if (!t || !t->built) return nb::set_error(NB_ERR_NOT_BUILT, "nb_bh_count_interactions: tree not built");
    if (!x || !y || !z || !out_dev) return nb::set_error(NB_ERR_INVALID_ARG, "null pointer");
    if (opening != NB_OPEN_THETA && opening != NB_OPEN_THETA_GROUP)
        return nb::set_error(NB_ERR_UNSUPPORTED, "nb_bh_count_interactions: theta rules only");
    NB_TRY(nb_need_records(t, NB_REC_FP64, "nb_bh_count_interactions"));
    cudaStream_t s = (cudaStream_t)stream_;
    NB_CUDA_TRY(cudaMemsetAsync(out_dev, 0, 2 * sizeof(unsigned long long), s));
    bh_count_kernel<<<nb::ceil_div(t->n, TR_THREADS), TR_THREADS, 0, s>>>(
        t->rec64, t->info, t->ids, x, y, z, t->n, t->params.theta,
        opening == NB_OPEN_THETA_GROUP ? 1 : 0, out_dev);
    return nb::check_launch("bh_count_kernel");
}

nb_status nb_bh_accel_learned_counted(nb_ctx* ctx, const nb_bh_tree* t, const double* x,
                                     const double* y, const double* z, double* ax, double* ay,
                                     double* az, double eps2, unsigned long long* counters_dev,
                                     nb_stream_t stream) {
    NB_CHECK_CTX(ctx);
    if (!t || !t->built) return nb::set_error(NB_ERR_NOT_BUILT, "tree not built");
    if (!counters_dev) return nb::set_error(NB_ERR_INVALID_ARG, "null counters");
    NB_TRY(nb_need_records(t, NB_REC_LEARNED, "nb_bh_accel_learned_counted"));
    NB_CUDA_TRY(cudaMemsetAsync(counters_dev, 0, 2 * sizeof(unsigned long long), (cudaStream_t)stream));
    return nb::launch_learned(ctx, t, x, y, z, ax, ay, az, eps2, counters_dev, (cudaStream_t)stream);
}

nb_status nb_bh_graph_create(nb_ctx* ctx, nb_bh_tree* t, const double* m, double* x, double* y,
                             double* z, double* vx, double* vy, double* vz, double* vhx,
                             double* vhy, double* vhz, double* ax, double* ay, double* az,
                             uint32_t n, double G, double eps2, double dt, int steps,
                             nb_opening opening, nb_precision prec, nb_graph** out) {
    NB_CHECK_CTX(ctx);
    if (!t || !out || steps < 1)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_graph_create: bad arguments");
    if (t->phase_timing)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_graph_create: phase timing is on");
    *out = nullptr;
    int ps = 0;  // one-time queries happen here, outside the capture
    for (nb_precision p : {NB_F64_IEEE, NB_F64, NB_DF64}) NB_TRY(lane_per_sm(p, &ps));
    NB_TRY(nb::learned_per_sm(&ps));
    cudaStream_t s;
    NB_CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        cudaStreamDestroy(s);
        return nb::cuda_error(e, "cudaStreamBeginCapture");
    }
    nb_status st = NB_OK;
    const nb_stream_t ns = (nb_stream_t)s;
    for (int k = 0; k < steps && st == NB_OK; ++k) {
        st = nb_leapfrog_kick_drift(ctx, vhx, vhy, vhz, vx, vy, vz, x, y, z, ax, ay, az, n, dt, ns);
        if (st == NB_OK) st = nb_bh_build(ctx, t, m, x, y, z, n, G, ns);
        if (st == NB_OK) st = nb_bh_accel(ctx, t, x, y, z, ax, ay, az, G, eps2, opening, prec, ns);
        if (st == NB_OK) st = nb_leapfrog_kick(ctx, vx, vy, vz, vhx, vhy, vhz, ax, ay, az, n, dt, ns);
    }
    return nb_finish_capture(s, st, steps, out);
}

}  // extern "C"
