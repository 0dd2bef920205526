// nb_bh.cu -- Barnes-Hut octree build on the GPU (replaces BarnesHutOctree::buildOctree,
// ParallelOctreeTopDownSubtrees.cpp:15-93, and its AABB / centre-of-mass / sortBodies passes).
//
// Pipeline (all on one stream, no host round trip):
//  1. AABB with the reference's conventions (nb_integrate.cu).
//  2. keys: per body the octant digit of every level from the reference's FP64 recurrence
//     (mid = min + edge/2, strict compares, z below the midpoint selects bit 0; child min corner =
//     parent min + child edge), mapped to the visit rank so that ascending keys are the
//     reference's DFS pop order; read off a 52-bit fixed-point position wherever the body is
//     provably far enough from every midpoint for the recurrence's rounding not to matter.
//  3. stable LSD radix sort of (key, body id).
//  4. bodies whose first 21 digits collide get their next 21 digits and are re-sorted in place.
//  5. splits: adjacent sorted bodies share a prefix of L digits; the split belongs to the cell at
//     level L containing both. Its cell range comes from galloping searches over the keys; the
//     leftmost split of each cell ("first split") stands for the cell.
//  6. DFS numbering: each sorted position p starts popc(mask[p]) internal cells plus its leaf;
//     an exclusive scan gives every node its DFS pre-order index and skip link.
// What later launches want zeroed or filled is written by earlier ones (keys: the sort's counters,
// second key words and level masks; splits: the child lists), the digit offsets are summed by the
// sort's passes and the node counts by the scan: 18 launches, where separate ones took 26 and 22 us
// more at 16,411 bodies. Each launch of the chain may start while the one before it ends
// (nb_grid_wait): 122 us for that build instead of 162.
//  7. bottom-up centre of mass: leaves and cells by blocks over chunks of 256 sorted positions
//     (deepest level first), the cells reaching past their chunk (at most one per level) by tiers
//     of blocks over 96 chunks each; children summed in octant order 0..7
//     (bit-identical to BarnesHutOctree.cpp:304-311), node records written with the sums.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "nb_aabb.cuh"
#include "nb_bh.cuh"
#include "nb_sort.cuh"

namespace nb {
nb_status launch_aabb(nb_ctx* ctx, const double* x, const double* y, const double* z, uint32_t n,
                      double* out_dev, cudaStream_t stream);
}

namespace {

constexpr int BH_THREADS = 256;
constexpr uint32_t RUN_LIMIT = 1u << 14;  // longest run of equal first key words we re-sort

// Order-preserving map of an FP64 value (no NaN, -0 already turned into +0) to uint64: the
// strict comparisons of the recurrence become integer comparisons (ALU instead of FP64 pipe).
__device__ __forceinline__ uint64_t ordered_bits(double v) {
    const uint64_t u = (uint64_t)__double_as_longlong(v);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// The edge halvings of the recurrence: exponent decrements while they stay exact (the normal,
// positive edges of <= 42 levels), otherwise (a zero or tiny box) FP64 divisions by 2.
struct Halving {
    double e;
    uint64_t e_bits;
    bool bits;
    __device__ explicit Halving(double edge) : e(edge) {
        e_bits = (uint64_t)__double_as_longlong(edge);
        bits = (e_bits >> 52) > 64 && (e_bits >> 52) < 0x7ff;
    }
    // edge / 2 of the next level
    __device__ double next() {
        if (bits) {
            e_bits -= 1ull << 52;
            return __longlong_as_double((long long)e_bits);
        }
        e = e / 2;
        return e;
    }
};

// Octant digits of levels [L0, last) appended to `key` for a body (ordered bits ox, oy, oz of
// its coordinates), from the cell mins entering level L0: the reference's FP64 recurrence
// (mid = min + edge/2 rounded as FP64, strict compares, child min = mid or min). Only the three
// midpoint additions per level run on the FP64 pipe: the compares are integer compares of
// order-preserving bit patterns (exact: a midpoint is never -0 since edge/2 > 0, and the body's
// -0 coordinates are taken as +0, which compares equal). Digits of levels below `first` are not
// appended.
__device__ uint64_t key_levels(Halving h, uint64_t ox, uint64_t oy, uint64_t oz, double mnx,
                               double mny, double mnz, int L0, int first, int last,
                               uint64_t key) {
    for (int L = L0; L < last; ++L) {
        const double ce = h.next();
        const double midx = __dadd_rn(mnx, ce);
        const double midy = __dadd_rn(mny, ce);
        const double midz = __dadd_rn(mnz, ce);
        const bool up = oy > ordered_bits(midy), rt = ox > ordered_bits(midx),
                   bk = oz < ordered_bits(midz);
        if (L >= first)
            key = (key << 3) |
                  nb_visit_of_octant((uint32_t)up * 4u + (uint32_t)rt * 2u + (uint32_t)bk);
        if (rt) mnx = midx;
        if (up) mny = midy;
        if (!bk) mnz = midz;
    }
    return key;
}

__device__ __forceinline__ uint64_t ordered_coord(double v) {
    return ordered_bits(v == 0.0 ? 0.0 : v);
}

// Octant digits of levels [word*21, word*21+21) for a body, from the root.
__device__ uint64_t key_word(const double* __restrict__ box, double px, double py, double pz,
                             int word) {
    const int first = word * NB_KEY_LEVELS;
    return key_levels(Halving(box[6]), ordered_coord(px), ordered_coord(py), ordered_coord(pz),
                      box[0], box[1], box[2], 0, first, first + NB_KEY_LEVELS, 0);
}

// Quantized keys (NB_BUILD_QUANTIZED_KEYS): every coordinate as a 42-bit fraction of the box,
// floor((v - min) * 2^42 / edge), one bit per level. Bodies fall into the cells of the
// reference's recurrence except within FP64 rounding of a cell midpoint (there the quantized
// rule puts them in the upper half). Bits interleave with the usual 3-way spread, the digits
// already in visit order: visit rank = 4 * (y upper) + 2 * (z lower) + (x lower).
__device__ __forceinline__ uint64_t spread3(uint64_t v) {  // bit i -> bit 3i, i < 21
    v &= 0x1fffffull;
    v = (v | v << 32) & 0x1f00000000ffffull;
    v = (v | v << 16) & 0x1f0000ff0000ffull;
    v = (v | v << 8) & 0x100f00f00f00f00full;
    v = (v | v << 4) & 0x10c30c30c30c30c3ull;
    v = (v | v << 2) & 0x1249249249249249ull;
    return v;
}

__device__ __forceinline__ uint64_t quantize42(double v, double mn, double scale) {
    const double q = (v - mn) * scale;
    const uint64_t top = (1ull << 42) - 1;
    if (!(q > 0.0)) return 0;
    const uint64_t u = __double2ull_rz(q);
    return u > top ? top : u;
}

__device__ uint64_t key_word_quantized(const double* __restrict__ box, double px, double py,
                                       double pz, int word) {
    const double scale = box[6] > 0.0 ? 4398046511104.0 / box[6] : 0.0;  // 2^42 / edge
    const uint64_t ix = quantize42(px, box[0], scale), iy = quantize42(py, box[1], scale),
                   iz = quantize42(pz, box[2], scale);
    const int shift = word == 0 ? NB_KEY_LEVELS : 0;
    const uint64_t m = 0x1fffffull;
    const uint64_t hx = (ix >> shift) & m, hy = (iy >> shift) & m, hz = (iz >> shift) & m;
    return (spread3(hy) << 2) | (spread3(~hz & m) << 1) | spread3(~hx & m);
}

// Box entries beyond the AABB, by the first four threads of the keys kernels.
using nbfix::box_extras;
using nbfix::BOX_WORDS;

// Zeroes what the launches after the keys count on: the sort's counters, the second key words and
// the level masks, by all threads of the grid.
struct BuildZero {
    uint4* sort;
    uint32_t sort_n;  // in 16-byte words
    uint64_t* key1;
    unsigned long long* mask;
};
__device__ __forceinline__ void build_zero(const BuildZero& Z, uint32_t i, uint32_t n) {
    for (uint32_t k = i; k < Z.sort_n; k += gridDim.x * blockDim.x)
        Z.sort[k] = make_uint4(0, 0, 0, 0);
    if (i < n) {
        Z.key1[i] = 0;
        Z.mask[i] = 0;
    }
}

__global__ void keys_quantized_kernel(const double* x, const double* y,
                                      const double* z, uint32_t n,
                                      double* __restrict__ box, uint64_t* __restrict__ key0,
                                      uint32_t* __restrict__ ids, BuildZero Z) {
    nb_grid_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    box_extras(box, i);
    build_zero(Z, i, n);
    if (i >= n) return;
    key0[i] = key_word_quantized(box, x[i], y[i], z[i], 0);
    ids[i] = i;
}

// First key word of every body, the digits of key_word bit for bit, mostly without the FP64
// recurrence. The recurrence's midpoints differ from the dyadic grid min + (2j + 1) edge /
// 2^(L+1) only by the rounding of its additions (the halvings are exact): after L + 1 of them by
// at most (L + 1) 2^-53 R, R = |min| + edge bounding every midpoint, i.e. (L + 1) R / (2 edge)
// units of edge / 2^52. A coordinate as a 52-bit fraction of the edge, U = floor((v - min) 2^52 /
// edge), is within 1.5 units of the exact value (three roundings), so when U is more than
// m = 10.5 R / edge + 4 units from every multiple of 2^31 (the grid boundaries of levels 0..20),
// the digits of those levels are bits 51..31 of U. Bodies inside a margin, and boxes whose edge
// the recurrence does not halve by exponent arithmetic, take the recurrence itself.
struct FixedGrid {
    double scale;  // 2^52 / edge
    long long margin[3];
    bool ok;
};

__device__ FixedGrid fixed_grid(const double* __restrict__ box) {
    FixedGrid g;
    const double e = box[6];
    const uint64_t eb = (uint64_t)__double_as_longlong(e);
    g.ok = (eb >> 52) > 64 && (eb >> 52) < 0x7ff;  // Halving's exponent mode: positive, normal
    g.scale = g.ok ? 4503599627370496.0 / e : 0.0;
    g.ok = g.ok && g.scale < 1e308;
#pragma unroll
    for (int a = 0; a < 3; ++a) {  // R / edge = |min| * scale / 2^52 + 1
        const double m = 10.5 * fma(fabs(box[a]), g.scale * 0x1p-52, 1.0) * (1.0 + 0x1p-30) + 4.0;
        g.ok = g.ok && m < 0x1p29;  // false for NaN as well
        g.margin[a] = g.ok ? (long long)m + 1 : 0;
    }
    return g;
}

// Bits 51..31 of U for one axis, or -1 when U lies within the margin of a grid boundary (or the
// coordinate is outside the box or NaN).
__device__ __forceinline__ long long fixed_digits(double v, double mn, double scale, long long m) {
    const double u = __dmul_rn(__dsub_rn(v, mn), scale);
    // 0 <= u <= 2^52, by its bits; the integer part by a shift
    const long long b = __double_as_longlong(u);
    if ((uint64_t)b > 0x4330000000000000ull && (b << 1) != 0) return -1;
    const int e = (int)(b >> 52);
    const long long U = e < 1023 ? 0 : ((b & 0xfffffffffffffll) | (1ll << 52)) >> (1075 - e);
    const long long hi = min((U + m) >> 31, 0x1fffffll), lo = max((U - m - 1) >> 31, 0ll);
    return hi == lo ? hi : -1;
}

// First key word of a body by the rule above.
__device__ __forceinline__ uint64_t exact_key(const double* __restrict__ box, const FixedGrid& g,
                                              double px, double py, double pz) {
    long long hx = -1, hy = -1, hz = -1;
    if (g.ok) {
        hx = fixed_digits(px, box[0], g.scale, g.margin[0]);
        hy = fixed_digits(py, box[1], g.scale, g.margin[1]);
        hz = fixed_digits(pz, box[2], g.scale, g.margin[2]);
    }
    if ((hx | hy | hz) < 0) return key_word(box, px, py, pz, 0);
    const uint64_t m = 0x1fffffull;  // visit rank = 4 (y upper) + 2 (z lower) + (x lower)
    return (spread3((uint64_t)hy) << 2) | (spread3(~(uint64_t)hz & m) << 1) |
           spread3(~(uint64_t)hx & m);
}

__global__ void __launch_bounds__(BH_THREADS)
keys_kernel(const double* x, const double* y,
            const double* z, uint32_t n, double* __restrict__ box,
            uint64_t* __restrict__ key0, uint32_t* __restrict__ ids, BuildZero Z) {
    __shared__ FixedGrid grid_s;  // once per block: it takes an FP64 division
    nb_grid_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    box_extras(box, i);
    build_zero(Z, i, n);
    if (threadIdx.x == 0) grid_s = fixed_grid(box);
    __syncthreads();
    if (i >= n) return;
    key0[i] = exact_key(box, grid_s, x[i], y[i], z[i]);
    ids[i] = i;
}

// Runs of equal first words: compute the second word and insertion-sort the run (stable).
__device__ __forceinline__ void fix_run(uint32_t p, const double* __restrict__ x,
                                        const double* __restrict__ y,
                                        const double* __restrict__ z, uint32_t n,
                                        const double* __restrict__ box, const uint64_t* key0,
                                        uint64_t* key1, uint32_t* ids, uint32_t* err,
                                        int quantized) {
    if (p + 1 >= n) return;
    const uint64_t k = key0[p];
    if (key0[p + 1] != k) return;
    if (p > 0 && key0[p - 1] == k) return;
    uint32_t r = 2;
    while (p + r < n && key0[p + r] == k && r < RUN_LIMIT) ++r;
    if (p + r < n && key0[p + r] == k) {
        atomicOr(err, NB_DEVERR_DEPTH);
        return;
    }
    for (uint32_t q = p; q < p + r; ++q) {
        const uint32_t b = ids[q];
        key1[q] = quantized ? key_word_quantized(box, x[b], y[b], z[b], 1)
                            : key_word(box, x[b], y[b], z[b], 1);
    }
    for (uint32_t q = p + 1; q < p + r; ++q) {  // insertion sort, stable
        const uint64_t kk = key1[q];
        const uint32_t bb = ids[q];
        uint32_t s = q;
        while (s > p && key1[s - 1] > kk) {
            key1[s] = key1[s - 1];
            ids[s] = ids[s - 1];
            --s;
        }
        key1[s] = kk;
        ids[s] = bb;
    }
}

__global__ void runs_fixup_kernel(const double* x, const double* y,
                                  const double* z, uint32_t n,
                                  const double* box, const uint64_t* key0,
                                  uint64_t* __restrict__ key1, uint32_t* __restrict__ ids,
                                  uint32_t* __restrict__ err, int quantized) {
    nb_grid_wait();
    fix_run(blockIdx.x * blockDim.x + threadIdx.x, x, y, z, n, box, key0, key1, ids, err,
            quantized);
}

// Number of leading octal digits two sorted positions share (0 .. 42).
__device__ __forceinline__ int shared_digits(const uint64_t* __restrict__ key0,
                                             const uint64_t* __restrict__ key1, uint32_t p,
                                             uint32_t q) {
    const uint64_t a = key0[p], b = key0[q];
    if (a != b) return (__clzll((long long)(a ^ b)) - 1) / 3;
    const uint64_t c = key1[p], d = key1[q];
    if (c != d) return NB_KEY_LEVELS + (__clzll((long long)(c ^ d)) - 1) / 3;
    return 2 * NB_KEY_LEVELS;
}

__device__ __forceinline__ void split_at(uint32_t j, const uint64_t* __restrict__ key0,
                                         const uint64_t* __restrict__ key1, uint32_t n,
                                         uint8_t* split_level, uint32_t* split_start,
                                         uint32_t* split_end, unsigned long long* mask,
                                         uint32_t* err) {
    if (j + 1 >= n) return;
    int L = shared_digits(key0, key1, j, j + 1);
    if (L >= 2 * NB_KEY_LEVELS) {
        atomicOr(err, NB_DEVERR_DEPTH);
        L = 2 * NB_KEY_LEVELS - 1;
    }
    split_level[j] = (uint8_t)L;
    // leftmost a <= j with shared_digits(a, j) >= L (galloping, then bisection)
    long long good = j, bad = -1;
    for (long long step = 1;; step <<= 1) {
        const long long c = good - step;
        if (c < 0) break;
        if (shared_digits(key0, key1, (uint32_t)c, j) >= L) {
            good = c;
        } else {
            bad = c;
            break;
        }
    }
    while (good - bad > 1) {
        const long long mid = bad + (good - bad) / 2;
        if (shared_digits(key0, key1, (uint32_t)mid, j) >= L) good = mid; else bad = mid;
    }
    const uint32_t a = (uint32_t)good;
    split_start[j] = a;
    const bool first = (a == j) || shared_digits(key0, key1, a, j) > L;
    if (!first) {
        split_end[j] = NB_NONE;
        return;
    }
    // rightmost b >= j+1 with shared_digits(j, b) >= L
    long long g2 = j + 1, b2 = n;
    for (long long step = 1;; step <<= 1) {
        const long long c = g2 + step;
        if (c >= (long long)n) break;
        if (shared_digits(key0, key1, j, (uint32_t)c) >= L) {
            g2 = c;
        } else {
            b2 = c;
            break;
        }
    }
    while (b2 - g2 > 1) {
        const long long mid = g2 + (b2 - g2) / 2;
        if (shared_digits(key0, key1, j, (uint32_t)mid) >= L) g2 = mid; else b2 = mid;
    }
    split_end[j] = (uint32_t)g2;
    atomicOr(&mask[a], 1ull << L);
}

__global__ void splits_kernel(const uint64_t* key0, const uint64_t* key1,
                              uint32_t n, uint8_t* __restrict__ split_level,
                              uint32_t* __restrict__ split_start, uint32_t* __restrict__ split_end,
                              unsigned long long* __restrict__ mask, uint32_t* __restrict__ children,
                              uint32_t* __restrict__ err) {
    nb_grid_wait();
    // the child lists start empty (two nodes per position at most): stores that the searches' round
    // trips leave room for
    const uint32_t blk = min(blockDim.x, n - blockIdx.x * blockDim.x);
    uint4* cl = reinterpret_cast<uint4*>(children) + (size_t)blockIdx.x * blockDim.x * 4;
    for (uint32_t k = threadIdx.x; k < blk * 4; k += blockDim.x)
        cl[k] = make_uint4(NB_NONE, NB_NONE, NB_NONE, NB_NONE);
    split_at(blockIdx.x * blockDim.x + threadIdx.x, key0, key1, n, split_level, split_start,
             split_end, mask, err);
}

__device__ __forceinline__ uint32_t node_index(const uint32_t* __restrict__ base,
                                               const unsigned long long* __restrict__ mask,
                                               uint32_t start, int level) {
    return base[start] + __popcll(mask[start] & ((1ull << level) - 1ull));
}

// Parent of the node covering sorted positions [a, b]: the cell at level max(dl, dr) holding the
// neighbouring split (dl = level of split a-1, dr = level of split b, -1 when absent).
__device__ __forceinline__ uint32_t parent_of(uint32_t a, uint32_t b, int dl, int dr,
                                              const uint8_t* __restrict__ split_level,
                                              const uint32_t* __restrict__ split_start,
                                              const uint32_t* __restrict__ base,
                                              const unsigned long long* __restrict__ mask) {
    if (dl < 0 && dr < 0) return NB_NONE;
    const uint32_t s = dl >= dr ? a - 1 : b;
    return node_index(base, mask, split_start[s], split_level[s]);
}

__device__ __forceinline__ uint32_t digit_at(const uint64_t* __restrict__ key0,
                                             const uint64_t* __restrict__ key1, uint32_t q, int L) {
    if (L < NB_KEY_LEVELS) return (uint32_t)(key0[q] >> (60 - 3 * L)) & 7u;
    return (uint32_t)(key1[q] >> (60 - 3 * (L - NB_KEY_LEVELS))) & 7u;
}

// The node tables emit_at writes (global memory).
struct NodeTable {
    uint8_t* level;
    uint32_t *first, *last, *skip, *body, *info, *children;
};

// The leaf of sorted position p and the internal cell whose first split it is.
__device__ __forceinline__ void emit_at(uint32_t p, uint32_t n, const uint32_t* ids,
                                        const uint8_t* split_level, const uint32_t* split_start,
                                        const uint32_t* split_end, const unsigned long long* mask,
                                        const uint32_t* base, const uint64_t* key0,
                                        const uint64_t* key1, const NodeTable& T) {
    if (p >= n) return;
    if (p == 0) T.info[0] = base[n];
    {  // leaf of the body at sorted position p
        const int dl = p > 0 ? (int)split_level[p - 1] : -1;
        const int dr = p + 1 < n ? (int)split_level[p] : -1;
        const uint32_t idx = base[p] + __popcll(mask[p]);
        T.level[idx] = (uint8_t)(max(dl, dr) + 1);
        T.first[idx] = p;
        T.last[idx] = p;
        T.skip[idx] = base[p + 1];
        T.body[idx] = ids[p];
        const uint32_t par = parent_of(p, p, dl, dr, split_level, split_start, base, mask);
        if (par != NB_NONE) {
            // the parent's level is the deeper boundary split; slot = visit rank there
            T.children[(size_t)par * 8 + digit_at(key0, key1, p, max(dl, dr))] = idx;
        }
    }
    if (p + 1 < n && split_end[p] != NB_NONE) {  // internal cell whose first split is p
        const uint32_t a = split_start[p], b = split_end[p];
        const int L = split_level[p];
        const uint32_t idx = node_index(base, mask, a, L);
        T.level[idx] = (uint8_t)L;
        T.first[idx] = a;
        T.last[idx] = b;
        T.skip[idx] = base[b + 1];
        T.body[idx] = NB_NONE;
        const int dl = a > 0 ? (int)split_level[a - 1] : -1;
        const int dr = b + 1 < n ? (int)split_level[b] : -1;
        const uint32_t par = parent_of(a, b, dl, dr, split_level, split_start, base, mask);
        if (par != NB_NONE) {
            T.children[(size_t)par * 8 + digit_at(key0, key1, a, max(dl, dr))] = idx;
        }
    }
}

__global__ void emit_kernel(uint32_t n, const uint32_t* ids,
                            const uint8_t* split_level,
                            const uint32_t* split_start,
                            const uint32_t* split_end,
                            const unsigned long long* mask,
                            const uint32_t* base, const uint64_t* key0,
                            const uint64_t* key1, NodeTable T) {
    nb_grid_wait();
    emit_at(blockIdx.x * blockDim.x + threadIdx.x, n, ids, split_level, split_start, split_end,
            mask, base, key0, key1, T);
}

// Steps 1 to 6 for small systems in one block, sharing the device functions above. Bound by
// latency: one block's barriers and dependent instructions. (Key, body) pairs sort bitonically
// (ties by body id: the stable order) in registers, with exchanges by shuffle within a warp; the
// cells' ranges come from the splits' levels and their minima over powers of two, a halving walk
// over bytes in shared memory; with all exchanges through shared memory and searches over the keys
// it took 41 us at 777 bodies, this way 28. The DFS numbering is a block scan. The whole build,
// this way against the chain of launches: 57 / 84 us at 777 bodies, 84 / 94 at 2,048; at 2,500 it
// would be 116 / 97, which is where the line is.
constexpr uint32_t SB_MAX_N = 2048;

constexpr int small_log2(uint32_t v) { return v <= 1 ? 0 : 1 + small_log2(v / 2); }
template <uint32_t CAP>
constexpr size_t small_smem_bytes() {  // keys, masks, ids, cell ranges, indices, split levels' minima
    return CAP * (8 + 8 + 8 + 4 + 4 + 4 + 4 + small_log2(CAP)) + 64;
}

__device__ __forceinline__ uint32_t small_block_scan(uint32_t v, uint32_t* warp_sums,
                                                     uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t ws = lane < blockDim.x / 32 ? warp_sums[lane] : 0u, wi = ws;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= (uint32_t)o) wi += t;
    }
    *total = __shfl_sync(0xffffffffu, wi, 31);
    return __shfl_sync(0xffffffffu, wi - ws, warp) + incl - v;
}

template <uint32_t CAP, uint32_t THREADS>
__global__ void __launch_bounds__(THREADS)
build_small_kernel(const double* x, const double* y,
                   const double* z, uint32_t n, double* __restrict__ box,
                   uint64_t* __restrict__ key0_out, uint64_t* __restrict__ key1_out,
                   uint32_t* __restrict__ ids_out, unsigned long long* __restrict__ mask_out,
                   uint32_t* __restrict__ base_out, NodeTable T, uint32_t* __restrict__ err,
                   int quantized) {
    nb_grid_wait();
    constexpr int PER = CAP / THREADS;  // positions per thread
    extern __shared__ __align__(16) unsigned char small_smem[];
    uint64_t* key0 = reinterpret_cast<uint64_t*>(small_smem);
    uint64_t* key1 = key0 + CAP;
    unsigned long long* mask = reinterpret_cast<unsigned long long*>(key1 + CAP);
    uint32_t* ids = reinterpret_cast<uint32_t*>(mask + CAP);
    uint32_t* split_start = ids + CAP;
    uint32_t* split_end = split_start + CAP;
    uint32_t* base = split_end + CAP;  // CAP + 1 entries
    // level_min[d][p]: the least split level of positions p .. p + 2^d - 1; d = 0: the levels
    uint8_t (*level_min)[CAP] = reinterpret_cast<uint8_t (*)[CAP]>(base + CAP + 1);
    uint8_t* split_level = level_min[0];
    __shared__ long long wmin[3][32], wmax[3][32];
    __shared__ uint32_t warp_sums[32];
    __shared__ double sbox[BOX_WORDS];
    __shared__ FixedGrid grid_s;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // box, with the reference's zero-initialised bounds
    double px[PER], py[PER], pz[PER];
    const long long zero = nbaabb::ord_of(0.0);
    long long mn[3] = {zero, zero, zero}, mx[3] = {zero, zero, zero};
#pragma unroll
    for (int h = 0; h < PER; ++h) {
        const uint32_t i = tid * PER + h;
        const bool in = i < n;
        px[h] = in ? x[i] : 0.0;
        py[h] = in ? y[i] : 0.0;
        pz[h] = in ? z[i] : 0.0;
    }
    // children lists start empty; written before the barriers below, filled after them
    for (uint32_t k = tid; k < 4 * n; k += THREADS)
        reinterpret_cast<uint4*>(T.children)[k] = make_uint4(NB_NONE, NB_NONE, NB_NONE, NB_NONE);
#pragma unroll
    for (int h = 0; h < PER; ++h) {
        const bool in = tid * PER + h < n;
        const long long o[3] = {nbaabb::ord_of(px[h]), nbaabb::ord_of(py[h]),
                                nbaabb::ord_of(pz[h])};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (!in) continue;
            mn[a] = min(mn[a], o[a]);
            mx[a] = max(mx[a], o[a]);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
            mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
        }
        if (lane == 0) {
            wmin[a][warp] = mn[a];
            wmax[a][warp] = mx[a];
        }
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            mn[a] = lane < THREADS / 32 ? wmin[a][lane] : zero;
            mx[a] = lane < THREADS / 32 ? wmax[a][lane] : zero;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
                mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
            }
        }
        if (lane == 0)
            nbaabb::cube_rule(nbaabb::val_of(mn[0]), nbaabb::val_of(mn[1]), nbaabb::val_of(mn[2]),
                              nbaabb::val_of(mx[0]), nbaabb::val_of(mx[1]), nbaabb::val_of(mx[2]),
                              sbox);
        __syncwarp();
        box_extras(sbox, lane);
        __syncwarp();
        if (lane < BOX_WORDS) box[lane] = sbox[lane];
        if (lane == 0 && !quantized) grid_s = fixed_grid(sbox);
    }
    __syncthreads();
    // (key, body) number e = tid * PER + h in registers; exchanges within a thread, by shuffles
    // within a warp, and through shared memory beyond
    uint64_t key[PER];
    uint32_t id[PER];
#pragma unroll
    for (int h = 0; h < PER; ++h) {
        const uint32_t i = tid * PER + h;
        key[h] = ~0ull;  // above every key (63 bits)
        id[h] = i;
        if (i < n)
            key[h] = quantized ? key_word_quantized(sbox, px[h], py[h], pz[h], 0)
                               : exact_key(sbox, grid_s, px[h], py[h], pz[h]);
        key1[i] = 0;
        mask[i] = 0;
    }
    uint32_t m = 2;  // positions to sort: a power of two
    while (m < n) m <<= 1;
    for (uint32_t k = 2; k <= m; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            if (j < (uint32_t)PER) {
#pragma unroll
                for (int h = 0; h < PER; ++h) {
#pragma unroll
                    for (int g = h + 1; g < PER; ++g) {
                        if ((uint32_t)(h ^ g) != j) continue;
                        const bool up = ((tid * PER + h) & k) == 0;
                        const bool gt = key[h] > key[g] || (key[h] == key[g] && id[h] > id[g]);
                        if (gt == up) {
                            const uint64_t tk = key[h];
                            key[h] = key[g];
                            key[g] = tk;
                            const uint32_t ti = id[h];
                            id[h] = id[g];
                            id[g] = ti;
                        }
                    }
                }
                continue;
            }
            const bool far = j >= 32u * PER;
            if (far) {
#pragma unroll
                for (int h = 0; h < PER; ++h) {
                    key0[tid * PER + h] = key[h];
                    ids[tid * PER + h] = id[h];
                }
                __syncthreads();
            }
#pragma unroll
            for (int h = 0; h < PER; ++h) {
                const uint32_t e = tid * PER + h;
                uint64_t ok;
                uint32_t oi;
                if (far) {
                    ok = key0[e ^ j];
                    oi = ids[e ^ j];
                } else {
                    ok = __shfl_xor_sync(0xffffffffu, key[h], j / PER);
                    oi = __shfl_xor_sync(0xffffffffu, id[h], j / PER);
                }
                const bool low = (e & j) == 0, up = (e & k) == 0;
                const bool gt = key[h] > ok || (key[h] == ok && id[h] > oi);
                if (gt == (low == up)) {  // the other one belongs here
                    key[h] = ok;
                    id[h] = oi;
                }
            }
            if (far) __syncthreads();
        }
    }
#pragma unroll
    for (int h = 0; h < PER; ++h) {
        key0[tid * PER + h] = key[h];
        ids[tid * PER + h] = id[h];
    }
    __syncthreads();
    for (uint32_t p = tid; p < n; p += THREADS)
        fix_run(p, x, y, z, n, sbox, key0, key1, ids, err, quantized);
    __syncthreads();
    // the splits' levels and their minima over powers of two, then the cells' ranges: a cell of
    // level L reaches from its split as far as no split is below L, and the split whose left side
    // has none at L stands for the cell (split_at's rules)
    const int log = __ffs((int)m) - 1;
    for (uint32_t p = tid; p < m; p += THREADS) {
        int L = 0;  // past the last split: below or at every level, never crossed
        if (p + 1 < n) {
            L = shared_digits(key0, key1, p, p + 1);
            if (L >= 2 * NB_KEY_LEVELS) {
                atomicOr(err, NB_DEVERR_DEPTH);
                L = 2 * NB_KEY_LEVELS - 1;
            }
        }
        split_level[p] = (uint8_t)L;
    }
    __syncthreads();
    for (int d = 1; d < log; ++d) {
        const uint32_t half = 1u << (d - 1);
        for (uint32_t p = tid; p < m; p += THREADS)
            level_min[d][p] = p + half < m ? min(level_min[d - 1][p], level_min[d - 1][p + half])
                                             : level_min[d - 1][p];
        __syncthreads();
    }
    for (uint32_t p = tid; p + 1 < n; p += THREADS) {
        const uint32_t L = split_level[p];
        uint32_t a = p, least = 255;
        for (int d = log - 1; d >= 0; --d) {
            const uint32_t w = 1u << d;
            if (a < w) continue;
            const uint32_t v = level_min[d][a - w];
            if (v >= L) {
                a -= w;
                least = min(least, v);
            }
        }
        split_start[p] = a;
        split_end[p] = NB_NONE;
        if (least > L) {  // the leftmost split of its cell
            uint32_t b = p;
            for (int d = log - 1; d >= 0; --d) {
                const uint32_t w = 1u << d;
                if (b + w < n && level_min[d][b] >= L) b += w;
            }
            split_end[p] = b;
            atomicOr(&mask[a], 1ull << L);
        }
    }
    __syncthreads();
    {
        const uint32_t p = PER * tid;
        uint32_t c[PER], sum = 0, total;
#pragma unroll
        for (int h = 0; h < PER; ++h) {
            c[h] = p + h < n ? __popcll(mask[p + h]) + 1 : 0u;
            sum += c[h];
        }
        uint32_t before = small_block_scan(sum, warp_sums, &total);
#pragma unroll
        for (int h = 0; h < PER; ++h) {
            if (p + h < n) base[p + h] = before;
            before += c[h];
        }
        if (tid == 0) base[n] = total;
    }
    __syncthreads();
    for (uint32_t p = tid; p < n; p += THREADS) {
        key0_out[p] = key0[p];
        key1_out[p] = key1[p];
        ids_out[p] = ids[p];
        mask_out[p] = mask[p];
        base_out[p] = base[p];
        emit_at(p, n, ids, split_level, split_start, split_end, mask, base, key0, key1, T);
    }
    if (tid == 0) base_out[n] = base[n];
}

struct ComArgs {
    uint32_t n;
    uint32_t* err;      // device error word
    uint32_t records;  // NB_REC_* sets to compute
    const double *m, *x, *y, *z;
    const double* box;
    double G;
    const uint64_t *key0, *key1;
    const uint32_t* ids;
    const unsigned long long* mask;
    const uint32_t* base;
    const uint8_t* node_level;
    const uint32_t *node_first, *node_last, *node_skip, *node_body;
    uint32_t* tier_slot;
    uint32_t* node_count;
    double *comx, *comy, *comz, *mass, *q;
    NodeRec64* rec64;
    nbfix::FixHi* fix_hi;
    uint4* fix_lo;
    NodeRec32* rec32;
    DfTerms* df_terms;
    NodeAux* aux;
    const uint32_t* node_first_pos;
    uint32_t* children;
    float4* sorted4;
    float4* sorted4lo;
};

// Edge of a cell of the given level: box edge * 2^-level by exponent arithmetic (exact, and no
// FP64 instructions) while the result stays a normal number, else ldexp.
__device__ __forceinline__ double cell_edge64(double box_edge, int level) {
    const long long bits = __double_as_longlong(box_edge);
    const int biased = (int)((bits >> 52) & 0x7ff);
    if (biased > level + 1 && biased < 0x7ff)
        return __longlong_as_double(bits - ((long long)level << 52));
    return ldexp(box_edge, -level);
}

__device__ __forceinline__ int biased_exp(double v) {
    return (int)(((uint64_t)__double_as_longlong(v) >> 52) & 0x7ff);
}

// RN(c / m) for the rounded product c = RN(x * m) of a leaf (its centre-of-mass numerator over its
// mass), without a division: c / m = x - err / m with err = x * m - c, the rounding error of the
// product, exact in one FMA and at most half a unit in c's last place, so c / m lies within one
// unit of x and rounds to x or to its neighbour on err's side. Which of them is decided by
// comparing |err| 2^(53 - e(x)) with m (beyond half a unit; a tie goes to the even one), both
// positive normal numbers, as integers. The IEEE division remains for x a power of two (whose units
// differ on its two sides), subnormal or extreme values, and masses that are not positive.
__device__ __forceinline__ double leaf_quotient(double x, double m, double c) {
    const long long xb = __double_as_longlong(x);
    const int ex = biased_exp(x), em = biased_exp(m), ec = biased_exp(c);
    const bool m_ok = __double_as_longlong(m) > 0 && em >= 64 && em <= 2040;
    if (m_ok && (xb << 1) == 0) return c;  // 0 / m
    if (!m_ok || ex == 0 || ex == 0x7ff || (xb & 0xfffffffffffffll) == 0 || ec < 128 || ec > 2040)
        return __ddiv_rn(c, m);
    const long long err = __double_as_longlong(fma(x, m, -c));
    if ((err << 1) == 0) return x;
    const long long t = (err & 0x7fffffffffffffffll) + ((long long)(1023 + 53 - ex) << 52);
    const long long mb = __double_as_longlong(m);
    if (t < mb || (t == mb && (xb & 1) == 0)) return x;
    return __longlong_as_double((err ^ xb) < 0 ? xb + 1 : xb - 1);
}

// RN(cx / m), RN(cy / m), RN(cz / m) from one reciprocal (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990): y = RN(1 / m) by Newton steps from the
// hardware estimate (m's mantissa not all ones); q1 = q0 + r0 y is within one unit of the quotient
// and q1 + r1 y with the exact remainder r1 = c - m q1 rounds to it. The IEEE division remains
// outside a range in which every intermediate is normal, the quotients included (a subnormal one can
// lie halfway between two doubles, where the last step's own rounding decides).
__device__ __forceinline__ void exact_quotients(double cx, double cy, double cz, double m,
                                                double& qx, double& qy, double& qz) {
    const int em = biased_exp(m);
    const uint64_t mant = (uint64_t)__double_as_longlong(m) & 0xfffffffffffffull;
    auto fits = [&](double c) {
        const int e = biased_exp(c);
        return (e >= 300 && e <= 1700 && abs(e - em) < 960) ||
               ((__double_as_longlong(c) << 1) == 0);
    };
    if (em < 300 || em > 1700 || mant == 0xfffffffffffffull || !fits(cx) || !fits(cy) ||
        !fits(cz)) {
        qx = __ddiv_rn(cx, m);
        qy = __ddiv_rn(cy, m);
        qz = __ddiv_rn(cz, m);
        return;
    }
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(m));
    y = fma(y, fma(-m, y, 1.0), y);
    y = fma(y, fma(-m, y, 1.0), y);
    y = fma(y, fma(-m, y, 1.0), y);
    auto quotient = [&](double c) {
        double q = c * y;
        q = fma(fma(-m, q, c), y, q);
        const double r = fma(fma(-m, q, c), y, q);
        return (__double_as_longlong(c) << 1) == 0 ? (m > 0.0 ? c : -c) : r;
    };
    qx = quotient(cx);
    qy = quotient(cy);
    qz = quotient(cz);
}

// The FP32 edge^2 of a cell of the given level: (float)(edge * edge), both scaled exactly from the
// box's while they stay normal.
__device__ __forceinline__ float cell_edge2(double box_edge, double edge, float box_edge2,
                                            int level) {
    const int e = (int)((__float_as_uint(box_edge2) >> 23) & 0xff);
    if (e > 2 * level + 1 && e < 0xff && biased_exp(box_edge) > 600)
        return __uint_as_float(__float_as_uint(box_edge2) - ((uint32_t)(2 * level) << 23));
    return (float)(edge * edge);
}

// Terms beyond rec32's: the centre minus the box centre, exactly, as a triple-float and G*mass as a
// double-float (their first terms are rec32's: both round the same FP64 values).
__device__ __forceinline__ DfTerms df_terms_of(double cx, double cy, double cz, double ox,
                                               double oy, double oz, double gm, float gmf,
                                               bool massive) {
    DfTerms t{};
    if (massive) {
        float hx, hy, hz;
        tf_split_diff(cx, ox, hx, t.mx, t.lx);
        tf_split_diff(cy, oy, hy, t.my, t.ly);
        tf_split_diff(cz, oz, hz, t.mz, t.lz);
        t.gl = (float)(gm - (double)gmf);
    }
    return t;
}

// Fixed-point record of a node with centre (cx, cy, cz) and mass m.
__device__ __forceinline__ void write_fix(const ComArgs& A, uint32_t idx, double cx, double cy,
                                          double cz, double m) {
    const nbfix::FixRec r = nbfix::make_rec(cx, cy, cz, m, __double2hiint(A.box[11]));
    A.fix_hi[idx] = nbfix::FixHi{r.x2, r.y2, r.z2, r.mh, r.x1, r.y1, r.z1, r.e};
    A.fix_lo[idx] = make_uint4(r.x0, r.y0, r.z0, r.ml);
}

__device__ void write_records(const ComArgs& A, uint32_t idx, double cx, double cy, double cz,
                              double sm, double qsum, uint32_t count, int level, uint32_t skip,
                              uint32_t body) {
    const bool massive = (__double_as_longlong(sm) << 1) != 0;  // sm != 0
    const double edge = cell_edge64(A.box[6], level);
    const double ox = A.box[7], oy = A.box[8], oz = A.box[9];  // box centre
    // centre = sums / mass: the IEEE quotients when the FP64 records are built (the reference's
    // values, also behind the FP32 pre-test's proven margin), else from one reciprocal (the FP32
    // records round it); massless cells get a finite centre (never used)
    double rcx = 0.0, rcy = 0.0, rcz = 0.0, inv = 0.0;
    if (massive) {
        if (A.records & NB_REC_FP64) exact_quotients(cx, cy, cz, sm, rcx, rcy, rcz);
        // 1/M from the hardware estimate and one Newton step (~2^-44: ample for the FP32
        // centres and the spread)
        if (!(A.records & NB_REC_FP64) || (A.records & NB_REC_LEARNED)) {
            asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(inv) : "d"(sm));
            inv = inv * fma(-sm, inv, 2.0);
        }
        if (!(A.records & NB_REC_FP64)) {
            rcx = cx * inv;
            rcy = cy * inv;
            rcz = cz * inv;
        }
    }
    if (A.records & NB_REC_FP64) {
        NodeRec64 r;
        r.cx = rcx;
        r.cy = rcy;
        r.cz = rcz;
        r.mass = sm;
        r.edge = edge;
        r.skip = skip;
        r.body = body;
        A.rec64[idx] = r;
        write_fix(A, idx, rcx, rcy, rcz, sm);
    }
    NodeRec32 q;
    const double gx = rcx - ox, gy = rcy - oy, gz = rcz - oz;
    if (massive) {
        q.cx = (float)gx;
        q.cy = (float)gy;
        q.cz = (float)gz;
    } else {  // massless cell: far away, contributes exactly 0
        q.cx = q.cy = q.cz = 1e30f;
    }
    q.gm = (float)(A.G * sm);
    q.edge2 = cell_edge2(A.box[6], edge, __int_as_float(__double2loint(A.box[11])), level);
    q.skip = skip;
    q.body = body;
    q.level = (uint32_t)level;
    A.rec32[idx] = q;
    if (A.records & NB_REC_DF) {
        A.df_terms[idx] = df_terms_of(rcx, rcy, rcz, ox, oy, oz, A.G * sm, q.gm, massive);
    }
    if (A.records & NB_REC_LEARNED) {
        // spread^2 = sum m |x-o|^2 / M - |c-o|^2 (o = box centre, which keeps both terms small);
        // the spread is a feature of the learned policy, not a sum of the reference: 1/M from the
        // reciprocal, the root in FP32
        NodeAux x;
        x.spread_rel = 0.f;
        x.lg_gm = __log2f(fmaxf(q.gm, 1e-37f));
        if (massive) {
            const double s2 = qsum * inv - (gx * gx + gy * gy + gz * gz);
            const float e = (float)edge;
            if (e > 0.f) x.spread_rel = sqrtf((float)(s2 > 0 ? s2 : 0.0)) / e;
        }
        x.count = count;
        x.first = A.node_first_pos[idx];
        A.aux[idx] = x;
    }
}

// Sums of internal node `idx` from its children (the reference's octant order 0..7, FP64 adds:
// bit-identical to BarnesHutOctree.cpp:304-311), its records, and its child list rewritten as the
// compacted visit-order list the learned traversal reads (emit_kernel wrote it by visit rank).
// c0, c1: the cell's child list as emit_kernel wrote it (loaded by the caller, possibly earlier).
__device__ void sum_children(const ComArgs& A, uint32_t idx, bool records, uint4 c0, uint4 c1) {
    uint4* cl = reinterpret_cast<uint4*>(A.children + (size_t)idx * 8);
    const uint32_t vs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const bool learned = (A.records & NB_REC_LEARNED) != 0;
    // every child's sums requested before the first is used (one round trip, not eight)
    double cx[8], cy[8], cz[8], cm[8], cq[8];
    uint32_t cc[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) {  // the reference's octant order 0..7
        const uint32_t ch = vs[nb_visit_of_octant(o)];
        cx[o] = cy[o] = cz[o] = cm[o] = cq[o] = 0.0;
        cc[o] = 0;
        if (ch != NB_NONE) {
            cx[o] = __ldcg(&A.comx[ch]);
            cy[o] = __ldcg(&A.comy[ch]);
            cz[o] = __ldcg(&A.comz[ch]);
            cm[o] = __ldcg(&A.mass[ch]);
            if (learned) cq[o] = __ldcg(&A.q[ch]);
            cc[o] = __ldcg(&A.node_count[ch]);
        }
    }
    // the compacted visit-order child list the learned traversal reads
    uint32_t list[8];
    int nch = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        list[t] = NB_NONE;
        if (vs[t] != NB_NONE) list[nch++] = vs[t];
    }
    cl[0] = make_uint4(list[0], list[1], list[2], list[3]);
    cl[1] = make_uint4(list[4], list[5], list[6], list[7]);
    double sx = 0, sy = 0, sz = 0, sm = 0, sq = 0;
    uint32_t count = 0;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        if (vs[nb_visit_of_octant(o)] == NB_NONE) continue;  // absent children add nothing
        sx = __dadd_rn(sx, cx[o]);
        sy = __dadd_rn(sy, cy[o]);
        sz = __dadd_rn(sz, cz[o]);
        sm = __dadd_rn(sm, cm[o]);
        if (learned) sq += cq[o];
        count += cc[o];
    }
    A.comx[idx] = sx;
    A.comy[idx] = sy;
    A.comz[idx] = sz;
    A.mass[idx] = sm;
    if (learned) A.q[idx] = sq;
    A.node_count[idx] = count;
    if (records)
        write_records(A, idx, sx, sy, sz, sm, sq, count, A.node_level[idx], A.node_skip[idx],
                      NB_NONE);
}

// Records of internal node `idx` from its final sums (written earlier by sum_children).
__device__ void cell_records(const ComArgs& A, uint32_t idx) {
    const bool learned = (A.records & NB_REC_LEARNED) != 0;
    write_records(A, idx, __ldcg(&A.comx[idx]), __ldcg(&A.comy[idx]), __ldcg(&A.comz[idx]),
                  __ldcg(&A.mass[idx]), learned ? __ldcg(&A.q[idx]) : 0.0,
                  __ldcg(&A.node_count[idx]), A.node_level[idx], A.node_skip[idx], NB_NONE);
}

// Sums and records of the leaf `idx` (body b at sorted position p). A leaf's centre of mass is
// its body: the FP64 records keep the reference's quotient (c / m, mostly decided without a
// division by leaf_quotient), the FP32 records take the body position itself (within their own
// rounding of that quotient), and the spread of a single body is 0.
struct NodeSums {
    double x, y, z, m, q;
};

__device__ NodeSums leaf_sums(const ComArgs& A, uint32_t idx, uint32_t p, uint32_t b) {
    const double mb = A.m[b];
    const bool massive = (__double_as_longlong(mb) << 1) != 0;  // mb != 0
    const double bx = A.x[b], by = A.y[b], bz = A.z[b];
    const double cx = __dmul_rn(bx, mb), cy = __dmul_rn(by, mb), cz = __dmul_rn(bz, mb);
    A.comx[idx] = cx;
    A.comy[idx] = cy;
    A.comz[idx] = cz;
    A.mass[idx] = mb;
    A.node_count[idx] = 1;
    const int level = A.node_level[idx];
    const uint32_t skip = A.node_skip[idx];
    const double edge = cell_edge64(A.box[6], level);
    const double ox = A.box[7], oy = A.box[8], oz = A.box[9];
    const bool fp64 = (A.records & NB_REC_FP64) != 0;
    double rcx = bx, rcy = by, rcz = bz;
    if (fp64 && massive) {
        rcx = leaf_quotient(bx, mb, cx);
        rcy = leaf_quotient(by, mb, cy);
        rcz = leaf_quotient(bz, mb, cz);
    }
    if (fp64) {
        NodeRec64 r;
        r.cx = massive ? rcx : 0.0;
        r.cy = massive ? rcy : 0.0;
        r.cz = massive ? rcz : 0.0;
        r.mass = mb;
        r.edge = edge;
        r.skip = skip;
        r.body = b;
        A.rec64[idx] = r;
        write_fix(A, idx, rcx, rcy, rcz, mb);
    }
    const double gx = rcx - ox, gy = rcy - oy, gz = rcz - oz;
    NodeRec32 q;
    q.cx = massive ? (float)gx : 1e30f;  // a massless body: far away, contributes exactly 0
    q.cy = massive ? (float)gy : 1e30f;
    q.cz = massive ? (float)gz : 1e30f;
    q.gm = (float)(A.G * mb);
    q.edge2 = cell_edge2(A.box[6], edge, __int_as_float(__double2loint(A.box[11])), level);
    q.skip = skip;
    q.body = b;
    q.level = (uint32_t)level;
    A.rec32[idx] = q;
    if (A.records & NB_REC_DF) {
        A.df_terms[idx] = df_terms_of(rcx, rcy, rcz, ox, oy, oz, A.G * mb, q.gm, massive);
    }
    NodeSums sums{cx, cy, cz, mb, 0.0};
    if (A.records & NB_REC_LEARNED) {  // spread sums and the FP32 body copies of the policy
        const double rx = bx - ox, ry = by - oy, rz = bz - oz;
        sums.q = mb * (rx * rx + ry * ry + rz * rz);
        A.q[idx] = sums.q;
        const float hx = (float)rx, hy = (float)ry, hz = (float)rz;
        A.sorted4[p] = make_float4(hx, hy, hz, q.gm);
        A.sorted4lo[p] = make_float4((float)(rx - (double)hx), (float)(ry - (double)hy),
                                     (float)(rz - (double)hz), 0.f);
        NodeAux x;
        x.spread_rel = 0.f;
        x.count = 1;
        x.first = p;
        x.lg_gm = __log2f(fmaxf(q.gm, 1e-37f));
        A.aux[idx] = x;
    }
    return sums;
}

// Centre of mass and records, bottom-up, in chunks of CW consecutive sorted positions. The nodes
// starting in a chunk are the DFS indices [base[P], base[P + CW]); the ones that also end in it
// ("local": all leaves and most cells) are summed by the chunk's block. A cell that starts in a
// chunk and reaches past its end holds the chunk's last body and the next one, so there is at
// most one such cell per level: each chunk lists them (<= CM_LEVELS) for the next tier, whose
// blocks cover CM_FAN chunks each and sum the listed cells that end inside their span, passing
// the rest up again, until one block spans all bodies. Every sum has its children's sums final
// before it starts (kernel order, then levels deepest first within a block), so no thread waits
// on another, and the FP64 work is spread over all SMs at every tier.
//  * com_chunk_kernel: one block per chunk. Its leaves' sums go to shared memory (and, like all
//    sums and records, to global memory), the local cells are sorted by level, each thread keeps
//    its cells' children as slots of the shared sums, and the levels are summed from there; the
//    cells' records follow in one sweep (FP64 work with full warps: on this part an FP64 warp
//    instruction costs the FP64 pipe the same time however few of its lanes are active).
//    Bound: per level a barrier and a chain of FP64 additions (68 cycles each) in the reference's
//    order. Against a leaf kernel and level sums through L2 by blocks of 4,096 positions
//    (~1,200 cycles per level): 777 bodies 53 -> 35 us, 16,411 127 -> 63, 131,101 145 -> 104,
//    1,048,576 332 -> 309; with four lanes per cell, the cluster and the tiers from shared memory
//    25, 43, 72 and 242 (the whole phase).
//  * com_tier_kernel: one block per span of CM_FAN lower-tier chunks, same scheme on the listed
//    cells.
constexpr int CW_MIN = 256;                       // sorted positions per chunk, at least
constexpr int CM_LEVELS = 2 * NB_KEY_LEVELS + 1;  // node levels 0..42
constexpr int CM_FAN = 96;                        // lower-tier chunks per upper-tier chunk
constexpr int CM_TIER_MAX = CM_LEVELS * CM_FAN;   // listed cells one upper-tier block reads
constexpr int CM_TIERS = 5;                       // 256 * 96^4 > 2^27 bodies
constexpr int CC_THREADS = 512;                   // threads per block of the tier kernel

// Exclusive prefix of the level counts and the deepest level with a cell (-1: none), by warp 0.
__device__ __forceinline__ void level_offsets(const uint32_t* cnt, uint32_t* off, int* deepest) {
    const uint32_t lane = threadIdx.x;
    if (lane >= 32) return;
    uint32_t run = 0;
    int top = -1;
    for (int l0 = 0; l0 < CM_LEVELS; l0 += 32) {
        const int l = l0 + (int)lane;
        const uint32_t c = l < CM_LEVELS ? cnt[l] : 0u;
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += v;
        }
        if (l < CM_LEVELS) off[l] = run + incl - c;
        run += __shfl_sync(0xffffffffu, incl, 31);
        const uint32_t some = __ballot_sync(0xffffffffu, c != 0);
        if (some) top = l0 + 31 - __clz((int)some);
    }
    if (lane == 0) *deepest = top;
}

// The visit-order child list of a cell, compacted: as the learned traversal reads it.
__device__ __forceinline__ void compact_children(const ComArgs& A, uint32_t idx) {
    uint32_t* cl = A.children + (size_t)idx * 8;
    const uint4 c0 = reinterpret_cast<const uint4*>(cl)[0], c1 = reinterpret_cast<const uint4*>(cl)[1];
    const uint32_t vs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    uint32_t nch = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t)
        if (vs[t] != NB_NONE) cl[nch++] = vs[t];
    for (uint32_t t = nch; t < 8; ++t) cl[t] = NB_NONE;
}

// Sums the `nf` cells nodes[off[l] .. off[l] + cnt[l]) of each level l, deepest first, in global
// memory, then writes their records. Block-wide; smem arrays given by the caller.
__device__ void sum_by_level(const ComArgs& A, uint32_t nf, const uint32_t* nodes,
                             const uint32_t* cnt, const uint32_t* off) {
    // deepest level first; each thread's first cell of the next level has its child list loaded
    // before the barrier (a list only changes when its own cell is summed), so a level costs one
    // round trip to the children's sums instead of two
    const uint4 none4 = make_uint4(NB_NONE, NB_NONE, NB_NONE, NB_NONE);
    auto list_of = [&](uint32_t idx, uint4& c0, uint4& c1) {
        const uint4* cl = reinterpret_cast<const uint4*>(A.children + (size_t)idx * 8);
        c0 = __ldcg(cl);
        c1 = __ldcg(cl + 1);
    };
    int l = CM_LEVELS - 1;
    while (l >= 0 && cnt[l] == 0) --l;  // uniform across the block
    uint4 p0 = none4, p1 = none4;
    if (l >= 0 && threadIdx.x < cnt[l]) list_of(nodes[off[l] + threadIdx.x], p0, p1);
    while (l >= 0) {
        const uint32_t c = cnt[l];
        int next = l - 1;
        while (next >= 0 && cnt[next] == 0) --next;
        for (uint32_t k = threadIdx.x; k < c; k += blockDim.x) {
            const uint32_t idx = nodes[off[l] + k];
            uint4 c0 = p0, c1 = p1;
            if (k != threadIdx.x) list_of(idx, c0, c1);
            sum_children(A, idx, false, c0, c1);
        }
        if (next >= 0 && threadIdx.x < cnt[next]) list_of(nodes[off[next] + threadIdx.x], p0, p1);
        __syncthreads();
        l = next;
    }
    for (uint32_t k = threadIdx.x; k < nf; k += blockDim.x) cell_records(A, nodes[k]);
}

// 0.0 + v
__device__ __forceinline__ double plus_zero(double v) {
    const long long b = __double_as_longlong(v);
    return __longlong_as_double((b << 1) == 0 ? 0ll : b);
}

// Shared memory of com_chunk_kernel: the sums of the chunk's nodes (the spread sums only when the
// learned records are built).
template <int CW>
constexpr size_t chunk_smem_bytes(bool learned) {
    return (size_t)(2 * CW + CM_LEVELS) * ((learned ? 5 : 4) * sizeof(double));
}

// The CTAS blocks of a chunk (one, or a cluster) share its leaves and the records of its cells; the
// sums are kept and added in the first one's shared memory.
template <int CW, int CH_THREADS, int CTAS>
__device__ __forceinline__ void com_chunk(const ComArgs& A, uint2* up, uint32_t* up_count) {
    static_assert(CW == CH_THREADS, "one leaf and at most one local cell per thread");
    namespace cg = cooperative_groups;
    auto all_sync = [] {
        if constexpr (CTAS > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    auto first_of = [](auto* ptr) {  // the same object in the chunk's first block
        if constexpr (CTAS > 1) return cg::this_cluster().map_shared_rank(ptr, 0);
        else return ptr;
    };
    const uint32_t rank = CTAS > 1 ? blockIdx.x % CTAS : 0u, chunk = blockIdx.x / CTAS;
    constexpr int CH_NODES = 2 * CW + CM_LEVELS;  // nodes starting in a chunk, at most
    extern __shared__ __align__(16) unsigned char com_smem[];
    const bool learned = (A.records & NB_REC_LEARNED) != 0;
    double* sx = reinterpret_cast<double*>(com_smem);
    double* sy = sx + CH_NODES;
    double* sz = sy + CH_NODES;
    double* sm = sz + CH_NODES;
    double* sq = sm + CH_NODES;  // learned only
    __shared__ uint16_t found[CW], order[CW];  // local cells as slots: as found, by level
    __shared__ __align__(16) uint16_t kids[CW][8];  // a cell's children as slots, octant order
    __shared__ uint8_t flev[CW];
    __shared__ int deepest;
    __shared__ uint32_t cnt[CM_LEVELS], off[CM_LEVELS], fill[CM_LEVELS];
    __shared__ uint32_t n_found, n_up;
    uint32_t nf = 0, my = 0, nkids = 0;
    bool cell = false;
    const uint32_t tid = threadIdx.x, P = chunk * CW;
    nb_grid_wait();
    const uint32_t Pend = min(P + (uint32_t)CW, A.n);
    const uint32_t d0 = A.base[P], d1 = A.base[Pend];
    if (tid < CM_LEVELS) cnt[tid] = fill[tid] = 0;
    if (tid == 0) n_found = n_up = 0;
    if (d1 - d0 > (uint32_t)CH_NODES) {  // a consistent tree never gets here
        if (tid == 0 && rank == 0) {
            atomicOr(A.err, NB_DEVERR_DEPTH);
            up_count[chunk] = 0;
        }
        return;
    }
    all_sync();  // the first block's memory is there
    if (const uint32_t p = P + tid * CTAS + rank; p < Pend) {
        const uint32_t idx = A.base[p] + __popcll(A.mask[p]), k = idx - d0;
        const NodeSums s = leaf_sums(A, idx, p, A.ids[p]);
        first_of(sx)[k] = s.x;
        first_of(sy)[k] = s.y;
        first_of(sz)[k] = s.z;
        first_of(sm)[k] = s.m;
        if (learned) first_of(sq)[k] = s.q;
    }
    if constexpr (CTAS > 1) all_sync();
    if (rank == 0) {
        for (uint32_t idx = d0 + tid; idx < d1; idx += CH_THREADS) {
            if (A.node_body[idx] != NB_NONE) continue;  // a leaf
            const int l = min((int)A.node_level[idx], CM_LEVELS - 1);
            if (A.node_last[idx] >= Pend) {  // reaches past the chunk: for the next tier
                const uint32_t g = atomicAdd(&n_up, 1u);
                if (g < (uint32_t)CM_LEVELS)
                    up[(size_t)chunk * CM_LEVELS + g] = make_uint2(idx, (uint32_t)l);
                else
                    atomicOr(A.err, NB_DEVERR_DEPTH);  // more than one per level: inconsistent
                continue;
            }
            const uint32_t slot = atomicAdd(&n_found, 1u);
            if (slot < (uint32_t)CW) {
                found[slot] = (uint16_t)(idx - d0);
                flev[slot] = (uint8_t)l;
                atomicAdd(&cnt[l], 1u);
            } else {
                atomicOr(A.err, NB_DEVERR_DEPTH);  // a consistent tree never gets here
            }
        }
        __syncthreads();
        nf = min(n_found, (uint32_t)CW);
        if (tid == 0) n_found = nf;  // for the other blocks
        if (tid == 0) up_count[chunk] = min(n_up, (uint32_t)CM_LEVELS);
        level_offsets(cnt, off, &deepest);
        __syncthreads();
        for (uint32_t k = tid; k < nf; k += CH_THREADS) {
            const uint32_t l = flev[k];
            order[off[l] + atomicAdd(&fill[l], 1u)] = found[k];
        }
        __syncthreads();
        // this thread's cell: its children in octant order as slots, and the compacted visit-order
        // child list the learned traversal reads
        cell = tid < nf;
        my = cell ? order[tid] : 0u;
        if (cell) {
            uint32_t* cl = A.children + (size_t)(d0 + my) * 8;
            const uint4 c0 = reinterpret_cast<const uint4*>(cl)[0],
                        c1 = reinterpret_cast<const uint4*>(cl)[1];
            const uint32_t vs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
            uint32_t nch = 0;
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (vs[t] != NB_NONE) cl[nch++] = vs[t];
            for (uint32_t t = nch; t < 8; ++t) cl[t] = NB_NONE;
#pragma unroll
            for (int o = 0; o < 8; ++o) {  // the reference's octant order 0..7
                const uint32_t ch = vs[nb_visit_of_octant(o)];
                if (ch != NB_NONE)
                    kids[tid][nkids++] = (uint16_t)min(ch - d0, (uint32_t)CH_NODES - 1);
            }
        }
        // deepest level first, four lanes per cell (x, y, z and mass; the first one the spread
        // too), a cell's children read before the adds: a thread per cell with its children one
        // after the other took 39 us instead of 31 at 1,024 bodies, 264 instead of 242 at 1,048,576
        // (the whole phase)
        for (uint32_t t = nkids; t < 8; ++t) kids[tid][t] = 0xffff;
        __syncthreads();
        for (int l = deepest; l >= 0; --l) {
            const uint32_t c = cnt[l], o0 = off[l];
            if (c == 0) continue;  // uniform across the block
            for (uint32_t pos = o0 + (tid >> 2); pos < o0 + c; pos += CH_THREADS / 4) {
                const uint4 kk = *reinterpret_cast<const uint4*>(kids[pos]);
                const uint32_t kw[4] = {kk.x, kk.y, kk.z, kk.w};
                auto add_up = [&](double* sv) {
                    double v[8];
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const uint32_t k = (kw[t >> 1] >> (16 * (t & 1))) & 0xffffu;
                        v[t] = sv[min(k, (uint32_t)CH_NODES - 1)];  // unused where there is no child
                    }
                    double sum = plus_zero(v[0]);  // 0.0 + v[0]
#pragma unroll
                    for (int t = 1; t < 8; ++t) {
                        if (((kw[t >> 1] >> (16 * (t & 1))) & 0xffffu) == 0xffffu) break;
                        sum = __dadd_rn(sum, v[t]);
                    }
                    sv[order[pos]] = sum;
                };
                add_up(sx + (tid & 3) * CH_NODES);
                if (learned && (tid & 3) == 0) add_up(sq);
            }
            __syncthreads();
        }
    }
    if constexpr (CTAS > 1) {
        all_sync();  // every sum is final
        nf = *first_of(&n_found);
        cell = tid * CTAS + rank < nf;
        my = cell ? first_of(order)[tid * CTAS + rank] : 0u;
    }
    if (cell) {
        const uint32_t idx = d0 + my;
        const double cx = first_of(sx)[my], cy = first_of(sy)[my], cz = first_of(sz)[my],
                     cm = first_of(sm)[my], cq = learned ? first_of(sq)[my] : 0.0;
        A.comx[idx] = cx;
        A.comy[idx] = cy;
        A.comz[idx] = cz;
        A.mass[idx] = cm;
        if (learned) A.q[idx] = cq;
        const uint32_t count = A.node_last[idx] - A.node_first[idx] + 1;
        A.node_count[idx] = count;
        write_records(A, idx, cx, cy, cz, cm, cq, count, A.node_level[idx], A.node_skip[idx], NB_NONE);
    }
    if constexpr (CTAS > 1) all_sync();  // the first block's memory stays until all have read it
}

template <int CW, int CH_THREADS>
__global__ void __launch_bounds__(CH_THREADS, 1024 / CH_THREADS)
com_chunk_kernel(ComArgs A, uint2* up, uint32_t* up_count) {
    com_chunk<CW, CH_THREADS, 1>(A, up, up_count);
}

// The whole of a system of 513 to CL_N bodies as one chunk of a cluster. In one block the leaves
// and the cells' records took 33,000 of 63,000 cycles at 777 bodies (one SM's FP64 pipe); the
// cluster takes 5 to 8 us off at 777 to 1,024 bodies, nothing at 500, and costs 3 at 100.
constexpr int CL_N = 1024, CL_CTAS = 8;
__global__ void __cluster_dims__(CL_CTAS, 1, 1) __launch_bounds__(CL_N, 1)
com_cluster_kernel(ComArgs A, uint2* up, uint32_t* up_count) {
    com_chunk<CL_N, CL_N, CL_CTAS>(A, up, up_count);
}

// Tier of `span` sorted positions per block: the cells listed by the CM_FAN lower-tier chunks of
// the span (in[c * CM_LEVELS + k], k < in_count[c]) that end inside it are summed here; the others
// go to up[] for the next tier (up == nullptr: the last tier, whose single block spans all bodies).
// Bound by latency: a block has a few hundred cells over 8 to 12 levels and a level waits for the
// one below. Up to CM_KEPT cells therefore sum from shared memory: all children outside the tier,
// which are final, are read ahead of the first level, the sums of the tier's own cells stay in
// shared memory (tier_slot finds a child's place in the block's list; what it names is checked, so
// that whatever an earlier launch left there does not matter), and four lanes take a cell's four
// components. With the children's sums read from global memory level by level, as for more cells
// than that, a level took 5,300 cycles and the kernel 66,000 at 16,411 bodies (9 levels, 201
// cells); this way 1,300 and 35,000: children packed to the front and read without branches (2,000
// a level otherwise), the records' other inputs requested before the levels.
constexpr int CM_KEPT = 512;
constexpr size_t tier_smem_bytes(bool learned) {
    return (size_t)CM_TIER_MAX * sizeof(uint32_t) +
           (size_t)CM_KEPT * ((learned ? 5 : 4) * 9 * sizeof(double) + 8 * sizeof(uint16_t));
}
constexpr uint32_t KID_NONE = 0xffff, KID_OUTSIDE = 0xfffe;  // else a place in the tier's list

__global__ void __launch_bounds__(CC_THREADS)
com_tier_kernel(ComArgs A, uint32_t span, const uint2* in,
                const uint32_t* in_count, uint32_t in_chunks, uint2* up,
                uint32_t* up_count) {
    extern __shared__ __align__(16) unsigned char com_smem[];
    const bool learned = (A.records & NB_REC_LEARNED) != 0;
    const int comps = learned ? 5 : 4;
    uint16_t* kid = reinterpret_cast<uint16_t*>(com_smem);             // [CM_KEPT][8], octant order
    double* kept = reinterpret_cast<double*>(kid + 8 * CM_KEPT);       // [comps][CM_KEPT]
    double* val = kept + comps * CM_KEPT;                              // [comps][CM_KEPT][8]
    uint32_t* nodes = reinterpret_cast<uint32_t*>(val + comps * CM_KEPT * 8);  // [CM_TIER_MAX]
    // the cells as found, only until they are in nodes[] by level
    uint32_t* found = reinterpret_cast<uint32_t*>(val);
    uint8_t* flev = reinterpret_cast<uint8_t*>(found + CM_TIER_MAX);
    static_assert((size_t)CM_TIER_MAX * 5 <= (size_t)CM_KEPT * 4 * 8 * sizeof(double), "found, flev");
    __shared__ uint32_t cnt[CM_LEVELS], off[CM_LEVELS], fill[CM_LEVELS], first[CM_FAN + 1];
    __shared__ uint32_t n_found, n_up;
    nb_grid_wait();
    const uint32_t tid = threadIdx.x, P = blockIdx.x * span;
    if (P >= A.n) return;
    const uint32_t Pend = (uint32_t)min((uint64_t)P + span, (uint64_t)A.n);
    if (tid < CM_LEVELS) cnt[tid] = fill[tid] = 0;
    if (tid == 0) n_found = n_up = 0;
    const uint32_t c0 = blockIdx.x * CM_FAN, chunks = min((uint32_t)CM_FAN, in_chunks - c0);
    if (tid < 32) {  // the chunks' entries, one after the other
        uint32_t run = 0;
        for (uint32_t b = 0; b < CM_FAN; b += 32) {
            const uint32_t c = b + tid < chunks ? in_count[c0 + b + tid] : 0u;
            uint32_t incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)tid >= o) incl += v;
            }
            first[b + tid] = run + incl - c;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (tid == 0) first[CM_FAN] = run;
    }
    __syncthreads();
    for (uint32_t e = tid; e < min(first[CM_FAN], (uint32_t)CM_TIER_MAX); e += CC_THREADS) {
        uint32_t lo = 0, hi = CM_FAN;  // first[lo] <= e < first[hi]
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (first[mid] <= e) lo = mid; else hi = mid;
        }
        const uint2 g = in[(size_t)(c0 + lo) * CM_LEVELS + (e - first[lo])];
        if (up != nullptr && A.node_last[g.x] >= Pend) {
            const uint32_t u = atomicAdd(&n_up, 1u);
            if (u < (uint32_t)CM_LEVELS) up[(size_t)blockIdx.x * CM_LEVELS + u] = g;
            else atomicOr(A.err, NB_DEVERR_DEPTH);
            continue;
        }
        atomicAdd(&cnt[g.y], 1u);
        const uint32_t slot = atomicAdd(&n_found, 1u);  // < CM_TIER_MAX: one per entry
        found[slot] = g.x;
        flev[slot] = (uint8_t)g.y;
    }
    __syncthreads();
    const uint32_t nf = n_found;
    if (tid == 0 && up_count != nullptr) up_count[blockIdx.x] = min(n_up, (uint32_t)CM_LEVELS);
    __shared__ int deepest;
    level_offsets(cnt, off, &deepest);
    __syncthreads();
    for (uint32_t k = tid; k < nf; k += CC_THREADS) {
        const uint32_t l = flev[k], idx = found[k], at = off[l] + atomicAdd(&fill[l], 1u);
        nodes[at] = idx;
        A.tier_slot[idx] = at;
    }
    __syncthreads();
    if (nf > (uint32_t)CM_KEPT) {
        sum_by_level(A, nf, nodes, cnt, off);
        return;
    }
    // the children: their places in the list, or their sums
    constexpr int AHEAD = 4;
    double* const sums[5] = {A.comx, A.comy, A.comz, A.mass, A.q};
    // a cell's eight children by eight neighbouring lanes, the ones that exist packed to the front
    for (uint32_t e0 = tid; e0 - (tid & 31) < nf * 8; e0 += CC_THREADS * AHEAD) {
        uint32_t ch[AHEAD], at[AHEAD];
        double v[AHEAD][5];
#pragma unroll
        for (int r = 0; r < AHEAD; ++r) {
            const uint32_t e = e0 + r * CC_THREADS;
            ch[r] = NB_NONE;
            if (e < nf * 8) ch[r] = A.children[(size_t)nodes[e >> 3] * 8 + nb_visit_of_octant(e & 7)];
        }
#pragma unroll
        for (int r = 0; r < AHEAD; ++r) {
            if (ch[r] == NB_NONE) continue;
            at[r] = A.tier_slot[ch[r]];
#pragma unroll
            for (int c = 0; c < 4; ++c) v[r][c] = __ldcg(sums[c] + ch[r]);
            if (learned) v[r][4] = __ldcg(sums[4] + ch[r]);
        }
#pragma unroll
        for (int r = 0; r < AHEAD; ++r) {
            const uint32_t e = e0 + r * CC_THREADS;
            const uint32_t group = tid & 24u;  // the cell's first lane
            const uint32_t have = (__ballot_sync(0xffffffffu, ch[r] != NB_NONE) >> group) & 0xffu;
            if (e >= nf * 8) continue;
            if ((e & 7) >= (uint32_t)__popc(have)) kid[e] = (uint16_t)KID_NONE;
            if (ch[r] == NB_NONE) continue;
            const uint32_t to = (e & ~7u) + __popc(have & ((1u << (e & 7)) - 1u));
            if (at[r] < nf && nodes[at[r]] == ch[r]) {
                kid[to] = (uint16_t)at[r];
            } else {
                kid[to] = (uint16_t)KID_OUTSIDE;
#pragma unroll
                for (int c = 0; c < 4; ++c) val[c * (CM_KEPT * 8) + to] = v[r][c];
                if (learned) val[4 * (CM_KEPT * 8) + to] = v[r][4];
            }
        }
    }
    __syncthreads();
    auto add_up = [&](uint32_t pos, int comp) {
        const uint4 kk = *reinterpret_cast<const uint4*>(kid + 8 * pos);
        const uint32_t kw[4] = {kk.x, kk.y, kk.z, kk.w};
        const double* const kc = kept + comp * CM_KEPT;
        const double* const vc = val + comp * (CM_KEPT * 8) + 8 * pos;
        uint32_t k[8];
        double v[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            k[o] = (kw[o >> 1] >> (16 * (o & 1))) & 0xffffu;
            const double* const from = k[o] < (uint32_t)CM_KEPT ? kc + k[o] : vc + o;
            v[o] = *from;  // unused where there is no child
        }
        double sum = 0.0;
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            if (k[o] == KID_NONE) break;  // absent children add nothing
            sum = __dadd_rn(sum, v[o]);
        }
        kept[comp * CM_KEPT + pos] = sum;
    };
    // what this thread's record needs besides the sums, requested before the levels
    static_assert(CM_KEPT <= CC_THREADS, "one record per thread");
    uint32_t idx = NB_NONE, pos0 = 0, pos1 = 0, skip = 0, level = 0;
    if (tid < nf) {
        idx = nodes[tid];
        pos0 = A.node_first[idx];
        pos1 = A.node_last[idx];
        skip = A.node_skip[idx];
        level = A.node_level[idx];
    }
    for (int l = deepest; l >= 0; --l) {
        const uint32_t c = cnt[l], o0 = off[l];
        if (c == 0) continue;  // uniform across the block
        for (uint32_t k = tid >> 2; k < c; k += CC_THREADS / 4) {
            add_up(o0 + k, (int)(tid & 3));
            if (learned && (tid & 3) == 0) add_up(o0 + k, 4);
        }
        __syncthreads();
    }
    if (idx != NB_NONE) {
        const uint32_t k = tid, count = pos1 - pos0 + 1;
        const double sx = kept[k], sy = kept[CM_KEPT + k], sz = kept[2 * CM_KEPT + k],
                     sm = kept[3 * CM_KEPT + k], sq = learned ? kept[4 * CM_KEPT + k] : 0.0;
        A.comx[idx] = sx;
        A.comy[idx] = sy;
        A.comz[idx] = sz;
        A.mass[idx] = sm;
        if (learned) A.q[idx] = sq;
        A.node_count[idx] = count;
        compact_children(A, idx);
        write_records(A, idx, sx, sy, sz, sm, sq, count, (int)level, skip, NB_NONE);
    }
}

// The kernels whose dynamic shared memory is above the default limit (before any capture of a
// build), once per device: five calls, 1.6 us in all.
template <typename K>
nb_status allow_smem(K kernel, size_t bytes) {
    NB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)bytes));
    return NB_OK;
}
nb_status build_prepare() {
    static std::atomic<bool> done[64];
    int dev = 0;
    NB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && done[dev]) return NB_OK;
    NB_TRY(allow_smem(build_small_kernel<1024, 1024>, small_smem_bytes<1024>()));
    NB_TRY(allow_smem(build_small_kernel<SB_MAX_N, 1024>, small_smem_bytes<SB_MAX_N>()));
    NB_TRY(allow_smem(com_tier_kernel, tier_smem_bytes(true)));
    NB_TRY(allow_smem(com_chunk_kernel<512, 512>, chunk_smem_bytes<512>(true)));
    NB_TRY(allow_smem(com_cluster_kernel, chunk_smem_bytes<CL_N>(true)));
    if (dev >= 0 && dev < 64) done[dev] = true;
    return NB_OK;
}

// ---------------------------------------------------------------------------------------------
// allocation
// ---------------------------------------------------------------------------------------------
struct Carver {
    char* base = nullptr;
    size_t off = 0;
    template <typename T>
    T* take(size_t count) {
        off = (off + 255) & ~(size_t)255;
        T* p = (T*)(base + off);
        off += count * sizeof(T);
        return p;
    }
};

void carve(nb_bh_tree* t, Carver& c) {
    const size_t n = t->n_max, cap = t->node_cap;
    t->box = c.take<double>(BOX_WORDS);
    t->info = c.take<uint32_t>(16);
    t->work = c.take<uint32_t>(16);
    t->sched = c.take<uint32_t>(32);
    t->group_cost = c.take<uint32_t>(n / 32 + 1);
    t->group_first = c.take<uint32_t>(n / 32 + 1);
    t->group_skip = c.take<uint32_t>(n / 1024 + 1);
    t->walk_len = c.take<uint32_t>(n);
    t->walk_ids = c.take<uint32_t>(n);
    t->walk_cost = c.take<uint32_t>((n + 31) / 32);
    t->key0 = c.take<uint64_t>(n);
    t->key1 = c.take<uint64_t>(n);
    t->key_alt = c.take<uint64_t>(n);
    t->ids = c.take<uint32_t>(n);
    t->ids_alt = c.take<uint32_t>(n);
    t->split_level = c.take<uint8_t>(n);
    t->split_start = c.take<uint32_t>(n);
    t->split_end = c.take<uint32_t>(n);
    t->mask = c.take<uint64_t>(n);
    t->base = c.take<uint32_t>(n + 1);
    t->sort_temp = c.take<char>(nb::radix_temp_bytes((uint32_t)n));
    t->scan_temp = c.take<uint32_t>(nb::scan_temp_bytes((uint32_t)n + 1) / 4 + 16);
    t->node_level = c.take<uint8_t>(cap);
    t->node_first = c.take<uint32_t>(cap);
    t->node_last = c.take<uint32_t>(cap);
    t->node_skip = c.take<uint32_t>(cap);
    t->node_body = c.take<uint32_t>(cap);
    t->tier_slot = c.take<uint32_t>(cap);
    t->node_count = c.take<uint32_t>(cap);
    t->node_comx = c.take<double>(cap);
    t->node_comy = c.take<double>(cap);
    t->node_comz = c.take<double>(cap);
    t->node_mass = c.take<double>(cap);
    t->rec64 = c.take<NodeRec64>(cap);
    t->fix_hi = c.take<nbfix::FixHi>(cap);
    t->fix_lo = c.take<uint4>(cap);
    t->rec32 = c.take<NodeRec32>(cap);
    t->df_terms = c.take<DfTerms>(cap);
    t->node_q = c.take<double>(cap);
    t->aux = c.take<NodeAux>(cap);
    t->children = c.take<uint32_t>(cap * 8);
    t->sorted4 = c.take<float4>(n);
    t->sorted4lo = c.take<float4>(n);
    // per tier, CM_LEVELS listed cells and a count per chunk (two lists, used in turn)
    const size_t chunks = (n + CW_MIN - 1) / CW_MIN;
    for (int k = 0; k < 2; ++k) {
        t->tier_cells[k] = c.take<uint2>(chunks * CM_LEVELS);
        t->tier_count[k] = c.take<uint32_t>(chunks);
    }
}

}  // namespace

extern "C" {

nb_status nb_bh_params_default(nb_bh_params* out) {
    if (!out) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_params_default: null pointer");
    out->theta = 1.05;  // Configuration.cpp:18
    out->storage_size_param = 16;
    out->stack_size_param = 16;
    out->max_build_level = 7;
    out->sort_bodies = 1;
    return NB_OK;
}

nb_status nb_bh_tree_create(nb_ctx* ctx, uint32_t n_max, const nb_bh_params* params,
                            nb_bh_tree** out) {
    NB_CHECK_CTX(ctx);
    if (!out) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_tree_create: null output");
    if (n_max == 0 || n_max > (1u << 27))
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_tree_create: n_max = %u out of range", n_max);
    NB_TRY(nb::radix_prepare());  // before any capture of a build
    NB_TRY(build_prepare());
    nb_bh_tree* t = new nb_bh_tree();
    t->n_max = n_max;
    t->node_cap = 2 * n_max;
    t->device = ctx->device;
    if (params) {
        t->params = *params;
    } else {
        nb_bh_params_default(&t->params);
    }
    Carver sizing;
    carve(t, sizing);
    void* mem = nullptr;
    cudaError_t e = cudaMalloc(&mem, sizing.off + 256);
    if (e != cudaSuccess) {
        delete t;
        return nb::cuda_error(e, "nb_bh_tree_create");
    }
    Carver real;
    real.base = (char*)mem;
    carve(t, real);
    e = cudaMemset(t->sched, 0, 32 * sizeof(uint32_t));  // no group order yet
    if (e != cudaSuccess) {
        cudaFree(mem);
        delete t;
        return nb::cuda_error(e, "nb_bh_tree_create");
    }
    // the carve order puts box first: its address is the allocation base (freed in destroy)
    *out = t;
    return NB_OK;
}

nb_status nb_bh_tree_destroy(nb_bh_tree* t) {
    if (!t) return NB_OK;
    if (t->phase_timing)
        for (auto& e : t->phase_ev) cudaEventDestroy(e);
    if (t->box) cudaFree(t->box);
    delete t;
    return NB_OK;
}

nb_status nb_bh_set_phase_timing(nb_bh_tree* t, int enable) {
    if (!t) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_set_phase_timing: null tree");
    NB_CUDA_TRY(cudaSetDevice(t->device));
    if (enable && !t->phase_timing) {
        for (auto& e : t->phase_ev) NB_CUDA_TRY(cudaEventCreate(&e));
    } else if (!enable && t->phase_timing) {
        for (auto& e : t->phase_ev) {
            cudaEventDestroy(e);
            e = nullptr;
        }
    }
    t->phase_timing = enable != 0;
    return NB_OK;
}

nb_status nb_bh_build_phase_ms(nb_bh_tree* t, float* ms) {
    if (!t || !ms) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_build_phase_ms: null argument");
    if (!t->phase_timing)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_build_phase_ms: phase timing is off");
    if (!t->built) return nb::set_error(NB_ERR_NOT_BUILT, "nb_bh_build_phase_ms: tree not built");
    NB_CUDA_TRY(cudaEventSynchronize(t->phase_ev[5]));
    for (int k = 0; k < 5; ++k)
        NB_CUDA_TRY(cudaEventElapsedTime(&ms[k], t->phase_ev[k], t->phase_ev[k + 1]));
    return NB_OK;
}

nb_status nb_bh_tree_set_theta(nb_bh_tree* t, double theta) {
    if (!t) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_tree_set_theta: null tree");
    if (!(theta >= 0)) return nb::set_error(NB_ERR_INVALID_ARG, "theta must be >= 0");
    t->params.theta = theta;
    return NB_OK;
}

nb_status nb_bh_build(nb_ctx* ctx, nb_bh_tree* t, const double* m, const double* x,
                      const double* y, const double* z, uint32_t n, double G,
                      nb_stream_t stream_) {
    NB_CHECK_CTX(ctx);
    if (!t) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_build: null tree");
    if (!m || !x || !y || !z) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_build: null array");
    if (n == 0 || n > t->n_max)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_build: n = %u (tree capacity %u)", n, t->n_max);
    cudaStream_t s = (cudaStream_t)stream_;
    t->built = false;
    t->n = n;
    t->G = G;
    const int grid = nb::ceil_div(n, BH_THREADS);
    auto mark = [&](int phase) -> nb_status {
        if (t->phase_timing) NB_CUDA_TRY(cudaEventRecord(t->phase_ev[phase], s));
        return NB_OK;
    };
    NB_TRY(mark(0));
    const bool quantized = (t->records & NB_BUILD_QUANTIZED_KEYS) != 0;
    const NodeTable T{t->node_level, t->node_first, t->node_last, t->node_skip,
                      t->node_body,  t->info,       t->children};
    if (n <= SB_MAX_N) {  // one block; its whole time counts as the cells phase
        for (int phase = 1; phase <= 3; ++phase) NB_TRY(mark(phase));
        auto go = [&](auto kernel, uint32_t threads, size_t smem) {
            return nb::launch_after(kernel, 1, threads, smem, s, x, y, z, n, t->box, t->key0,
                                    t->key1, t->ids, (unsigned long long*)t->mask, t->base, T,
                                    ctx->dev_error, quantized ? 1 : 0);
        };
        if (n <= 512)
            NB_CUDA_TRY(go(build_small_kernel<512, 512>, 512, small_smem_bytes<512>()));
        else if (n <= 1024)
            NB_CUDA_TRY(go(build_small_kernel<1024, 1024>, 1024, small_smem_bytes<1024>()));
        else
            NB_CUDA_TRY(go(build_small_kernel<SB_MAX_N, 1024>, 1024, small_smem_bytes<SB_MAX_N>()));
    } else {
        NB_TRY(nb::launch_aabb(ctx, x, y, z, n, t->box, s));
        NB_TRY(mark(1));
        const BuildZero Z{(uint4*)t->sort_temp, (uint32_t)(nb::radix_zero_bytes(n) / 16), t->key1,
                          (unsigned long long*)t->mask};
        if (quantized) {
            NB_CUDA_TRY(nb::launch_after(keys_quantized_kernel, grid, BH_THREADS, 0, s, x, y, z, n,
                                         t->box, t->key0, t->ids, Z));
        } else {
            NB_CUDA_TRY(nb::launch_after(keys_kernel, grid, BH_THREADS, 0, s, x, y, z, n, t->box,
                                         t->key0, t->ids, Z));
        }
        NB_TRY(mark(2));
        int in_alt = 0;
        NB_TRY(nb::radix_sort_pairs(t->key0, t->ids, t->key_alt, t->ids_alt, n, 0, 3 * NB_KEY_LEVELS,
                                    t->sort_temp, ctx->dev_error, s, &in_alt, NB_WAIT_LIMIT_DEFAULT, 0,
                                    true));
        if (in_alt) {  // an odd number of passes leaves the result in the alternate buffers
            NB_CUDA_TRY(cudaMemcpyAsync(t->key0, t->key_alt, (size_t)n * 8, cudaMemcpyDeviceToDevice, s));
            NB_CUDA_TRY(cudaMemcpyAsync(t->ids, t->ids_alt, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
        }
        NB_TRY(mark(3));
        NB_CUDA_TRY(nb::launch_after(runs_fixup_kernel, grid, BH_THREADS, 0, s, x, y, z, n, t->box,
                                     t->key0, t->key1, t->ids, ctx->dev_error, quantized ? 1 : 0));
        NB_CUDA_TRY(nb::launch_after(splits_kernel, grid, BH_THREADS, 0, s, t->key0, t->key1, n,
                                     t->split_level, t->split_start, t->split_end,
                                     (unsigned long long*)t->mask, t->children, ctx->dev_error));
        NB_TRY(nb::node_offsets((const unsigned long long*)t->mask, t->base, n, t->scan_temp, s));
        NB_CUDA_TRY(nb::launch_after(emit_kernel, grid, BH_THREADS, 0, s, n, t->ids, t->split_level,
                                     t->split_start, t->split_end,
                                     (const unsigned long long*)t->mask, t->base, t->key0, t->key1,
                                     T));
    }
    NB_TRY(mark(4));
    ComArgs A;
    A.n = n;
    A.records = t->records;
    A.m = m;
    A.x = x;
    A.y = y;
    A.z = z;
    A.box = t->box;
    A.G = G;
    A.key0 = t->key0;
    A.key1 = t->key1;
    A.ids = t->ids;
    A.mask = (const unsigned long long*)t->mask;
    A.base = t->base;
    A.node_level = t->node_level;
    A.node_first = t->node_first;
    A.node_last = t->node_last;
    A.node_skip = t->node_skip;
    A.err = ctx->dev_error;
    A.node_body = t->node_body;
    A.tier_slot = t->tier_slot;
    A.node_count = t->node_count;
    A.comx = t->node_comx;
    A.comy = t->node_comy;
    A.comz = t->node_comz;
    A.mass = t->node_mass;
    A.rec64 = t->rec64;
    A.fix_hi = t->fix_hi;
    A.fix_lo = t->fix_lo;
    A.rec32 = t->rec32;
    A.df_terms = t->df_terms;
    A.q = t->node_q;
    A.aux = t->aux;
    A.node_first_pos = t->node_first;
    A.children = t->children;
    A.sorted4 = t->sorted4;
    A.sorted4lo = t->sorted4lo;
    {
        const bool learned = (t->records & NB_REC_LEARNED) != 0;
        // one chunk for the smallest systems (no tier pass: 4 chunks and a tier cost 9 us more at
        // 300 bodies and the same at 777), else 256 positions per chunk
        const uint32_t cw = n <= 512 ? 512 : n <= (uint32_t)CL_N ? CL_N : 256;
        uint32_t chunks = (uint32_t)nb::ceil_div(n, cw);
        auto go = [&](auto kernel, uint32_t blocks, size_t smem) {
            return nb::launch_after(kernel, blocks, cw, smem, s, A, t->tier_cells[0],
                                    t->tier_count[0]);
        };
        NB_CUDA_TRY(cw == CL_N ? go(com_cluster_kernel, CL_CTAS, chunk_smem_bytes<CL_N>(learned))
                    : cw == 512 ? go(com_chunk_kernel<512, 512>, 1, chunk_smem_bytes<512>(learned))
                                : go(com_chunk_kernel<256, 256>, chunks,
                                     chunk_smem_bytes<256>(learned)));
        uint64_t span = cw;
        int in = 0;
        for (int tier = 1; tier <= CM_TIERS && chunks > 1; ++tier) {
            span *= CM_FAN;
            const uint32_t blocks = (uint32_t)((n + span - 1) / span);
            const bool last = blocks == 1;
            NB_CUDA_TRY(nb::launch_after(
                com_tier_kernel, blocks, CC_THREADS, tier_smem_bytes(learned), s, A,
                (uint32_t)std::min<uint64_t>(span, 0xffffffffu), t->tier_cells[in],
                t->tier_count[in], chunks, last ? nullptr : t->tier_cells[1 - in],
                last ? nullptr : t->tier_count[1 - in]));
            if (last) break;
            chunks = blocks;
            in = 1 - in;
        }
    }
    NB_TRY(mark(5));
    t->built = true;
    t->built_records = t->records;
    return NB_OK;
}

nb_status nb_bh_set_records(nb_bh_tree* t, unsigned int mask) {
    if (!t) return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_set_records: null tree");
    if (mask & ~(NB_REC_ALL | NB_BUILD_QUANTIZED_KEYS))
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_bh_set_records: unknown bits 0x%x", mask);
    t->records = mask;
    return NB_OK;
}

}  // extern "C"
