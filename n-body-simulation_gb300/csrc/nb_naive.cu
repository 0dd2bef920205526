// nb_naive.cu -- naive all-pairs acceleration (NaiveAlgorithm.cpp:262-482 semantics).
//
// Three arithmetic modes:
//  * NB_F64_IEEE: one thread per target body walks all sources j = 0..N-1 in order, every
//    operation separately rounded in the reference's order (r^2 summed left to right, den^3 as
//    (den*den)*den, 1/sqrt for rsqrt, acc += m*(r*den), G last). Bit-identical to the host
//    FP64 evaluation of NaiveAlgorithm.cpp:331-351.
//  * NB_F64: the same sum with the pair's separation, r^2 + eps^2 and m r^-3 in the fixed point of
//    nb_fix.cuh on the integer pipes and FP64 sums (3 FP64 operations per ordered pair): over all
//    bodies of a large system the symmetric kernel of nb_pair_sym.cu (each unordered pair once),
//    otherwise the one-sided naive_fix_kernel.
//  * NB_F32C: over all bodies of a large system, the symmetric FP32 pair kernel of
//    nb_pair_sym.cu (each unordered pair once, added to both bodies); otherwise (target ranges,
//    small systems) the one-sided FP32-compensated pair kernel of nb_pair.cuh (scalar FP32 pair
//    math, TwoSum accumulation, stream-K persistent CTAs, cp.async.bulk j-tiles behind bounded
//    mbarrier waits), run as a batch of one system.
//  * NB_DF64: double-float pair math on the FP32 pipe (FP64-accurate to ~1e-14); over all bodies
//    of a large system the double-float form of the symmetric pair kernel.
#include <cooperative_groups.h>

#include <algorithm>

#include "nb_fix.cuh"
#include "nb_internal.cuh"
#include "nb_pair.cuh"
#include "nb_pair_sym.cuh"

namespace {

// ---------------------------------------------------------------------------------------------
// FP64
// ---------------------------------------------------------------------------------------------
constexpr int F64_THREADS = 64;

__global__ void __launch_bounds__(F64_THREADS)
naive_ieee_kernel(const double* __restrict__ m, const double* __restrict__ x,
                  const double* __restrict__ y, const double* __restrict__ z,
                  double* __restrict__ ax, double* __restrict__ ay, double* __restrict__ az,
                  uint32_t n, uint32_t i_begin, uint32_t i_end, double G, double eps2) {
    __shared__ double sx[F64_THREADS], sy[F64_THREADS], sz[F64_THREADS], sm[F64_THREADS];
    const uint32_t i = i_begin + blockIdx.x * F64_THREADS + threadIdx.x;
    const bool active = i < i_end;
    double px = 0, py = 0, pz = 0;
    if (active) {
        px = x[i];
        py = y[i];
        pz = z[i];
    }
    double acc_x = 0, acc_y = 0, acc_z = 0;
    for (uint32_t k = 0; k < n; k += F64_THREADS) {
        const uint32_t j = k + threadIdx.x;
        if (j < n) {
            sx[threadIdx.x] = x[j];
            sy[threadIdx.x] = y[j];
            sz[threadIdx.x] = z[j];
            sm[threadIdx.x] = m[j];
        }
        __syncthreads();
        const uint32_t cnt = min((uint32_t)F64_THREADS, n - k);
        if (active) {
            for (uint32_t jj = 0; jj < cnt; ++jj) {
                const double r_x = __dsub_rn(sx[jj], px);
                const double r_y = __dsub_rn(sy[jj], py);
                const double r_z = __dsub_rn(sz[jj], pz);
                double den = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(r_x, r_x), __dmul_rn(r_y, r_y)),
                                                 __dmul_rn(r_z, r_z)),
                                       eps2);
                den = __dmul_rn(__dmul_rn(den, den), den);
                den = __ddiv_rn(1.0, __dsqrt_rn(den));
                acc_x = __dadd_rn(acc_x, __dmul_rn(sm[jj], __dmul_rn(r_x, den)));
                acc_y = __dadd_rn(acc_y, __dmul_rn(sm[jj], __dmul_rn(r_y, den)));
                acc_z = __dadd_rn(acc_z, __dmul_rn(sm[jj], __dmul_rn(r_z, den)));
            }
        }
        __syncthreads();
    }
    if (active) {
        ax[i] = __dmul_rn(acc_x, G);
        ay[i] = __dmul_rn(acc_y, G);
        az[i] = __dmul_rn(acc_z, G);
    }
}

// Adds the pair (source record f, body q) seen from body i at p to the sums: NB_F64's arithmetic.
// The pairs the fixed point cannot hold take the FP64 expressions; the self pair (its separation is
// 0) and massless sources mostly add nothing.
struct FixSums {
    double x, y, z;
};
__device__ __forceinline__ void fix_pair(const nbfix::FixRec& f, uint32_t q, uint32_t i,
                                         const nbfix::Fix3& p, int K, const nbfix::Eps2Table& e2,
                                         int sh_max, double eps2, const double* __restrict__ m,
                                         const double* __restrict__ x,
                                         const double* __restrict__ y,
                                         const double* __restrict__ z, FixSums& a) {
    double w, dx, dy, dz;
    if (sh_max < 0 || !nbfix::term(f, p, K, e2, sh_max, w, dx, dy, dz)) {
        w = dx = dy = dz = 0.0;
        if (!nbfix::adds_nothing(f, q == i, K, sh_max, eps2)) {
            dx = x[q] - x[i];
            dy = y[q] - y[i];
            dz = z[q] - z[i];
            w = nb_m_rinv3_f64(m[q], fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
        }
    }
    a.x = fma(w, dx, a.x);
    a.y = fma(w, dy, a.y);
    a.z = fma(w, dz, a.z);
}

// NB_F64, one-sided: target ranges, listed targets, systems below the symmetric kernel's sizes. One
// thread per target; the sources of a tile are converted to the fixed point of nb_fix.cuh by the
// block as it loads them, and a pair costs ~122 integer instructions and 3 FP64 ones instead of 16
// FP64 ones. blockIdx.y selects a chunk of `chunk` sources; with more than one chunk the partial
// sums (times G) go to part[(chunk index * targets + target) * 3 + axis].
//  Bound: the FP64 pipe (77% busy at 3 FMAs per pair) and dispatch. 8,192 bodies 2.16 -> 0.54 ms
//  (31 -> 125 Gpairs/s), 4,096 0.53 -> 0.16. 32 warps per SM in blocks of 256 (blocks of 128: 3%
//  slower, of 64: 16%).
constexpr int FX_THREADS = 256;
constexpr int FX_BLOCKS_PER_SM = 4;
// Source chunks: 32 blocks per SM in all (fewer leave a longer last wave: 16 are 4% slower at
// 16,384 bodies, 8 8%), but at most 128 chunks and at least 4 sources each, since every pair of a
// lone block's chain of tiles is ~0.5 us while its start and the combine pass are ~2 us each.
constexpr long long FX_GRID_PER_SM = 32;
constexpr uint32_t FX_CHUNKS_MAX = 128, FX_CHUNK_MIN = 4;
static_assert(NB_COUNTER_WORDS - NB_COUNTER_SCALE >= (int)nbfix::SCALE_WORDS, "scale words");

__global__ void __launch_bounds__(FX_THREADS, FX_BLOCKS_PER_SM)
naive_fix_kernel(const double* m, const double* x,
                 const double* y, const double* z,
                 double* __restrict__ ax, double* __restrict__ ay, double* __restrict__ az,
                 uint32_t n, const uint32_t* targets, uint32_t i_begin, uint32_t n_t,
                 double G, double eps2, uint32_t chunk, double* __restrict__ part,
                 const uint32_t* k_part, uint32_t k_words) {
    nb_grid_wait();
    __shared__ nbfix::FixRec src[FX_THREADS];
    __shared__ nbfix::Eps2Table e2;
    const int K = nbfix::block_scale(x, y, z, n, k_part, k_words);
    nbfix::fill_eps2(e2, eps2, K);
    __syncthreads();
    const uint32_t t = blockIdx.x * FX_THREADS + threadIdx.x;
    const bool active = t < n_t;
    const uint32_t i = active ? (targets != nullptr ? targets[t] : i_begin + t) : 0u;
    nbfix::Fix3 p;
    const int sh_max = nbfix::split3(x[i], y[i], z[i], K, p) ? e2.sh_max : -1;
    FixSums acc{0.0, 0.0, 0.0};
    const uint32_t j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
    for (uint32_t k = j0; k < j1; k += FX_THREADS) {
        const uint32_t j = k + threadIdx.x;
        __syncthreads();
        if (j < j1) src[threadIdx.x] = nbfix::make_rec(x[j], y[j], z[j], m[j], K);
        __syncthreads();
        const uint32_t cnt = active ? min((uint32_t)FX_THREADS, j1 - k) : 0u;
#pragma unroll 1
        for (uint32_t jj = 0; jj < cnt; ++jj)
            fix_pair(src[jj], k + jj, i, p, K, e2, sh_max, eps2, m, x, y, z, acc);
    }
    if (!active) return;
    if (gridDim.y == 1) {
        const uint32_t o = targets != nullptr ? t : i;
        ax[o] = acc.x * G;
        ay[o] = acc.y * G;
        az[o] = acc.z * G;
    } else {
        double* o = part + ((size_t)blockIdx.y * n_t + t) * 3;
        o[0] = acc.x * G;
        o[1] = acc.y * G;
        o[2] = acc.z * G;
    }
}

// The same for systems of up to FXC_MAX_N bodies, where one launch without global partials counts:
// a cluster of 8 CTAs per 32 targets, the sources split over the CTAs and each CTA's share over its
// 8 warps. The warps' sums are added in warp order in shared memory, the CTAs' sums in rank order
// by rank 0 through distributed shared memory.
//  Bound: the ~0.5 us latency of each of the n / 64 pairs a warp evaluates one after the other, and
//  ~4 us of start and reductions. 1,009 bodies: 48 us (FP64, chunks and a combine pass) -> 19 us;
//  2,048: 144 -> 50. At 3,000 bodies the chunked kernel above is 8% faster.
constexpr int FXC_CTAS = 8, FXC_WARPS = 8, FXC_THREADS = 32 * FXC_WARPS;
constexpr uint32_t FXC_MAX_N = 2048;
static_assert(FXC_MAX_N <= nbfix::SCALE_SCAN_N, "one launch");
static_assert(FXC_MAX_N <= FXC_CTAS * FXC_THREADS, "a CTA's share of the sources is one tile");

__global__ void __cluster_dims__(FXC_CTAS, 1, 1) __launch_bounds__(FXC_THREADS)
naive_fix_cluster_kernel(const double* m, const double* x,
                         const double* y, const double* z,
                         double* __restrict__ ax, double* __restrict__ ay,
                         double* __restrict__ az, uint32_t n,
                         const uint32_t* targets, uint32_t i_begin, uint32_t n_t,
                         double G, double eps2, const uint32_t* k_part,
                         uint32_t k_words) {
    nb_grid_wait();
    namespace cg = cooperative_groups;
    __shared__ nbfix::FixRec src[FXC_THREADS];
    __shared__ nbfix::Eps2Table e2;
    __shared__ double sums[FXC_WARPS][3][32], total[3][32];
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t t = (blockIdx.x / FXC_CTAS) * 32 + lane;
    const bool active = t < n_t;
    const uint32_t i = active ? (targets != nullptr ? targets[t] : i_begin + t) : 0u;
    const uint32_t share = (n + FXC_CTAS - 1) / FXC_CTAS;
    const uint32_t j0 = min(n, rank * share), j1 = min(n, j0 + share), j = j0 + threadIdx.x;
    // the target and this thread's source, requested before the scan for the scale
    const double px = x[i], py = y[i], pz = z[i];
    double jx = 0.0, jy = 0.0, jz = 0.0, jm = 0.0;
    if (j < j1) {
        jx = x[j];
        jy = y[j];
        jz = z[j];
        jm = m[j];
    }
    const int K = nbfix::block_scale(x, y, z, n, k_part, k_words);
    nbfix::fill_eps2(e2, eps2, K);
    if (j < j1) src[threadIdx.x] = nbfix::make_rec(jx, jy, jz, jm, K);
    __syncthreads();
    nbfix::Fix3 p;
    const int sh_max = nbfix::split3(px, py, pz, K, p) ? e2.sh_max : -1;
    FixSums acc{0.0, 0.0, 0.0};
#pragma unroll 1
    for (uint32_t jj = w; jj < j1 - j0; jj += FXC_WARPS)
        fix_pair(src[jj], j0 + jj, i, p, K, e2, sh_max, eps2, m, x, y, z, acc);
    sums[w][0][lane] = acc.x;
    sums[w][1][lane] = acc.y;
    sums[w][2][lane] = acc.z;
    __syncthreads();
    if (w < 3) {
        double s = sums[0][w][lane];
#pragma unroll
        for (int v = 1; v < FXC_WARPS; ++v) s += sums[v][w][lane];
        total[w][lane] = s;
    }
    cluster.sync();
    if (rank == 0 && w < 3) {
        double s = total[w][lane];
#pragma unroll
        for (int r = 1; r < FXC_CTAS; ++r) s += *cluster.map_shared_rank(&total[w][lane], r);
        if (active) (w == 0 ? ax : (w == 1 ? ay : az))[targets != nullptr ? t : i] = s * G;
    }
    cluster.sync();  // no CTA leaves while rank 0 reads its shared memory
}

// Adds the chunks' partial sums of each target in a fixed order: 32 targets per block, warp w takes
// chunks w, w + 8, ..., then the warps' sums in warp order (a chain of one thread per target over
// 64 chunks took 24 us: one load and one FP64 latency after the other).
constexpr int CC_WARPS = 8;

__global__ void __launch_bounds__(32 * CC_WARPS)
chunk_combine_kernel(const double* part, uint32_t chunks, uint32_t i_begin,
                     uint32_t i_end, double* __restrict__ ax, double* __restrict__ ay,
                     double* __restrict__ az) {
    nb_grid_wait();
    __shared__ double sum[CC_WARPS][3][32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, n_t = i_end - i_begin;
    const uint32_t t = blockIdx.x * 32 + lane;
    double s[3] = {0.0, 0.0, 0.0};
    if (t < n_t) {
#pragma unroll 4
        for (uint32_t c = w; c < chunks; c += CC_WARPS) {
            const double* o = part + ((size_t)c * n_t + t) * 3;
            s[0] += o[0];
            s[1] += o[1];
            s[2] += o[2];
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) sum[w][a][lane] = s[a];
    __syncthreads();
    if (w >= 3 || t >= n_t) return;
    double r = sum[0][w][lane];
    for (uint32_t v = 1; v < min((uint32_t)CC_WARPS, chunks); ++v) r += sum[v][w][lane];
    double* out = w == 0 ? ax : (w == 1 ? ay : az);
    out[i_begin + t] = r;
}

// Number and size (a multiple of `tile`) of the source chunks that give at least ~8 warps per SM
// when blocks_per_chunk blocks cover the targets.
void choose_chunks(const nb_ctx* ctx, int blocks_per_chunk, uint32_t n, uint32_t tile,
                   uint32_t* chunks, uint32_t* chunk) {
    uint32_t c = (uint32_t)nb::ceil_div(8LL * ctx->sm_count, blocks_per_chunk);
    c = min(c, 32u);
    c = min(c, (uint32_t)nb::ceil_div(n, tile));
    if (c < 1) c = 1;
    *chunk = (uint32_t)nb::ceil_div(nb::ceil_div(n, c), tile) * tile;
    *chunks = (uint32_t)nb::ceil_div(n, *chunk);
}

// ---------------------------------------------------------------------------------------------
// FP32, compensated: the batched pair kernel (nb_pair.cuh) with a batch of one system whose
// targets are [i_begin, i_end).
// ---------------------------------------------------------------------------------------------
int g_naive_pair_cfg = 0;  // tile configuration (nb_naive_set_pair_config)
// Symmetric kernel (nb_pair_sym.cu) for full target ranges (nb_naive_set_symmetric): mode 0
// never, 1 automatic, 2 always; and its FP32, FP64 and double-float shapes.
int g_naive_sym_mode = 1;
int g_naive_sym_cfg[3] = {0, 0, 0};
// Automatic selection wants at least this many units per persistent CTA (the one-sided kernels
// spread small systems better) and j-side partials (3 values per unit and tile body) below the
// cap.
constexpr uint64_t SYM_MIN_UNITS_PER_CTA = 7;
// FP64: from 4 units per CTA on (~9,900 bodies). 12,000 bodies (5.8 units): 0.97 ms against 1.10
// one-sided, 9,900: 0.76 / 0.77, 8,192 (2.8 units): 0.51 / 0.54, 4,096: 0.18 / 0.16; between the last
// two the one-sided kernel stays, which also runs in a capture without scratch.
constexpr uint64_t SYM_MIN_UNITS_F64 = 4;
constexpr size_t SYM_PART_CAP_BYTES = (size_t)4 << 30;

// Runs the symmetric kernel of arithmetic form `form` (nb::SymForm) for the whole system when
// the mode and the plan allow it; *done tells whether it did.
nb_status naive_sym(nb_ctx* ctx, int form, const double* m, const double* x, const double* y,
                    const double* z, double* ax, double* ay, double* az, uint32_t n, double G,
                    double eps2, cudaStream_t stream, bool* done) {
    *done = false;
    if (g_naive_sym_mode == 0) return NB_OK;
    // candidate shapes: the configured one, except in the automatic mode of the FP64 and
    // double-float forms, which take shape 0 (4,2,64) with 256-body I-blocks (fewer registers per
    // thread) and, where its partials do not fit, shape 1 (4,4,64) with 512 and half the partials.
    // FP64, shape 0 against 1: 157 / 146 Gpairs/s at 16,384 bodies, 161 / 159 at 32,768, 164 / 162
    // from 98,304 on; at 320,000, where shape 0 needs 4.4 GiB of partials, 165 / 163 and 149
    // one-sided.
    int cand[2] = {g_naive_sym_cfg[form], -1};
    if (g_naive_sym_mode == 1 && form != nb::SYM_F32) {
        cand[0] = 0;
        cand[1] = 1;
    }
    const uint64_t min_units = form == nb::SYM_F64 ? SYM_MIN_UNITS_F64 : SYM_MIN_UNITS_PER_CTA;
    int cfg = -1;
    nb::SymHostPlan hp;
    size_t pj_bytes = 0;
    for (int c : cand) {
        if (c < 0) break;
        NB_TRY(nb::sym_host_plan(form, c, &n, 1, ctx->sm_count, &hp));
        pj_bytes = nb::sym_part_j_bytes(form, c, hp.units);
        if (g_naive_sym_mode == 2 || (hp.units >= min_units * hp.ctas &&
                                      pj_bytes <= SYM_PART_CAP_BYTES)) {
            cfg = c;
            break;
        }
    }
    if (cfg < 0) return NB_OK;
    auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t table_bytes = al(2 * sizeof(nbsym::SymSys));
    const size_t src_bytes = al((size_t)hp.n_records * nb::sym_record_bytes(form));
    const size_t pi_bytes = al(nb::sym_part_i_bytes(form, cfg, hp.ctas, hp.n_blocks));
    void* base = nullptr;
    NB_TRY(nb::scratch(ctx, NB_SCRATCH_PAIR_SYM, table_bytes + src_bytes + pi_bytes + pj_bytes,
                       stream, &base));
    char* b = (char*)base;
    nbsym::SymSys* table = (nbsym::SymSys*)b;
    NB_TRY(nb::sym_single_table(table, hp, stream));
    nbsym::SymPlan S;
    S.sys = table;
    S.n_systems = 1;
    S.ctas = hp.ctas;
    S.n_total = hp.n_total;
    S.n_records = hp.n_records;
    S.units = hp.units;
    S.wait_limit = ctx->wait_limit;
    S.k_part = ctx->dev_counter + NB_COUNTER_SCALE;
    S.k_words = 0;
    if (form == nb::SYM_F64)
        NB_TRY(nb::launch_scale(x, y, z, n, ctx->dev_counter + NB_COUNTER_SCALE, &S.k_words,
                                stream));
    b += table_bytes;
    *done = true;
    return nb::sym_launch(form, cfg, S, m, x, y, z, G, eps2, b, b + src_bytes,
                          b + src_bytes + pi_bytes, ax, ay, az, ctx->dev_error, stream);
}

nb_status naive_f32c(nb_ctx* ctx, const double* m, const double* x, const double* y,
                     const double* z, double* ax, double* ay, double* az, uint32_t n,
                     uint32_t i_begin, uint32_t i_end, double G, double eps2,
                     cudaStream_t stream) {
    if (i_begin == 0 && i_end == n) {
        bool done = false;
        NB_TRY(naive_sym(ctx, nb::SYM_F32, m, x, y, z, ax, ay, az, n, G, eps2, stream, &done));
        if (done) return NB_OK;
    }
    const int cfg = g_naive_pair_cfg;
    const nb::PairConfig& C = nb::kPairConfigs[cfg];
    int per_sm = 0;
    NB_TRY(nb::pair_ctas_per_sm(cfg, &per_sm));
    const uint32_t n_t = i_end - i_begin;
    const uint32_t ib = (uint32_t)(C.threads * C.ip);
    const uint32_t n_ib = (n_t + ib - 1) / ib;
    const uint32_t n_jt = (n + C.jt - 1) / C.jt;
    const uint64_t units = (uint64_t)n_ib * n_jt;
    uint64_t ctas = (uint64_t)ctx->sm_count * per_sm;
    if (ctas > units) ctas = units;
    // scratch: plan arrays, duplicated sources, float4 targets, partials
    const size_t plan_bytes = 512;
    const size_t src_bytes = ((size_t)n * sizeof(nbpair::SrcDup) + 255) & ~(size_t)255;
    const size_t tgt_bytes = ((size_t)n * sizeof(float4) + 255) & ~(size_t)255;
    const size_t part_bytes = nb::pair_partial_floats(cfg, (uint32_t)ctas, n_ib) * sizeof(float);
    void* base = nullptr;
    NB_TRY(nb::scratch(ctx, NB_SCRATCH_NAIVE_F32, plan_bytes + src_bytes + tgt_bytes + part_bytes,
                       stream, &base));
    char* b = (char*)base;
    uint64_t* unit_off = (uint64_t*)b;
    uint32_t* sys_off = (uint32_t*)(b + 64);
    uint32_t* tgt_begin = (uint32_t*)(b + 128);
    uint32_t* t_off = (uint32_t*)(b + 192);
    uint32_t* ib_off = (uint32_t*)(b + 256);
    nbpair::SrcDup* src = (nbpair::SrcDup*)(b + plan_bytes);
    float4* tgt = (float4*)(b + plan_bytes + src_bytes);
    float* part = (float*)(b + plan_bytes + src_bytes + tgt_bytes);
    NB_TRY(nb::pair_plan_single(sys_off, tgt_begin, t_off, unit_off, ib_off, n, i_begin, i_end,
                                units, n_ib, stream));
    nbpair::Plan P;
    P.n_systems = 1;
    P.ctas = (uint32_t)ctas;
    P.units = units;
    P.sys_off = sys_off;
    P.tgt_begin = tgt_begin;
    P.t_off = t_off;
    P.unit_off = unit_off;
    P.ib_off = ib_off;
    P.wait_limit = ctx->wait_limit;
    return nb::pair_launch(cfg, P, m, x, y, z, n, n_t, G, eps2, src, tgt, part, ax, ay, az,
                           ctx->dev_error, stream);
}

// ---------------------------------------------------------------------------------------------
// Double-float (NB_DF64): FP64-accurate pair math on the FP32 pipe
// ---------------------------------------------------------------------------------------------
constexpr int DF_THREADS = 128;
constexpr int DF_TILE = 128;

// Source record: the position minus body 0 (exact) as triple-floats and G*m as a double-float.
struct __align__(16) SrcTF {
    float xh, xm, xl, yh, ym, yl, zh, zm, zl, gh, gl, pad;
};

__global__ void df_prepare_kernel(const double* __restrict__ m, const double* __restrict__ x,
                                  const double* __restrict__ y, const double* __restrict__ z,
                                  uint32_t n, double G, SrcTF* __restrict__ out) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    SrcTF r;
    tf_split_diff(x[b], x[0], r.xh, r.xm, r.xl);
    tf_split_diff(y[b], y[0], r.yh, r.ym, r.yl);
    tf_split_diff(z[b], z[0], r.zh, r.zm, r.zl);
    const double gm = G * m[b];
    r.gh = (float)gm;
    r.gl = (float)(gm - (double)r.gh);
    r.pad = 0.f;
    out[b] = r;
}

// One thread per target; sources in shared-memory tiles. Per pair: exact separations from the
// triple-floats, r^2 + eps^2 with TwoSums, 1/r from the hardware estimate with an error-free
// correction, G m / r^3 and the products in double-float (the same arithmetic as the
// Barnes-Hut double-float monopole), Neumaier-compensated sums per tile added into FP64. The
// self pair contributes exactly 0.
// blockIdx.y selects a chunk of `chunk` sources; with more than one chunk the partial sums go
// to part[(chunk index * n_t + target) * 3 + axis] and df_combine_kernel adds them in order.
__global__ void __launch_bounds__(DF_THREADS)
naive_df_kernel(const SrcTF* __restrict__ src, uint32_t n, uint32_t i_begin, uint32_t i_end,
                uint32_t chunk, float e2h, float e2l, double* __restrict__ ax,
                double* __restrict__ ay, double* __restrict__ az, double* __restrict__ part) {
    __shared__ SrcTF tile[DF_TILE];
    const uint32_t i = i_begin + blockIdx.x * DF_THREADS + threadIdx.x;
    const bool active = i < i_end;
    SrcTF me{};
    if (active) me = src[i];
    double sum_x = 0.0, sum_y = 0.0, sum_z = 0.0;
    const uint32_t j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
    for (uint32_t k = j0; k < j1; k += DF_TILE) {
        float ahx = 0.f, ahy = 0.f, ahz = 0.f, alx = 0.f, aly = 0.f, alz = 0.f;
        for (uint32_t j = threadIdx.x; j < DF_TILE && k + j < j1; j += DF_THREADS)
            tile[j] = src[k + j];
        __syncthreads();
        const uint32_t cnt = min((uint32_t)DF_TILE, j1 - k);
        if (active) {
            for (uint32_t jj = 0; jj < cnt; ++jj) {
                const SrcTF c = tile[jj];
                const nb_df dx = tf_diff(c.xh, c.xm, c.xl, me.xh, me.xm, me.xl);
                const nb_df dy = tf_diff(c.yh, c.ym, c.yl, me.yh, me.ym, me.yl);
                const nb_df dz = tf_diff(c.zh, c.zm, c.zl, me.zh, me.zm, me.zl);
                const nb_df sx = df_sqr(dx), sy = df_sqr(dy), sz = df_sqr(dz);
                nb_df a = df_two_sum(sx.h, sy.h);
                a.l += sx.l + sy.l;
                nb_df b = df_two_sum(a.h, sz.h);
                b.l += a.l + sz.l;
                nb_df e = df_two_sum(b.h, e2h);
                e.l += b.l + e2l;
                const nb_df r2 = df_two_sum(e.h, e.l);
                const float y0 = nb_rsqrt_f32(r2.h);
                const float q = y0 * y0, qe = fmaf(y0, y0, -q);
                const float th = r2.h * q;
                float te = fmaf(r2.h, q, -th);
                te = fmaf(r2.h, qe, te);
                te = fmaf(r2.l, q, te);
                const float ee = (1.0f - th) - te;
                const nb_df inv = df_fast_two_sum(y0, y0 * (ee * fmaf(0.375f, ee, 0.5f)));
                const nb_df w = df_mul(nb_df{c.gh, c.gl}, df_mul(df_sqr(inv), inv));
                const nb_df tx = df_mul(dx, w), ty = df_mul(dy, w), tz = df_mul(dz, w);
                nb_df t = df_two_sum(ahx, tx.h);
                ahx = t.h;
                alx += t.l + tx.l;
                t = df_two_sum(ahy, ty.h);
                ahy = t.h;
                aly += t.l + ty.l;
                t = df_two_sum(ahz, tz.h);
                ahz = t.h;
                alz += t.l + tz.l;
            }
            // the tile's compensated sum into FP64 (3 FP64 adds per tile): the FP32 low part
            // of a compensated sum over all n terms would lose digits at large n
            sum_x += (double)ahx + (double)alx;
            sum_y += (double)ahy + (double)aly;
            sum_z += (double)ahz + (double)alz;
        }
        __syncthreads();
    }
    if (!active) return;
    if (gridDim.y == 1) {
        ax[i] = sum_x;
        ay[i] = sum_y;
        az[i] = sum_z;
    } else {
        double* o = part + ((size_t)blockIdx.y * (i_end - i_begin) + (i - i_begin)) * 3;
        o[0] = sum_x;
        o[1] = sum_y;
        o[2] = sum_z;
    }
}


nb_status naive_df64(nb_ctx* ctx, const double* m, const double* x, const double* y,
                     const double* z, double* ax, double* ay, double* az, uint32_t n,
                     uint32_t i_begin, uint32_t i_end, double G, double eps2,
                     cudaStream_t stream) {
    // split the sources into chunks when the targets alone give too few warps per SM
    const uint32_t n_t = i_end - i_begin;
    const int blocks = nb::ceil_div(n_t, DF_THREADS);
    uint32_t chunks = 1, chunk = n;
    choose_chunks(ctx, blocks, n, DF_TILE, &chunks, &chunk);
    const size_t src_bytes = ((size_t)n * sizeof(SrcTF) + 255) & ~(size_t)255;
    const size_t part_bytes = chunks > 1 ? (size_t)chunks * n_t * 3 * sizeof(double) : 0;
    void* base = nullptr;
    NB_TRY(nb::scratch(ctx, NB_SCRATCH_NAIVE_DF, src_bytes + part_bytes, stream, &base));
    SrcTF* src = (SrcTF*)base;
    double* part = (double*)((char*)base + src_bytes);
    df_prepare_kernel<<<nb::ceil_div(n, 256), 256, 0, stream>>>(m, x, y, z, n, G, src);
    NB_TRY(nb::check_launch("df_prepare_kernel"));
    const float e2h = (float)eps2, e2l = (float)(eps2 - (double)e2h);
    naive_df_kernel<<<dim3(blocks, chunks), DF_THREADS, 0, stream>>>(
        src, n, i_begin, i_end, chunk, e2h, e2l, ax, ay, az, part);
    NB_TRY(nb::check_launch("naive_df_kernel"));
    if (chunks == 1) return NB_OK;
    chunk_combine_kernel<<<nb::ceil_div(n_t, 32), 32 * CC_WARPS, 0, stream>>>(part, chunks, i_begin,
                                                                     i_end, ax, ay, az);
    return nb::check_launch("chunk_combine_kernel");
}

// One-sided NB_F64 for the n_t targets i_begin .. or the listed ones (whose results are packed).
nb_status naive_fix(nb_ctx* ctx, const double* m, const double* x, const double* y,
                    const double* z, double* ax, double* ay, double* az, uint32_t n,
                    const uint32_t* targets, uint32_t i_begin, uint32_t n_t, double G, double eps2,
                    cudaStream_t stream) {
    uint32_t* k_part = ctx->dev_counter + NB_COUNTER_SCALE;
    uint32_t k_words = 0;
    NB_TRY(nb::launch_scale(x, y, z, n, k_part, &k_words, stream));
    if (n <= FXC_MAX_N) {
        NB_CUDA_TRY(nb::launch_after(naive_fix_cluster_kernel, nb::ceil_div(n_t, 32) * FXC_CTAS,
                                     FXC_THREADS, 0, stream, m, x, y, z, ax, ay, az, n, targets,
                                     i_begin, n_t, G, eps2, k_part, k_words));
        return NB_OK;
    }
    const int blocks = nb::ceil_div(n_t, FX_THREADS);
    uint32_t chunks = (uint32_t)std::min<long long>(
        nb::ceil_div(FX_GRID_PER_SM * ctx->sm_count, blocks), FX_CHUNKS_MAX);
    uint32_t chunk = std::max<uint32_t>((uint32_t)nb::ceil_div(n, chunks), FX_CHUNK_MIN);
    if (chunk > FX_THREADS) chunk = (uint32_t)nb::ceil_div(chunk, FX_THREADS) * FX_THREADS;
    chunks = (uint32_t)nb::ceil_div(n, chunk);
    // A capture that finds no scratch large enough cannot wait for an allocation: the partials are then
    // the graph's own memory. (So the chunks, and with them the sums' order, never depend on what ran
    // before.)
    const size_t part_bytes = chunks > 1 ? (size_t)chunks * n_t * 3 * sizeof(double) : 0;
    const bool own = part_bytes > ctx->scratch[NB_SCRATCH_NAIVE_DF].bytes && nb::is_capturing(stream);
    void* base = nullptr;
    if (own) {
        NB_CUDA_TRY(cudaMallocAsync(&base, part_bytes, stream));
    } else if (chunks > 1) {
        NB_TRY(nb::scratch(ctx, NB_SCRATCH_NAIVE_DF, part_bytes, stream, &base));
    }
    double* part = (double*)base;
    NB_CUDA_TRY(nb::launch_after(naive_fix_kernel, dim3(blocks, chunks), FX_THREADS, 0, stream, m, x,
                                 y, z, ax, ay, az, n, targets, i_begin, n_t, G, eps2, chunk, part,
                                 k_part, k_words));
    if (chunks == 1) return NB_OK;
    const uint32_t first = targets != nullptr ? 0 : i_begin;
    NB_CUDA_TRY(nb::launch_after(chunk_combine_kernel, nb::ceil_div(n_t, 32), 32 * CC_WARPS, 0, stream,
                                 part, chunks, first, first + n_t, ax, ay, az));
    if (own) NB_CUDA_TRY(cudaFreeAsync(base, stream));
    return NB_OK;
}

nb_status naive_dispatch(nb_ctx* ctx, const double* m, const double* x, const double* y,
                         const double* z, double* ax, double* ay, double* az, uint32_t n,
                         uint32_t i_begin, uint32_t i_end, double G, double eps2,
                         nb_precision prec, cudaStream_t stream) {
    NB_CHECK_CTX(ctx);
    if (n == 0 || i_begin >= i_end) return NB_OK;
    if (!m || !x || !y || !z || !ax || !ay || !az)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_naive_accel: null array pointer");
    if (i_end > n) return nb::set_error(NB_ERR_INVALID_ARG, "nb_naive_accel: i_end > n");
    const uint32_t n_t = i_end - i_begin;
    switch (prec) {
        case NB_F64_IEEE:
            naive_ieee_kernel<<<nb::ceil_div(n_t, F64_THREADS), F64_THREADS, 0, stream>>>(
                m, x, y, z, ax, ay, az, n, i_begin, i_end, G, eps2);
            return nb::check_launch("naive_ieee_kernel");
        case NB_F64: {
            if (i_begin == 0 && i_end == n) {
                bool done = false;
                NB_TRY(naive_sym(ctx, nb::SYM_F64, m, x, y, z, ax, ay, az, n, G, eps2, stream,
                                 &done));
                if (done) return NB_OK;
            }
            return naive_fix(ctx, m, x, y, z, ax, ay, az, n, nullptr, i_begin, n_t, G, eps2,
                             stream);
        }
        case NB_F32C:
            return naive_f32c(ctx, m, x, y, z, ax, ay, az, n, i_begin, i_end, G, eps2, stream);
        case NB_DF64: {
            if (i_begin == 0 && i_end == n) {
                bool done = false;
                NB_TRY(naive_sym(ctx, nb::SYM_DF, m, x, y, z, ax, ay, az, n, G, eps2, stream,
                                 &done));
                if (done) return NB_OK;
            }
            return naive_df64(ctx, m, x, y, z, ax, ay, az, n, i_begin, i_end, G, eps2, stream);
        }
        default:
            return nb::set_error(NB_ERR_INVALID_ARG, "nb_naive_accel: unknown precision %d",
                                 (int)prec);
    }
}

}  // namespace

extern "C" {

nb_status nb_naive_accel(nb_ctx* ctx, const double* m, const double* x, const double* y,
                         const double* z, double* ax, double* ay, double* az, uint32_t n,
                         double G, double eps2, nb_precision prec, int block_size,
                         nb_stream_t stream) {
    if (block_size < 0)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_naive_accel: block_size must be >= 0");
    return naive_dispatch(ctx, m, x, y, z, ax, ay, az, n, 0, n, G, eps2, prec,
                          (cudaStream_t)stream);
}

nb_status nb_naive_accel_targets(nb_ctx* ctx, const double* m, const double* x, const double* y,
                                 const double* z, uint32_t n, const uint32_t* targets,
                                 uint32_t n_targets, double* ax, double* ay, double* az, double G,
                                 double eps2, nb_stream_t stream) {
    NB_CHECK_CTX(ctx);
    if (!m || !x || !y || !z || !targets || !ax || !ay || !az)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_naive_accel_targets: null pointer");
    if (n == 0 || n_targets == 0) return NB_OK;
    return naive_fix(ctx, m, x, y, z, ax, ay, az, n, targets, 0, n_targets, G, eps2,
                     (cudaStream_t)stream);
}

nb_status nb_naive_set_pair_config(int config) {
    if (config < 0 || config >= nb::NB_PAIR_CONFIGS)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_naive_set_pair_config: config %d", config);
    g_naive_pair_cfg = config;
    return NB_OK;
}

nb_status nb_naive_set_symmetric(int mode, int config_f32, int config_f64, int config_df) {
    if (mode < 0 || mode > 2)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_naive_set_symmetric: mode %d", mode);
    const int cfg[3] = {config_f32, config_f64, config_df};
    for (int f = 0; f < 3; ++f)
        if (cfg[f] < 0 || cfg[f] >= nb::sym_config_count(f))
            return nb::set_error(NB_ERR_INVALID_ARG, "nb_naive_set_symmetric: config %d of form %d",
                                 cfg[f], f);
    g_naive_sym_mode = mode;
    for (int f = 0; f < 3; ++f) g_naive_sym_cfg[f] = cfg[f];
    return NB_OK;
}

nb_status nb_naive_accel_range(nb_ctx* ctx, const double* m, const double* x, const double* y,
                               const double* z, double* ax, double* ay, double* az, uint32_t n,
                               uint32_t i_begin, uint32_t i_end, double G, double eps2,
                               nb_precision prec, nb_stream_t stream) {
    return naive_dispatch(ctx, m, x, y, z, ax, ay, az, n, i_begin, i_end, G, eps2, prec,
                          (cudaStream_t)stream);
}

}  // extern "C"
