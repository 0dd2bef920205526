// nb_integrate.cu -- leapfrog kick-drift-kick, energy and AABB kernels (all FP64).
#include <algorithm>
#include <mutex>

#include "nb_aabb.cuh"
#include "nb_fix.cuh"
#include "nb_internal.cuh"

namespace {

constexpr int EW_THREADS = 256;

// NaiveAlgorithm.cpp:154-163 / BarnesHutAlgorithm.cpp:171-181. Each statement is a separately
// rounded multiply and add, exactly as the reference writes it.
__global__ void kick_drift_kernel(double* __restrict__ vhx, double* __restrict__ vhy,
                                  double* __restrict__ vhz, const double* vx,
                                  const double* vy, const double* vz,
                                  double* __restrict__ x, double* __restrict__ y,
                                  double* __restrict__ z, const double* ax,
                                  const double* ay, const double* az,
                                  uint32_t n, double dt) {
    nb_grid_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double h = dt / 2.0, px = x[i], py = y[i], pz = z[i];
    const double hx = __dadd_rn(vx[i], __dmul_rn(ax[i], h));
    const double hy = __dadd_rn(vy[i], __dmul_rn(ay[i], h));
    const double hz = __dadd_rn(vz[i], __dmul_rn(az[i], h));
    vhx[i] = hx;
    vhy[i] = hy;
    vhz[i] = hz;
    x[i] = __dadd_rn(px, __dmul_rn(hx, dt));
    y[i] = __dadd_rn(py, __dmul_rn(hy, dt));
    z[i] = __dadd_rn(pz, __dmul_rn(hz, dt));
}

// NaiveAlgorithm.cpp:217-221 / BarnesHutAlgorithm.cpp:234-238.
__global__ void kick_kernel(double* __restrict__ vx, double* __restrict__ vy,
                            double* __restrict__ vz, const double* vhx,
                            const double* vhy, const double* vhz,
                            const double* ax, const double* ay,
                            const double* az, uint32_t n, double dt) {
    nb_grid_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double h = dt / 2.0;
    const double nvx = __dadd_rn(vhx[i], __dmul_rn(ax[i], h));
    const double nvy = __dadd_rn(vhy[i], __dmul_rn(ay[i], h));
    const double nvz = __dadd_rn(vhz[i], __dmul_rn(az[i], h));
    vx[i] = nvx;
    vy[i] = nvy;
    vz[i] = nvz;
}

// Part 2 of one step followed by part 1 of the next: v = vh + a*dt/2; vh = v + a*dt/2;
// x += vh*dt. The same roundings as running the two kernels back to back.
__global__ void kick_kick_drift_kernel(double* __restrict__ vx, double* __restrict__ vy,
                                       double* __restrict__ vz, double* __restrict__ vhx,
                                       double* __restrict__ vhy, double* __restrict__ vhz,
                                       double* __restrict__ x, double* __restrict__ y,
                                       double* __restrict__ z, const double* ax,
                                       const double* ay,
                                       const double* az, uint32_t n, double dt) {
    nb_grid_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double h = dt / 2.0, px = x[i], py = y[i], pz = z[i];
    const double kx = __dmul_rn(ax[i], h), ky = __dmul_rn(ay[i], h), kz = __dmul_rn(az[i], h);
    const double nvx = __dadd_rn(vhx[i], kx), nvy = __dadd_rn(vhy[i], ky),
                 nvz = __dadd_rn(vhz[i], kz);
    vx[i] = nvx;
    vy[i] = nvy;
    vz[i] = nvz;
    const double hx = __dadd_rn(nvx, kx), hy = __dadd_rn(nvy, ky), hz = __dadd_rn(nvz, kz);
    vhx[i] = hx;
    vhy[i] = hy;
    vhz[i] = hz;
    x[i] = __dadd_rn(px, __dmul_rn(hx, dt));
    y[i] = __dadd_rn(py, __dmul_rn(hy, dt));
    z[i] = __dadd_rn(pz, __dmul_rn(hz, dt));
}

// ---------------------------------------------------------------------------------------------
// Energy: per target body j the kinetic term and the potential sum over sources i < j
// (nBodyAlgorithm.cpp:48-64), then a fixed-order reduction (deterministic).
//
// Bodies in rows of 128 targets; a row's units are its tiles of sources up to the diagonal, and
// the units of all rows form one sequence that the CTAs split into equal contiguous ranges, so the
// triangle's rows of unequal length load the SMs evenly. 1/r comes from the fixed point of
// nb_fix.cuh (within one rounding of exact); of a pair's work only the sum, G m_i * (1/r), is on the
// FP64 pipe. Pairs the fixed point cannot hold (closer than 2^(K-29), or coordinates beyond its
// exponent range) take the FP64 expression.
//  Bound: dispatch of 107 instructions per unordered pair, half of them 64-bit (issue 58%, integer
//  pipe 54%, wide multiplies 57%, FP64 pipe 38% of cycles), against 14 FP64 operations at 1/75 of
//  the FP32 rate before. 50,021 bodies: 49.2 -> 5.45 ms (25 -> 230 Gpairs/s). 48 warps per SM (24
//  to 40: 1 to 7% slower).
// ---------------------------------------------------------------------------------------------
constexpr int EN_THREADS = 128;        // targets per row, sources per tile at most
constexpr int EN_CTAS_PER_SM = 12;

// tile: sources per unit (a divisor of EN_THREADS); k_part, k_words: nbfix::block_scale.
__global__ void __launch_bounds__(EN_THREADS, EN_CTAS_PER_SM)
energy_kernel(const double* __restrict__ m, const double* __restrict__ x,
              const double* __restrict__ y, const double* __restrict__ z,
              const double* __restrict__ vx, const double* __restrict__ vy,
              const double* __restrict__ vz, uint32_t n, double G, uint32_t tile, uint64_t units,
              const uint32_t* __restrict__ k_part, uint32_t k_words, double2* __restrict__ part) {
    __shared__ nbfix::FixRec src[EN_THREADS];  // positions; G times the mass as a double in (mh, ml)
    __shared__ double red_k[EN_THREADS / 32], red_p[EN_THREADS / 32];
    const uint32_t tid = threadIdx.x;
    const int K = nbfix::block_scale(x, y, z, n, k_part, k_words);
    const bool usable = nbfix::k_usable(K);  // the same in all threads
    const uint32_t q = EN_THREADS / tile;    // tiles per row of sources
    const uint64_t u0 = units * blockIdx.x / gridDim.x, u1 = units * (blockIdx.x + 1) / gridDim.x;
    // row of u0: the largest with q row (row + 1) / 2 <= u0
    uint32_t row = (uint32_t)((sqrt(8.0 * (double)(u0 / q) + 1.0) - 1.0) * 0.5);
    while ((uint64_t)q * row * (row + 1) / 2 > u0) --row;
    while ((uint64_t)q * (row + 1) * (row + 2) / 2 <= u0) ++row;
    uint32_t t = (uint32_t)(u0 - (uint64_t)q * row * (row + 1) / 2);  // tile of the row
    uint32_t j = 0;
    bool active = false, paired = false;  // paired: the row so far has pairs for this target
    nbfix::Fix3 p{};
    double mj = 0, ek = 0, ep = 0, acc = 0;
    bool load = true;
    for (uint64_t u = u0; u < u1; ++u) {
        if (load) {  // a row begins (or the CTA's range does)
            load = false;
            j = row * EN_THREADS + tid;
            active = j < n;
            mj = active ? m[j] : 0.0;
            if (active) {
                nbfix::split3(x[j], y[j], z[j], K, p);
                if (t == 0) {
                    const double v = vx[j] * vx[j] + vy[j] * vy[j] + vz[j] * vz[j];
                    ek += 0.5 * mj * v;
                }
            }
            acc = 0;
            paired = false;
        }
        const uint32_t i0 = t * tile;
        __syncthreads();
        if (tid < tile && i0 + tid < n) {
            const uint32_t i = i0 + tid;
            nbfix::Fix3 c;
            nbfix::split3(x[i], y[i], z[i], K, c);
            const double mi = G * m[i];  // first: m / r may overflow where G m m / r does not
            src[tid] = nbfix::FixRec{c.x2, c.y2, c.z2, (uint32_t)__double2hiint(mi),
                                     c.x1, c.y1, c.z1, (uint32_t)__double2loint(mi),
                                     c.x0, c.y0, c.z0, 0};
        }
        __syncthreads();
        const uint32_t cnt = active && j > i0 ? min(tile, j - i0) : 0u;
        paired = paired || cnt != 0;
#pragma unroll 1
        for (uint32_t ii = 0; ii < cnt; ++ii) {
            const nbfix::FixRec f = src[ii];
            const nbfix::Fix3 c{f.x2, f.y2, f.z2, f.x1, f.y1, f.z1, f.x0, f.y0, f.z0};
            nbfix::Sep s;
            double inv;
            if (usable && nbfix::separation(c, p, nbfix::SH_MAX, s)) {
                inv = nbfix::scaled_double(nbfix::rinv1(nbfix::norm2(s) + nbfix::NORM2_BIAS),
                                           1023 - K + s.sh);
            } else {
                const uint32_t i = i0 + ii;
                const double rx = x[j] - x[i], ry = y[j] - y[i], rz = z[j] - z[i];
                inv = nb_rsqrt_f64(fma(rx, rx, fma(ry, ry, rz * rz)));
            }
            acc = fma(__hiloint2double((int)f.mh, (int)f.ml), inv, acc);
        }
        if (++t == q * (row + 1) || u + 1 == u1) {  // the row (or the CTA's range) ends
            if (paired) ep = fma(mj, acc, ep);  // without pairs a mass of infinity adds nothing
            t = 0;
            ++row;
            load = true;
        }
    }
    // block reduction in a fixed order
    for (int off = 16; off > 0; off >>= 1) {
        ek += __shfl_down_sync(0xffffffffu, ek, off);
        ep += __shfl_down_sync(0xffffffffu, ep, off);
    }
    if ((tid & 31) == 0) {
        red_k[tid >> 5] = ek;
        red_p[tid >> 5] = ep;
    }
    __syncthreads();
    if (tid == 0) {
        double k2 = 0, p2 = 0;
        for (int w = 0; w < EN_THREADS / 32; ++w) {
            k2 += red_k[w];
            p2 += red_p[w];
        }
        part[blockIdx.x] = make_double2(k2, p2);
    }
}

// CTAs of an energy evaluation (its partials), at most `most`.
struct EnergyShape {
    uint32_t ctas, tile;
    uint64_t units;
};
EnergyShape energy_shape(uint32_t n, int sm_count, uint32_t most) {
    EnergyShape e;
    const uint64_t rows = (n + EN_THREADS - 1) / EN_THREADS, full = (uint64_t)sm_count * EN_CTAS_PER_SM;
    // smaller tiles where the rows alone do not give every CTA two units
    uint32_t q = 1;
    while (q < 8 && q * rows * (rows + 1) / 2 < 2 * full) q *= 2;
    e.tile = EN_THREADS / q;
    e.units = q * rows * (rows + 1) / 2;
    e.ctas = (uint32_t)std::min<uint64_t>(std::min<uint64_t>(full, most), e.units);
    return e;
}

// Adds the CTAs' partials. Most of an energy may sit in a few of them, next to which the up to 1,824
// partials and the levels of a tree would each leave a rounding of the whole; so they are added as
// 128-bit integers in units of 2^-111 of the largest one's power of two and rounded once. (In
// double-doubles the same took 6 us more at 300 bodies and 14 more at 3,001: FP64 instructions.)
constexpr int EF_THREADS = 256;

__device__ __forceinline__ uint32_t sum_exponent(double v) {  // of the units below, at least 1
    return max((uint32_t)__double2hiint(v) >> 20 & 0x7ffu, 1u);
}
// v in units of 2^(e - 1133), e at least its exponent; bits below are dropped
__device__ __forceinline__ __int128 sum_term(double v, uint32_t e) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    unsigned long long m = b & 0xfffffffffffffull;
    if ((b >> 52 & 0x7ff) != 0) m |= 1ull << 52;
    const uint32_t down = e - sum_exponent(v);
    __int128 t = down <= 58 ? (__int128)m << (58 - down) : (__int128)(down < 122 ? m >> (down - 58) : 0);
    return (long long)b < 0 ? -t : t;
}
__device__ __forceinline__ __int128 sum_over_lanes(__int128 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long lo =
            __shfl_xor_sync(0xffffffffu, (unsigned long long)(unsigned __int128)v, o);
        const long long hi = __shfl_xor_sync(0xffffffffu, (long long)(v >> 64), o);
        v += ((__int128)hi << 64) + (__int128)(unsigned __int128)lo;
    }
    return v;
}
__device__ double sum_value(__int128 v, uint32_t e) {  // v 2^(e - 1133), rounded to nearest
    unsigned __int128 a = v < 0 ? -(unsigned __int128)v : (unsigned __int128)v;
    int up = 0;  // a normalised to 64 bits, the bits below kept as one
    const unsigned long long h = (unsigned long long)(a >> 64);
    unsigned long long top = (unsigned long long)a;
    if (h != 0) {
        up = 64 - __clzll((long long)h);
        top = (unsigned long long)(a >> up) |
              ((a & (((unsigned __int128)1 << up) - 1)) != 0 ? 1ull : 0ull);
    }
    const double r = scalbn(__ull2double_rn(top), up + (int)e - 1133);
    return v < 0 ? -r : r;
}

__global__ void __launch_bounds__(EF_THREADS)
energy_finalize(const double2* __restrict__ part, uint32_t nparts, double* __restrict__ out) {
    __shared__ uint32_t exps[2][EF_THREADS / 32];
    __shared__ __int128 sums[2][EF_THREADS / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t ke = 1, pe = 1;
    for (uint32_t b = threadIdx.x; b < nparts; b += EF_THREADS) {
        const double2 v = part[b];
        ke = max(ke, sum_exponent(v.x));
        pe = max(pe, sum_exponent(v.y));
    }
    ke = __reduce_max_sync(0xffffffffu, ke);
    pe = __reduce_max_sync(0xffffffffu, pe);
    if (lane == 0) {
        exps[0][warp] = ke;
        exps[1][warp] = pe;
    }
    __syncthreads();
    ke = __reduce_max_sync(0xffffffffu, exps[0][lane % (EF_THREADS / 32)]);
    pe = __reduce_max_sync(0xffffffffu, exps[1][lane % (EF_THREADS / 32)]);
    __int128 k = 0, p = 0;
    for (uint32_t b = threadIdx.x; b < nparts; b += EF_THREADS) {
        const double2 v = part[b];
        k += sum_term(v.x, ke);
        p += sum_term(v.y, pe);
    }
    k = sum_over_lanes(k);
    p = sum_over_lanes(p);
    if (lane == 0) {
        sums[0][warp] = k;
        sums[1][warp] = p;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    k = p = 0;
    for (int w = 0; w < EF_THREADS / 32; ++w) {
        k += sums[0][w];
        p += sums[1][w];
    }
    double ek = sum_value(k, ke), u = sum_value(p, pe);
    if (ke == 0x7ff || pe == 0x7ff) {  // infinities and NaN among them: as FP64 adds them
        ek = u = 0.0;
        for (uint32_t b = 0; b < nparts; ++b) {
            ek += part[b].x;
            u += part[b].y;
        }
    }
    const double ep = -u;
    out[0] = ek;
    out[1] = ep;
    out[2] = ek + ep;
    out[3] = (2.0 * ek) / fabs(ep);
}

nb_status energy_launch(const EnergyShape& e, const double* m, const double* x, const double* y,
                        const double* z, const double* vx, const double* vy, const double* vz,
                        uint32_t n, double G, uint32_t* k_part, double2* part, double* out,
                        cudaStream_t stream) {
    uint32_t k_words = 0;
    NB_TRY(nb::launch_scale(x, y, z, n, k_part, &k_words, stream));
    energy_kernel<<<e.ctas, EN_THREADS, 0, stream>>>(m, x, y, z, vx, vy, vz, n, G, e.tile, e.units,
                                                     k_part, k_words, part);
    NB_TRY(nb::check_launch("energy_kernel"));
    energy_finalize<<<1, EF_THREADS, 0, stream>>>(part, e.ctas, out);
    return nb::check_launch("energy_finalize");
}

// ---------------------------------------------------------------------------------------------
// AABB: order-preserving integer images of the doubles make min/max integer-pipe work; every
// accumulator starts at the image of 0.0 (the reference's zero-initialised partials), the last
// block to finish reduces the per-block partials in a fixed order and applies the cube rule of
// BarnesHutOctree.cpp:161-190 with separately rounded IEEE operations.
// ---------------------------------------------------------------------------------------------
constexpr int AABB_THREADS = 256;
using nbaabb::MinMax6;
using nbaabb::cube_rule;
using nbaabb::ord_of;
using nbaabb::val_of;

// One word per block for nbfix::block_scale.
__global__ void __launch_bounds__(256)
scale_kernel(const double* __restrict__ x, const double* __restrict__ y,
             const double* __restrict__ z, uint32_t n, uint32_t* __restrict__ out) {
    __shared__ uint32_t most;
    if (threadIdx.x == 0) most = 0;
    __syncthreads();
    const uint32_t e = __reduce_max_sync(
        0xffffffffu,
        nbfix::max_exponent(x, y, z, n, blockIdx.x * 256 + threadIdx.x, gridDim.x * 256));
    if ((threadIdx.x & 31) == 0) atomicMax(&most, e);
    __syncthreads();
    if (threadIdx.x == 0) out[blockIdx.x] = most;
}

__global__ void __launch_bounds__(AABB_THREADS)
aabb_kernel(const double* x, const double* y,
            const double* z, uint32_t n, MinMax6* __restrict__ part,
            unsigned int* __restrict__ counter, double* __restrict__ out) {
    nb_grid_wait();
    const long long zero = ord_of(0.0);
    long long mn[3] = {zero, zero, zero}, mx[3] = {zero, zero, zero};
    const double* p[3] = {x, y, z};
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const long long o = ord_of(p[a][i]);
            mn[a] = min(mn[a], o);
            mx[a] = max(mx[a], o);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        for (int off = 16; off > 0; off >>= 1) {
            mn[a] = min(mn[a], __shfl_down_sync(0xffffffffu, mn[a], off));
            mx[a] = max(mx[a], __shfl_down_sync(0xffffffffu, mx[a], off));
        }
    }
    __shared__ MinMax6 warp_part[AABB_THREADS / 32];
    __shared__ bool last;
    if ((threadIdx.x & 31) == 0) {
        for (int a = 0; a < 3; ++a) {
            warp_part[threadIdx.x >> 5].v[a] = mn[a];
            warp_part[threadIdx.x >> 5].v[3 + a] = mx[a];
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        MinMax6 r = warp_part[0];
        for (int w = 1; w < AABB_THREADS / 32; ++w)
            for (int a = 0; a < 3; ++a) {
                r.v[a] = min(r.v[a], warp_part[w].v[a]);
                r.v[3 + a] = max(r.v[3 + a], warp_part[w].v[3 + a]);
            }
        part[blockIdx.x] = r;
        __threadfence();
        const unsigned int done = atomicAdd(counter, 1u);
        last = (done == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    // the last block reduces all blocks' partials with all its threads
    __threadfence();
    for (int a = 0; a < 3; ++a) {
        mn[a] = zero;
        mx[a] = zero;
    }
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
        const MinMax6 q = part[b];
        for (int a = 0; a < 3; ++a) {
            mn[a] = min(mn[a], q.v[a]);
            mx[a] = max(mx[a], q.v[3 + a]);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        for (int off = 16; off > 0; off >>= 1) {
            mn[a] = min(mn[a], __shfl_down_sync(0xffffffffu, mn[a], off));
            mx[a] = max(mx[a], __shfl_down_sync(0xffffffffu, mx[a], off));
        }
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        for (int a = 0; a < 3; ++a) {
            warp_part[threadIdx.x >> 5].v[a] = mn[a];
            warp_part[threadIdx.x >> 5].v[3 + a] = mx[a];
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        MinMax6 r = warp_part[0];
        for (int w = 1; w < AABB_THREADS / 32; ++w)
            for (int a = 0; a < 3; ++a) {
                r.v[a] = min(r.v[a], warp_part[w].v[a]);
                r.v[3 + a] = max(r.v[3 + a], warp_part[w].v[3 + a]);
            }
        cube_rule(val_of(r.v[0]), val_of(r.v[1]), val_of(r.v[2]), val_of(r.v[3]),
                  val_of(r.v[4]), val_of(r.v[5]), out);
        *counter = 0;  // ready for the next launch on this context
    }
}

}  // namespace

namespace nb {

// Words for nbfix::block_scale: none for systems that every CTA scans itself.
nb_status launch_scale(const double* x, const double* y, const double* z, uint32_t n,
                       uint32_t* k_part, uint32_t* k_words, cudaStream_t stream) {
    *k_words = 0;
    if (n <= nbfix::SCALE_SCAN_N) return NB_OK;
    *k_words = std::min<uint32_t>(nbfix::SCALE_WORDS, (uint32_t)nb::ceil_div(n, 1024));
    scale_kernel<<<*k_words, 256, 0, stream>>>(x, y, z, n, k_part);
    return nb::check_launch("scale_kernel");
}

// Enqueues the AABB of (x, y, z) into out_dev[7]. Used by nb_aabb and the tree build.
nb_status launch_aabb(nb_ctx* ctx, const double* x, const double* y, const double* z,
                      uint32_t n, double* out_dev, cudaStream_t stream) {
    int blocks = nb::ceil_div(n, AABB_THREADS * 4);
    if (blocks > ctx->sm_count * 4) blocks = ctx->sm_count * 4;
    if (blocks < 1) blocks = 1;
    void* part = nullptr;
    NB_TRY(nb::scratch(ctx, NB_SCRATCH_AABB, (size_t)blocks * sizeof(MinMax6), stream,
                       &part));
    NB_CUDA_TRY(nb::launch_after(aabb_kernel, blocks, AABB_THREADS, 0, stream, x, y, z, n,
                                 (MinMax6*)part, ctx->dev_counter + 0, out_dev));
    return NB_OK;
}

}  // namespace nb

extern "C" {

nb_status nb_leapfrog_kick_drift(nb_ctx* ctx, double* vhx, double* vhy, double* vhz,
                                 const double* vx, const double* vy, const double* vz, double* x,
                                 double* y, double* z, const double* ax, const double* ay,
                                 const double* az, uint32_t n, double dt, nb_stream_t stream) {
    NB_CHECK_CTX(ctx);
    if (n == 0) return NB_OK;
    if (!vhx || !vhy || !vhz || !vx || !vy || !vz || !x || !y || !z || !ax || !ay || !az)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_leapfrog_kick_drift: null array pointer");
    NB_CUDA_TRY(nb::launch_after(kick_drift_kernel, nb::ceil_div(n, EW_THREADS), EW_THREADS, 0,
                                 (cudaStream_t)stream, vhx, vhy, vhz, vx, vy, vz, x, y, z, ax, ay, az, n, dt));
    return NB_OK;
}

nb_status nb_leapfrog_kick(nb_ctx* ctx, double* vx, double* vy, double* vz, const double* vhx,
                           const double* vhy, const double* vhz, const double* ax,
                           const double* ay, const double* az, uint32_t n, double dt,
                           nb_stream_t stream) {
    NB_CHECK_CTX(ctx);
    if (n == 0) return NB_OK;
    if (!vhx || !vhy || !vhz || !vx || !vy || !vz || !ax || !ay || !az)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_leapfrog_kick: null array pointer");
    NB_CUDA_TRY(nb::launch_after(kick_kernel, nb::ceil_div(n, EW_THREADS), EW_THREADS, 0,
                                 (cudaStream_t)stream, vx, vy, vz, vhx, vhy, vhz, ax, ay, az, n, dt));
    return NB_OK;
}

nb_status nb_leapfrog_kick_kick_drift(nb_ctx* ctx, double* vx, double* vy, double* vz,
                                      double* vhx, double* vhy, double* vhz, double* x, double* y,
                                      double* z, const double* ax, const double* ay,
                                      const double* az, uint32_t n, double dt,
                                      nb_stream_t stream) {
    NB_CHECK_CTX(ctx);
    if (n == 0) return NB_OK;
    if (!vhx || !vhy || !vhz || !vx || !vy || !vz || !x || !y || !z || !ax || !ay || !az)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_leapfrog_kick_kick_drift: null pointer");
    NB_CUDA_TRY(nb::launch_after(kick_kick_drift_kernel, nb::ceil_div(n, EW_THREADS), EW_THREADS, 0,
                                 (cudaStream_t)stream, vx, vy, vz, vhx, vhy, vhz, x, y, z, ax, ay, az, n, dt));
    return NB_OK;
}

nb_status nb_energy(nb_ctx* ctx, const double* m, const double* x, const double* y,
                    const double* z, const double* vx, const double* vy, const double* vz,
                    uint32_t n, double G, double* out_dev, nb_stream_t stream) {
    NB_CHECK_CTX(ctx);
    if (!m || !x || !y || !z || !vx || !vy || !vz || !out_dev)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_energy: null pointer");
    if (n == 0) return nb::set_error(NB_ERR_INVALID_ARG, "nb_energy: n == 0");
    const EnergyShape e = energy_shape(n, ctx->sm_count, 0xffffffffu);
    const size_t part_bytes = (size_t)e.ctas * sizeof(double2);
    void* part = nullptr;
    NB_TRY(nb::scratch(ctx, NB_SCRATCH_ENERGY, part_bytes + nbfix::SCALE_WORDS * sizeof(uint32_t),
                       (cudaStream_t)stream, &part));
    return energy_launch(e, m, x, y, z, vx, vy, vz, n, G, (uint32_t*)((char*)part + part_bytes),
                         (double2*)part, out_dev, (cudaStream_t)stream);
}

nb_status nb_aabb(nb_ctx* ctx, const double* x, const double* y, const double* z, uint32_t n,
                  double* out_dev, nb_stream_t stream) {
    NB_CHECK_CTX(ctx);
    if (!x || !y || !z || !out_dev) return nb::set_error(NB_ERR_INVALID_ARG, "nb_aabb: null pointer");
    return nb::launch_aabb(ctx, x, y, z, n, out_dev, (cudaStream_t)stream);
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Energy without any allocation.
//
// Some callers cannot let this library allocate device memory: an application that reserves the
// GPU's memory up front for its own pool and forbids later cudaMalloc calls, or a time-critical
// loop that cannot pay for cudaMalloc's device-wide synchronisation and unpredictable latency.
// nb_energy needs a context (whose creation allocates) and grows per-block scratch on demand;
// nb_energy_noalloc runs the same kernels with their per-block partial sums and scale words in the
// fixed array below instead. Nothing in the array needs clearing between calls: every call writes each
// partial it later reads. All calls share the array, so calls that overlap on the GPU (two
// streams, two host threads) race and must be serialised by the caller.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr uint32_t NOALLOC_MAX_BLOCKS = 8192;  // 8192 * 16 B = 128 KiB of scratch per device

// Per-block (kinetic, potential) partials. Every GPU that loads the library holds this array
// until the process exits. Host code must not pass the symbol itself to a kernel: its host-side
// name is only a stand-in, so the device address is looked up once per device below.
static __device__ __align__(256) double2 g_energy_noalloc_partials[NOALLOC_MAX_BLOCKS];
constexpr uint32_t NOALLOC_K_AT = NOALLOC_MAX_BLOCKS - nbfix::SCALE_WORDS / 4;  // scale words at the end

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};

// Device address of the partials array on the current device (looked up on first use).
nb_status noalloc_partials(double2** out) {
    int dev = -1;
    NB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES)
        return nb::set_error(NB_ERR_UNSUPPORTED, "nb_energy_noalloc: device %d not supported", dev);
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_energy_noalloc_partials);
        if (e != cudaSuccess) return nb::cuda_error(e, "nb_energy_noalloc: cudaGetSymbolAddress");
        g_noalloc_addr[dev] = p;
    }
    *out = (double2*)g_noalloc_addr[dev];
    return NB_OK;
}

}  // namespace

extern "C" {

nb_status nb_energy_noalloc(const double* m, const double* x, const double* y, const double* z,
                            const double* vx, const double* vy, const double* vz, uint32_t n,
                            double G, double* out_dev, nb_stream_t stream) {
    if (!m || !x || !y || !z || !vx || !vy || !vz || !out_dev)
        return nb::set_error(NB_ERR_INVALID_ARG, "nb_energy_noalloc: null pointer");
    if (n == 0) return nb::set_error(NB_ERR_INVALID_ARG, "nb_energy_noalloc: n == 0");
    if (n > NB_ENERGY_NOALLOC_MAX_N)
        return nb::set_error(NB_ERR_INVALID_ARG,
                             "nb_energy_noalloc: n = %u exceeds the fixed scratch limit of %u "
                             "bodies; use nb_energy", n, (unsigned)NB_ENERGY_NOALLOC_MAX_N);
    double2* part = nullptr;
    NB_TRY(noalloc_partials(&part));
    int dev = 0, sms = 0;
    NB_CUDA_TRY(cudaGetDevice(&dev));
    NB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return energy_launch(energy_shape(n, sms, NOALLOC_K_AT), m, x, y, z, vx, vy, vz, n, G,
                         (uint32_t*)(part + NOALLOC_K_AT), part, out_dev, (cudaStream_t)stream);
}

}  // extern "C"
