// nb_fix.cuh -- FP64-accurate pair arithmetic on the integer pipes.
//
// This part runs an FP64 instruction 75 times slower than an FP32 one (1.67 lanes per clock and SM
// measured, against 64 for 32-bit integer operations and 32 for 32 x 32 -> 64-bit multiply-adds),
// so a pair's separation, r^2 + eps^2 and m r^-3 are computed in fixed point and only the sums
// (one DFMA per axis) stay on the FP64 pipe.
//
//  * Coordinates: 96-bit two's complement multiples of 2^(K - 93), K chosen so that every
//    coordinate is below 2^K. A double above 2^(K - 41) is represented exactly, a smaller one is
//    rounded to 2^(K - 94) where it has lower bits, and marked.
//  * A pair: the three exact differences as magnitudes, shifted left by a common `sh` until the
//    largest is in [2^29, 2^30) by its first word; r^2 + eps^2 as a 64-bit integer D in [2^60,
//    2^64) (truncation errors below 2^-55 of it, centred); r^-3 from an estimate Y of D^(-1/2) good
//    to 2^-28 (MUFU and one Newton step), its residual e = 1 - D Y^2, of which 32 bits remain, and
//    Y^3 (1 + 3e/2) (dropped terms below 2^-55), times the mass's 53 bits, rounded once to a
//    double. In all within 2^-52.2 of exact, root mean square 2^-54.2 (the final rounding alone:
//    2^-54.4).
//  * What the integers cannot hold is left to the caller's FP64 expressions: a pair closer than
//    2^(K - 29), a component below 2^(K - 38) between bodies one of which is marked as rounded (so
//    small components keep their own relative accuracy), masses that are not positive normal
//    numbers, coordinates outside 2^K, scales beyond the exponent range, eps^2 too large for the
//    scale.
//
// Everything up to the device-only part also compiles as plain C++, for the CPU tests.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define NB_FIX_FN __host__ __device__ __forceinline__
#else
#define NB_FIX_FN inline
#endif
#ifdef __CUDA_ARCH__
#define NB_FIX_DEV 1
#else
#define NB_FIX_DEV 0
#endif

namespace nbfix {

constexpr int NO_EXP = INT32_MIN;   // FixRec::e of a source the FP64 expressions must handle
constexpr int ZERO_MASS = NO_EXP + 1;  // FixRec::e of a massless source with fitting coordinates
constexpr int K_MAX = 300;          // |K| beyond this: FP64 expressions for everything
constexpr int SH_MAX = 29;          // largest common shift

// A source: coordinate words (most significant first), the mass's mantissa (64 bits, top bit set,
// the lowest 11 clear but for bit 0, which marks rounded coordinates; it moves the truncated mass
// product by less than 1/8 of its last unit) and its biased exponent - 3 K.
struct alignas(16) FixRec {
    uint32_t x2, y2, z2, mh;
    uint32_t x1, y1, z1, ml;
    uint32_t x0, y0, z0;
    int e;
};

// The same as it is stored: a 32-byte half (one load) and a 16-byte half {x0, y0, z0, ml}.
struct alignas(32) FixHi {
    uint32_t x2, y2, z2, mh, x1, y1, z1;
    int e;
};

struct Fix3 {
    uint32_t x2, y2, z2, x1, y1, z1, x0, y0, z0;
    uint32_t rounded;  // bit 0: a coordinate has bits below the last word's
};

NB_FIX_FN uint64_t bits_of(double v) {
#if NB_FIX_DEV
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    std::memcpy(&u, &v, 8);
    return u;
#endif
}
NB_FIX_FN double double_of(uint32_t hi, uint32_t lo) {
#if NB_FIX_DEV
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo;
    double v;
    std::memcpy(&v, &u, 8);
    return v;
#endif
}
NB_FIX_FN uint32_t float_bits(float v) {
#if NB_FIX_DEV
    return __float_as_uint(v);
#else
    uint32_t u;
    std::memcpy(&u, &v, 4);
    return u;
#endif
}
// the high word of (hi:lo) << (s & 31)
NB_FIX_FN uint32_t fsl(uint32_t lo, uint32_t hi, uint32_t s) {
#if NB_FIX_DEV
    return __funnelshift_l(lo, hi, s);
#else
    s &= 31;
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}
NB_FIX_FN int clz32(uint32_t v) {
#if NB_FIX_DEV
    return __clz((int)v);
#else
    return v ? __builtin_clz(v) : 32;
#endif
}
// the position of the highest bit of v, all ones for 0
NB_FIX_FN uint32_t top_bit(uint32_t v) {
#if NB_FIX_DEV
    uint32_t p;
    asm("bfind.u32 %0, %1;" : "=r"(p) : "r"(v));
    return p;
#else
    return v ? 31u - (uint32_t)__builtin_clz(v) : 0xffffffffu;
#endif
}
NB_FIX_FN float rsqrt_est(float v) {
#if NB_FIX_DEV
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(v));
    return y;
#else
    return 1.0f / sqrtf(v);
#endif
}
// the high word of a * b
NB_FIX_FN uint32_t mul_hi(uint32_t a, uint32_t b) {
#if NB_FIX_DEV
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
NB_FIX_FN int mul_hi(int a, int b) {
#if NB_FIX_DEV
    return __mulhi(a, b);
#else
    return (int)(((int64_t)a * b) >> 32);
#endif
}
// a - b over three words
NB_FIX_FN void sub96(uint32_t a2, uint32_t a1, uint32_t a0, uint32_t b2, uint32_t b1, uint32_t b0,
                     uint32_t& d2, uint32_t& d1, uint32_t& d0) {
#if NB_FIX_DEV
    asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
        : "=r"(d0), "=r"(d1), "=r"(d2)
        : "r"(a0), "r"(a1), "r"(a2), "r"(b0), "r"(b1), "r"(b2));
#else
    const uint64_t l = (uint64_t)a0 - b0;
    const uint64_t m = (uint64_t)a1 - b1 - (l >> 63);
    d0 = (uint32_t)l;
    d1 = (uint32_t)m;
    d2 = a2 - b2 - (uint32_t)(m >> 63);
#endif
}

// K of a set of coordinates: the smallest with every |v| below 2^K (v_max = the largest |v|).
// Outside +-K_MAX the scale is unusable.
NB_FIX_FN int k_of(double v_max) { return (int)((bits_of(v_max) >> 52) & 0x7ff) - 1022; }
NB_FIX_FN bool k_usable(int K) { return K >= -K_MAX && K <= K_MAX; }

// A tree's box: [0..6] its AABB (nb_aabb), [7..9] the centre and [10], [11] the scale of its records:
// K, and K again with the FP32 edge^2 as the bits of one double. From the AABB, by calls 0 to 3 (of
// four threads: none reads what another writes).
constexpr int BOX_WORDS = 12;
NB_FIX_FN void box_extras(double* box, uint32_t i) {
    if (i < 3) box[7 + i] = box[i] + box[6] / 2;
    if (i == 3) {
        uint64_t v = 0;  // the largest |coordinate|
        for (int k = 0; k < 6; ++k) {
            const uint64_t u = bits_of(box[k]) & 0x7fffffffffffffffull;
            v = u > v ? u : v;
        }
        const int K = k_of(double_of((uint32_t)(v >> 32), (uint32_t)v));
        box[10] = (double)K;
        box[11] = double_of((uint32_t)K, float_bits((float)(box[6] * box[6])));
    }
}

// The words of v as a multiple of 2^(K - 93), rounded to nearest where v has lower bits, which are
// or'ed into `lost`; false when v is not finite or beyond 2^K.
NB_FIX_FN bool split96(double v, int K, uint32_t& w2, uint32_t& w1, uint32_t& w0, uint32_t& lost) {
    const uint64_t u = bits_of(v);
    const uint32_t uh = (uint32_t)(u >> 32), ul = (uint32_t)u;
    const int be = (int)((uh >> 20) & 0x7ff);
    const int s = be - 982 - K;  // v = mantissa * 2^(be - 1075) = mantissa * 2^s units
    // the 53-bit mantissa shifted left by s + 64 in five words, of which the upper three stay and
    // the top bit of the second rounds
    const bool in = s >= -53 && be != 0;
    const uint32_t mh = (uh & 0xfffffu) | 0x100000u, r = (uint32_t)(s + 64) & 31u,
                   q = in ? (uint32_t)(s + 64) >> 5 : 4u;
    const uint32_t a0 = ul << r, a1 = fsl(ul, mh, r), a2 = fsl(mh, 0, r);
    w0 = q == 0 ? a2 : q == 1 ? a1 : q == 2 ? a0 : 0u;
    w1 = q == 1 ? a2 : q == 2 ? a1 : q == 3 ? a0 : 0u;
    w2 = q == 2 ? a2 : q == 3 ? a1 : 0u;
    const uint32_t half = (q == 0 ? a1 : q == 1 ? a0 : 0u) >> 31;
    lost |= q == 0 ? a0 | a1 : q == 1 ? a0 : in ? 0u : (uh << 1) | ul;
    // plus the half; negative values as the complement plus one
    const uint32_t neg = (uint32_t)((int)uh >> 31);
    const uint64_t t = (uint64_t)w0 + half;
    uint64_t c = (uint64_t)((uint32_t)t ^ neg) + (neg & 1u);
    const uint64_t t1 = (uint64_t)w1 + (t >> 32);
    w0 = (uint32_t)c;
    c = (uint64_t)((uint32_t)t1 ^ neg) + (c >> 32);
    w1 = (uint32_t)c;
    w2 = ((w2 + (uint32_t)(t1 >> 32)) ^ neg) + (uint32_t)(c >> 32);
    return be != 0x7ff && (s < 41 || (s == 41 && (uh & 0xfffffu) == 0 && ul == 0));
}

NB_FIX_FN bool split3(double x, double y, double z, int K, Fix3& f) {
    uint32_t lost = 0;
    const bool a = split96(x, K, f.x2, f.x1, f.x0, lost);
    const bool b = split96(y, K, f.y2, f.y1, f.y0, lost);
    const bool c = split96(z, K, f.z2, f.z1, f.z0, lost);
    f.rounded = lost != 0 ? 1u : 0u;
    return a && b && c && k_usable(K);
}

// The mantissa and exponent of a mass; false when it is not a positive normal number.
NB_FIX_FN bool split_mass(double m, uint32_t& mh, uint32_t& ml, int& biased) {
    const uint64_t u = bits_of(m);
    biased = (int)(u >> 52);
    const uint64_t mant = (u << 11) | (1ull << 63);
    mh = (uint32_t)(mant >> 32);
    ml = (uint32_t)mant;
    return biased >= 1 && biased < 0x7ff;
}

NB_FIX_FN FixRec make_rec(double x, double y, double z, double m, int K) {
    FixRec r;
    Fix3 f;
    int be;
    const bool ok = split3(x, y, z, K, f);
    const bool mk = split_mass(m, r.mh, r.ml, be);
    r.ml |= f.rounded;
    r.x2 = f.x2;
    r.y2 = f.y2;
    r.z2 = f.z2;
    r.x1 = f.x1;
    r.y1 = f.y1;
    r.z1 = f.z1;
    r.x0 = f.x0;
    r.y0 = f.y0;
    r.z0 = f.z0;
    r.e = !ok ? NO_EXP : (mk ? be - 3 * K : (m == 0.0 ? ZERO_MASS : NO_EXP));
    return r;
}

// eps^2 in units of D at shift sh: D counts 4^(K - 30 - sh).
NB_FIX_FN double eps2_units(double eps2, int K, int sh) {
    return eps2 * double_of((uint32_t)(1023 + 2 * (sh + 30 - K)) << 20, 0);  // |K| <= K_MAX
}
constexpr double EPS2_LIMIT = 4611686018427387904.0;  // 2^62: eps^2 in units of D stays below

// A pair's separation: per axis the sign (0 or all ones), the magnitude shifted by sh (two words;
// complements of negative values, one unit of the exact difference's last word short) and the
// difference's unshifted last word.
struct Sep {
    uint32_t xs, ys, zs, xh, yh, zh, xl, yl, zl, x0, y0, z0;
    int sh;
};

// c - p, normalised; false when the pair is too close for the integers (the caller's FP64
// expressions then).
NB_FIX_FN bool separation(const Fix3& c, const Fix3& p, int sh_max, Sep& s) {
    uint32_t x2, x1, y2, y1, z2, z1;
    sub96(c.x2, c.x1, c.x0, p.x2, p.x1, p.x0, x2, x1, s.x0);
    sub96(c.y2, c.y1, c.y0, p.y2, p.y1, p.y0, y2, y1, s.y0);
    sub96(c.z2, c.z1, c.z0, p.z2, p.z1, p.z0, z2, z1, s.z0);
    s.xs = (uint32_t)((int)x2 >> 31);
    s.ys = (uint32_t)((int)y2 >> 31);
    s.zs = (uint32_t)((int)z2 >> 31);
    const uint32_t t = (x2 ^ s.xs) | (y2 ^ s.ys) | (z2 ^ s.zs);  // below 2^30
    const int n = 29 - (int)top_bit(t);
    const int sh = n < sh_max ? n : sh_max;
    s.sh = sh;
    s.xh = fsl(x1, x2, sh) ^ s.xs;
    s.yh = fsl(y1, y2, sh) ^ s.ys;
    s.zh = fsl(z1, z2, sh) ^ s.zs;
    s.xl = fsl(s.x0, x1, sh) ^ s.xs;
    s.yl = fsl(s.y0, y1, sh) ^ s.ys;
    s.zl = fsl(s.z0, z1, sh) ^ s.zs;
    return t != 0;
}

// Truncation of norm2 in its own units, on average: 4/3 per axis (the squares of the low words) and
// 4 per axis (the halves of the cross products).
constexpr uint32_t NORM2_BIAS = 16;

// r^2 in units 4^(K - 30 - sh), truncated by 0 to 36 units: 4 times the squares of the first words
// and 8 times their products with the second words.
NB_FIX_FN uint64_t norm2(const Sep& s) {
    const uint64_t r = (uint64_t)s.xh * s.xh + (uint64_t)s.yh * s.yh + (uint64_t)s.zh * s.zh;
    const uint32_t h = mul_hi(s.xh, s.xl) + mul_hi(s.yh, s.yl) + mul_hi(s.zh, s.zl);
    return (r << 2) + ((uint64_t)h << 3);
}

// Y ~ 2^61 D^(-1/2) to 2^-28 and below 2^31 (the rounded estimate reaches 2^31 for D up to
// 2^60 + 2^32, where one unit less is as good: its users multiply it as a signed word), and
// e = 1 - D Y^2 / 2^122 in units 2^-58 (|e| < 2^31); W = Y^2. D Y^2 is so near 2^122 that of its upper
// half only the low 32 bits are formed.
NB_FIX_FN int rsqrt_residual(uint64_t D, uint32_t& Y, uint64_t& W) {
    const uint32_t dh = (uint32_t)(D >> 32), dl = (uint32_t)D;
    const float f = rsqrt_est((float)dh) * 35184372088832.0f;  // 2^45: at most 2^31
#if NB_FIX_DEV
    const int y0 = __float2int_rz(f);  // saturates
#else
    const int y0 = f < 2147483648.0f ? (int)f : 2147483647;
#endif
    // the estimate's own residual to 2^-31: D y0^2 / 2^64 = 2^58 (1 - e0), |e0| < 2^-20
    const uint64_t w0 = (uint64_t)(uint32_t)y0 * (uint32_t)y0;
    const uint64_t p = (uint64_t)dh * (uint32_t)(w0 >> 32) + mul_hi(dh, (uint32_t)w0);
    const int ne0 = (int)(fsl((uint32_t)p, (uint32_t)(p >> 32), 5) ^ 0x80000000u);  // -e0 2^31
    Y = (uint32_t)(y0 - (int)(((int64_t)y0 * ne0 + 0x80000000ll) >> 32));  // rounded
    Y = Y < 0x7fffffffu ? Y : 0x7fffffffu;
    W = (uint64_t)Y * Y;
    const uint32_t wh = (uint32_t)(W >> 32), wl = (uint32_t)W;
    return -(int)(dh * wh + mul_hi(dh, wl) + mul_hi(dl, wh) + 1u);
}

// D^(-3/2) 2^151 (between 2^55 and 2^61): Y^2 (Y + 3eY/2), the correction below Y's last bit
NB_FIX_FN uint64_t rinv3(uint64_t D) {
    uint32_t Y;
    uint64_t W;
    const int e = rsqrt_residual(D, Y, W);
    const uint64_t c = (uint64_t)(((int64_t)(int)Y * (e + (e >> 1))) >> 26);  // in units 2^-32 of Y's
    const uint32_t yh = Y + (uint32_t)(c >> 32), yl = (uint32_t)c;
    const uint32_t wh = (uint32_t)(W >> 32), wl = (uint32_t)W;
    return (uint64_t)wh * yh + mul_hi(wl, yh) + mul_hi(wh, yl);
}

// D^(-1/2) 2^93 (between 2^61 and 2^63): Y (1 + e/2)
NB_FIX_FN uint64_t rinv1(uint64_t D) {
    uint32_t Y;
    uint64_t W;
    const int e = rsqrt_residual(D, Y, W);
    return ((uint64_t)Y << 32) + (uint64_t)(((int64_t)(int)Y * e) >> 27);
}

// A 64-bit integer v > 0 as a double scaled so that 2^63 has the biased exponent `be`,
// rounded to nearest.
NB_FIX_FN double scaled_double(uint64_t v, int be) {
    const uint32_t vh = (uint32_t)(v >> 32), vl = (uint32_t)v;
    const int n = clz32(vh);
    const uint32_t h = fsl(vl, vh, n), l = vl << n;
    const uint32_t r = (l >> 10) & 1u;
    uint64_t o = ((uint64_t)((((uint32_t)(be - n - 1)) << 20) + (h >> 11)) << 32) |
                 ((h << 21) | (l >> 11));
    o += r;
    return double_of((uint32_t)(o >> 32), (uint32_t)o);
}

// The same for 2^32 <= v < 2^62: the half added before the last shift cannot carry out.
NB_FIX_FN double scaled_double_62(uint64_t v, int be) {
    const uint32_t vh = (uint32_t)(v >> 32), vl = (uint32_t)v;
    const uint32_t p = top_bit(vh), n = 30u - p;
    const uint64_t o = (((uint64_t)fsl(vl, vh, n) << 32) | (vl << n)) + 0x200u;
    const uint32_t mh = (uint32_t)(o >> 32), ml = (uint32_t)o;
    return double_of(((uint32_t)(be - 32 + (int)p) << 20) + (mh >> 10), (mh << 22) | (ml >> 10));
}

// m D^(-3/2) for a source's mass and exponent word: the double; `ok` false when its exponent
// leaves the normal range.
NB_FIX_FN double mass_rinv3(uint64_t S, uint32_t mh, uint32_t ml, int e, int sh, bool& ok) {
    const uint32_t s_h = (uint32_t)(S >> 32), s_l = (uint32_t)S;
    const uint64_t F = (uint64_t)s_h * mh + mul_hi(s_h, ml) + mul_hi(s_l, mh);
    const int be = e + 3 * sh + 3;  // exponent of 2^63; F is below 2^61 and above 2^53
    ok = (uint32_t)(be - 16) < 2016u;
    return scaled_double_62(F, be);
}

// One axis of the separation as a double (its sign and its two words rounded to 53 bits); base =
// 993 + K - sh in the exponent's place. Components with 2^20 or more in the first word have at least
// 53 bits in two words; pairs whose largest one is below 2^29 there (an eps^2 far above r^2 limits the
// shift) take the third word as well. Truncated to 53 bits instead (and so one unit short for negative
// differences that a double holds), accelerations came out 9e-17 low on average; rounding costs 1 to
// 2.5% (16,384 bodies 1.744 -> 1.771 ms).
constexpr uint32_t AXIS_TWO_WORDS = 1u << 20, AXIS_LARGEST = 1u << 29;
NB_FIX_FN double axis(uint32_t s, uint32_t h, uint32_t l, uint32_t base) {
    const uint32_t p = top_bit(h), n = 30u - p;
    const uint64_t v = (((uint64_t)fsl(l, h, n) << 32) | (l << n)) + 0x200u;  // as above
    const uint32_t mh = (uint32_t)(v >> 32), ml = (uint32_t)v;
    const uint32_t hi = base + (p << 20) + (mh >> 10);
    return double_of(hi | (s & 0x80000000u), (mh << 22) | (ml >> 10));
}

// Any component, x = the third word: where the first word is 0 the complement's missing unit is
// added back.
NB_FIX_FN double axis_small(uint32_t s, uint32_t h, uint32_t l, uint32_t x, int base) {
    if (h == 0) {
        const uint64_t v = (((uint64_t)l << 32) | x) + (s & 1u);
        if (v == 0) {
            if (s == 0) return 0.0;
            h = 1;  // -2^64 units
            l = 0;
        } else {
            h = (uint32_t)(v >> 32);
            l = (uint32_t)v;
            base -= 32;
            if (h == 0) {
                h = l;
                l = 0;
                base -= 32;
            }
        }
        x = 0;
    }
    const int n = clz32(h);
    const uint32_t mh = fsl(l, h, n), ml = fsl(x, l, n);
    uint64_t o = ((uint64_t)(((uint32_t)(base - n - 1) << 20) + (mh >> 11)) << 32) |
                 ((mh << 21) | (ml >> 11));
    o += (ml >> 10) & 1u;
    return double_of((uint32_t)(o >> 32) | (s & 0x80000000u), (uint32_t)o);
}

// Whether a component is below 2^55 units: then a rounded coordinate may have cost it bits that a
// double holds.
NB_FIX_FN bool axis_tiny(uint32_t h, uint32_t l, int sh) {
    return ((((uint64_t)h << 32) | l) >> (23 + sh)) == 0;
}

// False when a component needs the coordinates' own bits (`rounded`: either body's mark).
NB_FIX_FN bool axes(const Sep& s, int K, double& dx, double& dy, double& dz,
                    uint32_t rounded = 0) {
    const int base = 1025 + K - s.sh;
    bool fits = true;
    uint32_t least = s.xh < s.yh ? s.xh : s.yh;
    least = least < s.zh ? least : s.zh;
    if (least >= AXIS_TWO_WORDS && (s.xh | s.yh | s.zh) >= AXIS_LARGEST) {
        const uint32_t b = (uint32_t)(base - 32) << 20;
        dx = axis(s.xs, s.xh, s.xl, b);
        dy = axis(s.ys, s.yh, s.yl, b);
        dz = axis(s.zs, s.zh, s.zl, b);
    } else {
        if (rounded != 0)
            fits = !(axis_tiny(s.xh, s.xl, s.sh) || axis_tiny(s.yh, s.yl, s.sh) ||
                     axis_tiny(s.zh, s.zl, s.sh));
        dx = axis_small(s.xs, s.xh, s.xl, (s.x0 << s.sh) ^ s.xs, base);
        dy = axis_small(s.ys, s.yh, s.yl, (s.y0 << s.sh) ^ s.ys, base);
        dz = axis_small(s.zs, s.zh, s.zl, (s.z0 << s.sh) ^ s.zs, base);
    }
    return fits;
}

#ifdef __CUDACC__
// eps^2 per shift, filled by one warp of a block (the caller's __syncthreads() follows).
struct Eps2Table {
    uint64_t units[32];
    int sh_max;  // -1: the FP64 expressions for every pair
};
__device__ __forceinline__ void fill_eps2(Eps2Table& t, double eps2, int K) {
    if (threadIdx.x >= 32) return;
    const int sh = (int)threadIdx.x;
    const double u = sh <= SH_MAX && k_usable(K) ? eps2_units(eps2, K, sh) : -1.0;
    const bool fits = u >= 0.0 && u < EPS2_LIMIT;
    t.units[sh] = fits ? __double2ull_rn(u) + NORM2_BIAS : 0;
    const uint32_t b = __ballot_sync(0xffffffffu, fits);  // a run from bit 0
    if (sh == 0) t.sh_max = __clz((int)~__brev(b)) - 1;
}

// Factor w = m (r^2 + eps^2)^(-3/2) and separation of a source seen from p: every sum is
// fma(w, d, sum). False when the caller has to evaluate the pair in FP64. sh_max >= 0.
// (A form without branches, two or four pairs interleaved, measured 20% slower: it does more work
// per pair and the chip is not short of warps.)
__device__ __forceinline__ bool term(const FixRec& f, const Fix3& p, int K, const Eps2Table& t,
                                     int sh_max, double& w, double& dx, double& dy, double& dz) {
    if (f.e <= ZERO_MASS) return false;
    const Fix3 c{f.x2, f.y2, f.z2, f.x1, f.y1, f.z1, f.x0, f.y0, f.z0};
    Sep s;
    if (!separation(c, p, sh_max, s)) return false;
    const uint64_t D = norm2(s) + t.units[s.sh];  // with norm2's bias
    bool ok;
    w = mass_rinv3(rinv3(D), f.mh, f.ml, f.e, s.sh, ok);
    const bool fits = axes(s, K, dx, dy, dz, (f.ml | p.rounded) & 1u);
    return ok && fits;
}

// Whether a pair that term() refuses adds exactly 0 in the FP64 expressions too: a massless source,
// or a body paired with itself (`self`), whose separation is 0, with a finite factor either way
// (eps^2 and the mass far from the exponent limits). The target fits the fixed point (sh_max >= 0).
__device__ __forceinline__ bool adds_nothing(const FixRec& f, bool self, int K, int sh_max,
                                             double eps2) {
    return sh_max >= 0 && eps2 > 1e-60 &&
           (f.e == ZERO_MASS || (self && f.e > ZERO_MASS && f.e + 3 * K < 1600));
}

// The scale of a system whose coordinates a kernel reads directly: the largest exponent, from
// k_part[0 .. k_words) (nb::launch_scale) or, for small systems (k_words = 0), by a scan of the
// bodies in every block. All threads of the block call it.
constexpr uint32_t SCALE_SCAN_N = 2048;
constexpr uint32_t SCALE_WORDS = 128;

// Largest biased exponent of the coordinates of bodies b0, b0 + step, ...
__device__ __forceinline__ uint32_t max_exponent(const double* __restrict__ x,
                                                 const double* __restrict__ y,
                                                 const double* __restrict__ z, uint32_t n,
                                                 uint32_t b0, uint32_t step) {
    uint32_t e = 0;
    for (uint32_t b = b0; b < n; b += step) {
        const uint32_t h = max((uint32_t)__double2hiint(x[b]) & 0x7fffffffu,
                               max((uint32_t)__double2hiint(y[b]) & 0x7fffffffu,
                                   (uint32_t)__double2hiint(z[b]) & 0x7fffffffu));
        e = max(e, h >> 20);
    }
    return e;
}

__device__ __forceinline__ int block_scale(const double* __restrict__ x,
                                           const double* __restrict__ y,
                                           const double* __restrict__ z, uint32_t n,
                                           const uint32_t* __restrict__ k_part,
                                           uint32_t k_words) {
    __shared__ uint32_t most;
    if (threadIdx.x == 0) most = 0;
    __syncthreads();
    uint32_t e = 0;
    if (k_words == 0) {
        e = max_exponent(x, y, z, n, threadIdx.x, blockDim.x);
    } else {
        for (uint32_t k = threadIdx.x; k < k_words; k += blockDim.x) e = max(e, k_part[k]);
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&most, e);
    __syncthreads();
    return (int)most - 1022;
}
#endif

}  // namespace nbfix
