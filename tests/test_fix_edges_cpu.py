"""The fixed-point pair arithmetic of nb_fix.cuh (as plain C++) where its words are at their limits,
against 80-digit decimal arithmetic."""

import ctypes as C
import os
import random
import subprocess
from decimal import Decimal, getcontext

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "nb_fix.cuh"
using namespace nbfix;
extern "C" void inverse_powers(uint64_t D, uint64_t* out) {
    out[0] = rinv3(D);
    out[1] = rinv1(D);
}
// out: w, dx, dy, dz, 1 / sqrt(r^2 + eps^2); returns 0 when the pair needs the FP64 expressions
extern "C" int fix_pair(const double* c, const double* p, double m, double eps2, double v_max,
                        double* out) {
    const int K = k_of(v_max);
    Fix3 P;
    const FixRec r = make_rec(c[0], c[1], c[2], m, K);
    if (!split3(p[0], p[1], p[2], K, P) || r.e <= ZERO_MASS) return 0;
    int sh_max = -1;
    while (sh_max < SH_MAX && eps2 >= 0 && eps2_units(eps2, K, sh_max + 1) < EPS2_LIMIT) ++sh_max;
    if (sh_max < 0) return 0;
    Sep s;
    const Fix3 q{r.x2, r.y2, r.z2, r.x1, r.y1, r.z1, r.x0, r.y0, r.z0};
    if (!separation(q, P, sh_max, s)) return 0;
    const uint64_t D = norm2(s) + (uint64_t)(eps2_units(eps2, K, s.sh) + 0.5) + NORM2_BIAS;
    bool ok;
    out[0] = mass_rinv3(rinv3(D), r.mh, r.ml, r.e, s.sh, ok);
    const bool fits = axes(s, K, out[1], out[2], out[3], (r.ml | P.rounded) & 1u);
    out[4] = scaled_double(rinv1(D), 1023 - K + s.sh);
    return ok && fits;
}
"""


@pytest.fixture(scope="module")
def fix(tmp_path_factory):
    d = tmp_path_factory.mktemp("fix")
    (d / "fix.cpp").write_text(SOURCE)
    so = str(d / "libfix.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "n-body-simulation_gb300", "csrc"), str(d / "fix.cpp"), "-o",
                    so], check=True)
    lib = C.CDLL(so)
    lib.inverse_powers.argtypes = [C.c_uint64, C.POINTER(C.c_uint64)]
    lib.fix_pair.argtypes = [C.POINTER(C.c_double)] * 2 + [C.c_double] * 3 + [C.POINTER(C.c_double)]
    getcontext().prec = 80
    return lib


def pair(fix, c, p, m, eps2, v_max):
    out = (C.c_double * 5)()
    ok = fix.fix_pair((C.c_double * 3)(*c), (C.c_double * 3)(*p), m, eps2, v_max, out)
    return list(out) if ok else None


# D^(-3/2) and D^(-1/2): the estimate leaves D's low word out (2^-29 of it) and is rounded to an integer
# of at least 2^29 (or clamped one unit below 2^31), so its residual is about 2^-28 and the dropped terms
# 15/8 and 3/8 of 2^-56; D^(-3/2) 2^151 is at least 2^55 and truncated by less than 3 units, D^(-1/2) 2^93
# at least 2^61 and by one.
@pytest.mark.parametrize("base", [1 << 60, (1 << 60) + (1 << 32), 1 << 61, 1 << 62, 3 << 62, (1 << 64) - 1])
def test_inverse_powers_at_the_limits(fix, base):
    rng = random.Random(base)
    out = (C.c_uint64 * 2)()
    for i in range(2000):
        step = int(2.0 ** rng.uniform(0, 34)) if i else 0
        for D in (base + step, base - step):
            if not 1 << 60 <= D < 1 << 64:
                continue
            fix.inverse_powers(D, out)
            root = Decimal(D).sqrt()
            assert abs(Decimal(out[0]) * Decimal(D) * root / Decimal(1 << 151) - 1) <= Decimal(2.0 ** -52.9)
            assert abs(Decimal(out[1]) * root / Decimal(1 << 93) - 1) <= Decimal(2.0 ** -56.0)


def test_pairs_at_powers_of_two(fix):
    """r^2 + eps^2 at and just above powers of four, along each axis and in both directions. Bounds
    of test_pairs_against_decimal in test_fix_cpu.py."""
    rng = random.Random(11)
    for i in range(6000):
        j = rng.randint(-20, 3)
        d = 2.0 ** j * (1.0 + (0.0 if i % 5 == 0 else 2.0 ** -rng.uniform(27, 52)))
        eps2 = 0.0 if i % 3 == 0 else d * d * 2.0 ** -rng.uniform(27, 60)
        c, p, a = [0.0, 0.0, 0.0], [0.0, 0.0, 0.0], i % 3
        c[a] = d if i % 2 else -d
        got = pair(fix, c, p, 1.25, eps2, 15.0)
        r2 = Decimal(d) ** 2 + Decimal(eps2)
        assert got is not None
        assert abs(Decimal(got[0]) * r2 * r2.sqrt() / Decimal(1.25) - 1) <= Decimal(2.0 ** -52.4), (d, eps2)
        assert abs(Decimal(got[4]) * r2.sqrt() - 1) <= Decimal(2.0 ** -52.4), (d, eps2)


@pytest.mark.parametrize("size", [1e-8, 1e-11, 1e-13, 1e-16, 1e-20, 1e-27, 1e-40, 1e-320])
@pytest.mark.parametrize("eps2", [0.0, 1e-6])
def test_small_components(fix, size, eps2):
    """A box of 30 whose z coordinates are of the given size on one or both sides: the component keeps
    its 53 bits or the pair is left to FP64 -- which pairs with one z of ordinary size never are, nor
    those of a plane (z exactly 0)."""
    rng = random.Random(3)
    left = 0
    for i in range(400):
        c, p = ([rng.uniform(-1.0, 1.0) * 15.0 for _ in range(3)] for _ in range(2))
        one_side = i % 4 == 0
        c[2] = rng.uniform(-1.0, 1.0) * size
        if not one_side:
            p[2] = rng.choice((rng.uniform(-1.0, 1.0) * size, 0.0, c[2] * (1.0 + 2.0 ** -20)))
        if i % 2:
            c, p = p, c
        got = pair(fix, c, p, 1.5, eps2, 15.0)
        if got is None:
            left += 1
            assert not one_side and size < 1e-10
            continue
        d = [Decimal(a) - Decimal(b) for a, b in zip(c, p)]
        for g, v in zip(got[1:], d):
            # 2^-52 for the truncation to 53 bits and 2 half units of 2^-55 for the coordinates
            assert abs(Decimal(g) - v) <= abs(v) * Decimal(2.0 ** -52 + 2.0 ** -55)
        r2 = sum(v * v for v in d) + Decimal(eps2)
        assert abs(Decimal(got[0]) * r2 * r2.sqrt() / Decimal(1.5) - 1) <= Decimal(2.0 ** -52.4)
    assert left == 0 if size >= 1e-8 else left > 0 if size <= 1e-13 else True
    c[2] = p[2] = 0.0
    assert pair(fix, c, p, 1.5, eps2, 15.0) is not None


def test_components_are_rounded(fix):
    """Differences that doubles hold are exact, with either sign (of the words kept, those of a negative
    one fall short by a unit); others are within half a unit in the last place where the two words have
    four bits and more beyond it (2^-53, and 2^-57 twice for those words' own truncation)."""
    rng = random.Random(17)
    for i in range(2000):
        c, p = ([float(rng.randint(-12, 12)) * 2.0 ** -rng.randint(0, 6) for _ in range(3)]
                for _ in range(2))
        got = pair(fix, c, p, 1.0, 1e-9, 15.0)
        d = [a - b for a, b in zip(c, p)]
        if got is None:
            assert max(map(abs, d)) < 2.0 ** -25
            continue
        most = max(map(abs, d))
        for g, v in zip(got[1:], d):
            if abs(v) >= most * 2.0 ** -6 or v == 0.0:
                assert g == v
    for i in range(4000):
        f = 2.0 ** -rng.uniform(0, 20)
        p = [rng.uniform(-1.0, 1.0) * 14.0 for _ in range(3)]
        c = [v + rng.uniform(0.03, 1.0) * rng.choice((-1, 1)) * f for v in p]
        got = pair(fix, c, p, 1.0, 1e-9, 15.0)
        for g, a, b in zip(got[1:], c, p):
            v = Decimal(a) - Decimal(b)
            assert abs(Decimal(g) - v) <= abs(v) * Decimal(2.0 ** -53 + 2.0 ** -56)
