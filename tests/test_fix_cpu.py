"""The fixed-point pair arithmetic of nb_fix.cuh, compiled as plain C++, against 60-digit decimal
arithmetic. Tolerances: the factor m (r^2 + eps^2)^(-3/2) is one rounding (2^-53) after a chain
whose truncations stay below 1.5 x 20 / 2^60 (norm, centred), 1.5 x 2^-56.6 (residual) and 2^-54
(products and dropped terms): 2^-52.4 in all; a separation component is exact up to its truncation to 53 bits (2^-52), where the fixed-point
grid (2^(K - 94) per coordinate) holds the coordinates."""

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
    axes(s, K, out[1], out[2], out[3]);
    out[4] = scaled_double(rinv1(D), 1023 - K + s.sh);
    return ok;
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
    lib.fix_pair.argtypes = [C.POINTER(C.c_double)] * 2 + [C.c_double] * 3 + [C.POINTER(C.c_double)]

    def pair(c, p, m, eps2, v_max):
        out = (C.c_double * 5)()
        ok = lib.fix_pair((C.c_double * 3)(*c), (C.c_double * 3)(*p), m, eps2, v_max, out)
        return list(out) if ok else None

    return pair


@pytest.mark.parametrize("box,eps2,lo", [(30.0, 1e-22, 20), (30.0, 0.0, 28), (1.0, 1e-6, 20),
                                         (30.0, 0.3, 20), (3e40, 1e-12, 28), (1e-40, 0.0, 28)])
def test_pairs_against_decimal(fix, box, eps2, lo):
    """Separations from the box down to 2^-lo of it, small components, coordinates on the grid."""
    getcontext().prec = 60
    rng = random.Random(5)
    used = 0
    for i in range(3000):
        f = 2.0 ** -rng.uniform(0, lo)
        p = [rng.uniform(0.25, 1.0) * rng.choice((-1, 1)) * box * 0.9 for _ in range(3)]
        c = [v + rng.uniform(-1, 1) * f * box * 0.1 * (2.0 ** -rng.uniform(0, 20) if i % 3 == a else 1.0)
             for a, v in enumerate(p)]
        if i % 7 == 0:
            c[i % 3] = p[i % 3]  # an exactly vanishing component
        m = rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-80, 100)
        got = fix(c, p, m, eps2, box)
        if got is None:
            continue
        used += 1
        d = [Decimal(a) - Decimal(b) for a, b in zip(c, p)]
        r2 = sum(v * v for v in d) + Decimal(eps2)
        w = Decimal(m) / (r2 * r2.sqrt())
        assert abs(Decimal(got[0]) / w - 1) <= Decimal(2.0 ** -52.4)
        assert abs(Decimal(got[4]) * r2.sqrt() - 1) <= Decimal(2.0 ** -52.4)
        for g, v in zip(got[1:], d):
            assert abs(Decimal(g) - v) <= abs(v) * Decimal(2.0 ** -52)
    assert used > 2000


def test_what_the_integers_leave_to_fp64(fix):
    p, c = [0.5, 0.25, -0.125], [0.75, 0.25, 0.5]
    assert fix(c, p, 1.0, 1e-6, 1.0) is not None
    assert fix(p, p, 1.0, 1e-6, 1.0) is None  # coincident
    assert fix([0.5 + 2.0 ** -33, 0.25, -0.125], p, 1.0, 1e-6, 1.0) is None  # too close
    for m in (0.0, -1.0, float("inf"), float("nan"), 5e-324):
        assert fix(c, p, m, 1e-6, 1.0) is None
    for v in (float("inf"), float("nan"), 3.0):  # not finite, or outside the scale
        assert fix([v, 0.25, 0.5], p, 1.0, 1e-6, 1.0) is None
        assert fix(c, [v, 0.25, 0.5], 1.0, 1e-6, 1.0) is None
    for e in (-1e-6, float("nan"), 1e30):
        assert fix(c, p, 1.0, e, 1.0) is None
    assert fix(c, p, 1e308, 1e-6, 1.0) is None  # the factor itself exceeds the doubles
    assert fix([v * 1e-60 for v in c], [v * 1e-60 for v in p], 1e300, 0.0, 1e-60) is None  # overflow
    assert fix([v * 1e-200 for v in c], [v * 1e-200 for v in p], 1.0, 0.0, 1e-200) is None
