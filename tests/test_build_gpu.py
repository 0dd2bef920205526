"""Octree build at the edges of its kernels -- the one-block build (up to 2,048 bodies, three sizes of
it), the centre-of-mass chunks (one of up to 512 or 1,024 positions, or 256 and tiers of 96 chunks) --
and of its division-free quotients: every cell equal to the oracle's, bit for bit, and the accelerations of the
IEEE traversal (which read the quotients) too."""

import numpy as np
import pytest

import oracle
from helpers import bodies, canonical_compare, dev, host
from test_bh_gpu import _clustered, _midpoints

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from nbody.lib import Context
    c = Context(0)
    yield c
    c.close()


def check(ctx, d, storage=16, accelerations=True):
    import torch
    from nbody.lib import BHTree
    n = len(d["m"])
    t = {k: dev(d[k]) for k in ("m", "x", "y", "z")}
    tree = BHTree(ctx, n, theta=0.7)
    tree.build(t["m"], t["x"], t["y"], t["z"], d["G"])
    ctx.sync()
    ot = oracle.build_subtrees(d["m"], d["x"], d["y"], d["z"], max_level=7, threads=4,
                               storage_param=storage)
    assert tree.stats()["ref_node_count"] == ot.node_count
    np.testing.assert_array_equal(np.array(tree.stats()["aabb"]), ot.aabb)
    assert canonical_compare(ot, tree.export_ref_layout(n), n) == ot.node_count
    if accelerations:
        a = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
        tree.accel(t["x"], t["y"], t["z"], *a, d["G"], 1e-6, "theta", "f64_ieee")
        ctx.sync()
        ref = oracle.bh_accel(ot, d["x"], d["y"], d["z"], d["G"], 1e-6, 0.7, threads=4)
        for g, r in zip(a, ref):
            np.testing.assert_array_equal(host(g), r)
    tree.close()


@pytest.mark.parametrize("n", [1, 2, 3, 33, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2048,
                               2049, 4095, 4096, 4097, 24576, 24577])
def test_sizes(ctx, n):
    check(ctx, bodies("plummer", n, seed=n))


@pytest.mark.parametrize("n", [1000, 2400, 6000])
def test_deep_clumps_and_midpoints(ctx, n):
    check(ctx, _clustered(n, 3), storage=256)
    check(ctx, _midpoints(n, 4), storage=256)


@pytest.mark.parametrize("n", [900, 5000])
def test_quotients_of_special_values(ctx, n):
    """Coordinates and masses on powers of two, zeros, mantissas of ones, wide exponent ranges."""
    rng = np.random.default_rng(n)
    d = bodies("plummer", n, seed=2)
    d["m"] = d["m"] * 2.0 ** rng.integers(-60, 60, n)
    d["m"][1::7] = 2.0 ** rng.integers(-20, 20, len(d["m"][1::7]))
    d["m"][2::7] = np.nextafter(2.0, 0.0)
    d["m"][3::50] = 1e-300
    for k, o in (("x", 0), ("y", 1), ("z", 2)):
        v = d[k]
        v[o::11] = np.sign(v[o::11]) * 2.0 ** rng.integers(-12, 2, len(v[o::11]))
        v[o + 3::13] = 0.0
        v[o + 5::17] = np.nextafter(1.0, 0.0) * rng.uniform(0.5, 2.0, len(v[o + 5::17]))
    p = np.stack([d["x"], d["y"], d["z"]], axis=1)
    keep = np.unique(p, axis=0, return_index=True)[1]
    for k in ("m", "x", "y", "z"):
        d[k] = np.ascontiguousarray(d[k][np.sort(keep)])
    check(ctx, d, storage=64)


@pytest.mark.parametrize("n", [700, 5000])
def test_massless_bodies(ctx, n):
    d = bodies("plummer", n, seed=9)
    d["m"][::3] = 0.0
    check(ctx, d)


@pytest.mark.parametrize("n", [2000, 4500])
def test_coincident_bodies_are_reported(ctx, n):
    from nbody.lib import BHTree, NBodyError
    d = bodies("plummer", n, seed=1)
    for k in ("x", "y", "z"):
        d[k][7] = d[k][1003]
    tree = BHTree(ctx, n)
    tree.build(*[dev(d[k]) for k in ("m", "x", "y", "z")], 1.0)
    with pytest.raises(NBodyError, match="DEPTH"):
        ctx.sync()
    tree.close()


@pytest.mark.parametrize("n", [1023, 1025, 131072, 131073, 262144, 262145, 524289])
def test_sort_at_tile_edges(ctx, n):
    """The tile sizes of the sort's passes: stable, with many equal keys."""
    import torch
    from nbody.lib import util_radix_sort_pairs
    rng = np.random.default_rng(n)
    k = (rng.integers(0, 997, n).astype(np.int64) << 40) | rng.integers(0, 3, n)
    keys, vals = torch.from_numpy(k).cuda(), torch.arange(n, dtype=torch.int32, device="cuda")
    util_radix_sort_pairs(ctx, keys, vals, 0, 63)
    ctx.sync()
    order = np.argsort(k, kind="stable")
    np.testing.assert_array_equal(host(vals), order)
    np.testing.assert_array_equal(host(keys), k[order])


@pytest.mark.parametrize("n", [4096, 4097, 2048 * 4096, 2048 * 4096 + 1])
def test_scan_at_tile_edges(ctx, n):
    """Tiles that add the totals before them themselves (up to 2,048) and the launch that does it."""
    import torch
    from nbody.lib import util_exclusive_scan_u32
    v = np.random.default_rng(n).integers(0, 5, n).astype(np.int32)
    t = torch.from_numpy(v).cuda()
    out = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    util_exclusive_scan_u32(ctx, t, out)
    ctx.sync()
    np.testing.assert_array_equal(host(out), np.concatenate([[0], np.cumsum(v)]))


def _nested(clumps, levels, per_level, seed):
    """Clumps whose bodies halve their distance to the centre every `per_level` bodies."""
    rng = np.random.default_rng(seed)
    k = np.repeat(np.arange(levels), per_level)
    c = np.repeat(rng.uniform(-1, 1, (clumps, 3)), len(k), axis=0)
    r = 2.0 ** -(7.0 + np.tile(k, clumps))[:, None] * rng.uniform(0.5, 1.0, (len(c), 3))
    p = c + r * rng.choice([-1.0, 1.0], (len(c), 3))
    d = {key: np.ascontiguousarray(p[:, i]) for i, key in enumerate("xyz")}
    d["m"] = rng.uniform(0.5, 1.5, len(c))
    d["G"] = 1.0
    return d


@pytest.mark.parametrize("clumps", [20, 100, 130])
def test_many_cells_across_chunks(ctx, clumps):
    """Deep clumps: a tier with more cells than it keeps in shared memory (from about 50 clumps on),
    and one below; one and two tiers. The clumps' cores are smaller than the FP32 records resolve, so
    the walk's opening tests there have to be left to FP64."""
    check(ctx, _nested(clumps, 28, 9, clumps), storage=512)


def test_subnormal_quotients(ctx):
    """Cells whose centre's z lies halfway between two subnormal numbers: (4 * 1 + 1 * 5) / 6 of the
    smallest one and the like, with masses that keep the numerators normal."""
    tiny = 2.0 ** -1074
    rng = np.random.default_rng(6)
    rows = []
    for i, (a, b) in enumerate([(4, 1), (13, 1), (7, 10), (1, 4), (2, 5), (16, 13), (21, 0), (0, 3)]):
        x, y = -1.5 + 0.4 * i, rng.uniform(-1.0, 1.0)
        rows += [(2.0 ** 400, x, y, a * tiny), (5 * 2.0 ** 400, x + 2.0 ** -11, y, b * tiny),
                 (1.0, x + 0.1, y + 0.2, 0.0)]
    m, x, y, z = np.array(rows).T.copy()
    check(ctx, {"m": m, "x": x, "y": y, "z": z, "G": 1.0}, storage=64)
