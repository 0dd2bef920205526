"""Calls captured into graphs: the scratch that a graph's kernels use stays theirs, whatever the context
does afterwards, and the results' bits do not depend on what ran before the capture."""

import numpy as np
import pytest

from helpers import bodies, dev, host

pytestmark = pytest.mark.gpu


def arrays(n):
    import torch
    d = bodies("plummer", n, seed=n)
    return [dev(d[k]) for k in ("m", "x", "y", "z")], [
        torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]


def call(c, t, a, what, targets):
    n = t[0].numel()
    if what == "targets":
        c.naive_accel_targets(*t, targets, *a, 1.0, 1e-6)
    elif what == "range":
        c.naive_accel_range(*t, *a, 5, n - 3, 1.0, 1e-6, "f64")
    else:
        c.naive_accel(*t, *a, 1.0, 1e-6, what)


@pytest.mark.parametrize("what", ["targets", "range", "f64", "df64", "f32c"])
@pytest.mark.parametrize("warm", [False, True])
def test_replay_after_the_scratch_has_grown(what, warm):
    """Captured with enough scratch (or, NB_F64, with none), then a larger call, new allocations, and the
    replay: the bits of the ordinary call."""
    import torch
    from nbody.lib import Context
    if not warm and what in ("df64", "f32c"):
        pytest.skip("their first call allocates, which a capture cannot")
    n = 3000
    t, a = arrays(n)
    tg = torch.arange(n, dtype=torch.int32, device="cuda")
    other = Context(0)
    call(other, t, a, what, tg)
    other.sync()
    want = [host(v).copy() for v in a]
    c = Context(0)
    if warm:
        call(c, t, a, what, tg)
        c.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        call(c, t, a, what, tg)
    big, big_a = arrays(9000)
    call(c, big, big_a, what, torch.arange(9000, dtype=torch.int32, device="cuda"))
    c.sync()
    fresh = [torch.full((1 << k,), 7.0, dtype=torch.float64, device="cuda") for k in range(12, 22)]
    for _ in range(2):
        for v in a:
            v.fill_(np.nan)
        g.replay()
        torch.cuda.synchronize()
        lo, hi = (5, n - 3) if what == "range" else (0, n)
        for v, w in zip(a, want):
            np.testing.assert_array_equal(host(v)[lo:hi], w[lo:hi])
    assert all((f == 7.0).all() for f in fresh)
    del g
    c.close()
    other.close()
