"""Performance cases of the N-body library: leapfrog steps with Barnes-Hut and all-pairs forces,
ensembles, energies and the opening policy's training step, each through the calls of nbody.lib
that a simulation program makes.

``listed`` gives the fixed cases, ``draw`` more of the same ranges, ``prepare`` a program's state
(bodies on the device, context, tree or batch), ``run`` one pass, ``work`` the bytes and operations
a pass cannot do without and ``exact`` a pass's results in FP64 from plain torch.
"""

from __future__ import annotations

import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "n-body-simulation_gb300")
for _p in (_ROOT, _PKG):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from nbody import generators  # noqa: E402
from nbody import lib  # noqa: E402

DEV = "cuda"
F64 = torch.float64
NET = 1377  # parameters of the opening network: W1[8][32], b1, W2[32][32], b2, w3, b3
TRAIN_ROWS = 1 << 20


def listed():
    return [
        # a planetary system of the size of the reference's own example input: launches count
        {"name": "bh_f64_777", "kind": "bh", "dist": "disc", "n": 777, "theta": 1.05,
         "opening": "theta", "precision": "f64"},
        # an ordinary interactive run, odd size
        {"name": "bh_f64_16411", "kind": "bh", "dist": "disc", "n": 16411, "theta": 0.5,
         "opening": "theta", "precision": "f64"},
        # the headline run
        {"name": "bh_f64_1m", "kind": "bh", "dist": "disc", "n": 1048576, "theta": 0.5,
         "opening": "theta", "precision": "f64"},
        # a star cluster: deep tree, dense core, softening
        {"name": "bh_f64_plummer_131101", "kind": "bh", "dist": "plummer", "n": 131101,
         "theta": 0.7, "opening": "theta", "precision": "f64"},
        # the double-float option at a large ordinary size
        {"name": "bh_df64_262144", "kind": "bh", "dist": "disc", "n": 262144, "theta": 0.5,
         "opening": "theta", "precision": "df64"},
        # the learned opening policy on the disc + cluster mix
        {"name": "bh_learned_524309", "kind": "bh", "dist": "mix", "n": 524309, "theta": 0.3,
         "opening": "learned", "precision": "f32c"},
        # a small all-pairs run
        {"name": "naive_f64_1009", "kind": "naive", "dist": "disc", "n": 1009,
         "precision": "f64"},
        # the reference's plain algorithm at its ordinary size
        {"name": "naive_f64_16384", "kind": "naive", "dist": "disc", "n": 16384,
         "precision": "f64"},
        # single-precision pair forces of a softened star cluster
        {"name": "naive_f32c_65536", "kind": "naive", "dist": "plummer", "n": 65536,
         "precision": "f32c"},
        # many small clusters of uneven size advanced together by one captured step
        {"name": "ensemble_128", "kind": "ensemble", "systems": 128, "lo": 256, "hi": 16384},
        # the energy check of a run
        {"name": "energy_50021", "kind": "energy", "dist": "disc", "n": 50021},
        # one optimiser step of the opening network at its trainer's batch size
        {"name": "train_8192", "kind": "train", "rows": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bh", "bh", "bh", "naive", "naive", "ensemble", "energy", "train"])
    dist = rng.choice(["disc", "plummer"])
    if kind == "bh":
        opening, precision = rng.choice([
            ("theta", "f64"), ("theta", "f64"), ("theta", "f64"), ("theta", "f64_ieee"),
            ("theta", "df64"), ("theta", "f32c"), ("group", "f64"), ("group", "f32c"),
            ("learned", "f32c")])
        theta = round(rng.uniform(0.4, 1.05), 3)
        hi = {"f64_ieee": 65536, "f64": 400000}.get(precision, 600000)
        if opening == "group" and precision == "f64":
            hi = 65536
        n = _log_int(rng, 64, hi)
        if opening == "learned":
            dist, theta, n = "mix", 0.3, _log_int(rng, 4096, 1000003)
        return {"kind": "bh", "dist": dist, "n": n, "theta": theta, "opening": opening,
                "precision": precision}
    if kind == "naive":
        precision = rng.choice(["f64", "f64", "f64_ieee", "df64", "f32c"])
        hi = {"f64": 36000, "f64_ieee": 8000, "df64": 70000, "f32c": 262144}[precision]
        return {"kind": "naive", "dist": dist, "n": _log_int(rng, 64, hi),
                "precision": precision}
    if kind == "ensemble":
        lo = _log_int(rng, 64, 2048)
        return {"kind": "ensemble", "systems": _log_int(rng, 8, 256), "lo": lo,
                "hi": _log_int(rng, 2 * lo, 16384)}
    if kind == "energy":
        return {"kind": "energy", "dist": dist, "n": _log_int(rng, 64, 50000)}
    return {"kind": "train", "rows": _log_int(rng, 512, 65536)}


# -- inputs -----------------------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _u(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=F64)


def _disc(g, n):
    """A central mass, up to 8 planets on circular orbits and a belt of small bodies (AU, kg, days),
    distributed as generators.heliocentric_disc. Returns m, pos (3), vel (3), acc (3)."""
    G = generators.reference_G()
    mu = G * generators.MSUN_KG
    k = n - 1
    planets = min(8, k)
    a, e, inc = _u(g, k, 2.1, 3.3), _u(g, k, 0.0, 0.2), _u(g, k, 0.0, math.radians(10.0))
    m = torch.exp(_u(g, k, math.log(1e-15), math.log(1e-10)))
    a[:planets] = _u(g, planets, 0.4, 30.0)
    m[:planets] = torch.exp(_u(g, planets, math.log(1.6e-7), math.log(1e-3)))
    e[:planets] = 0.0
    inc[:planets] = 0.0
    node, peri, mean = (_u(g, k, 0.0, 2 * math.pi) for _ in range(3))
    E = mean.clone()
    for _ in range(12):  # Kepler's equation by Newton-Raphson
        E = E - (E - e * torch.sin(E) - mean) / (1.0 - e * torch.cos(E))
    b = torch.sqrt(1.0 - e * e)
    ox, oy = a * (torch.cos(E) - e), a * b * torch.sin(E)
    f = torch.sqrt(mu / a) / (1.0 - e * torch.cos(E))
    ovx, ovy = -f * torch.sin(E), f * b * torch.cos(E)
    cw, sw, cO, sO = torch.cos(peri), torch.sin(peri), torch.cos(node), torch.sin(node)
    ci, si = torch.cos(inc), torch.sin(inc)
    rows = ((cw * cO - sw * ci * sO, -(sw * cO + cw * ci * sO)),
            (cw * sO + sw * ci * cO, cw * ci * cO - sw * sO), (sw * si, cw * si))
    zero = torch.zeros(1, device=DEV, dtype=F64)
    pos = [torch.cat([zero, ox * p + oy * q]) for p, q in rows]
    vel = [torch.cat([zero, ovx * p + ovy * q]) for p, q in rows]
    m = torch.cat([zero + 1.0, m]) * generators.MSUN_KG
    r2 = (pos[0] * pos[0] + pos[1] * pos[1] + pos[2] * pos[2]).clamp_min(1e-4)
    acc = [-mu * p / (r2 * torch.sqrt(r2)) for p in pos]  # the central mass's pull
    acc[0][0] = 1e-7  # the central body's own small acceleration
    return m, pos, vel, acc


def _iso(g, n):
    cz, ph = _u(g, n, -1.0, 1.0), _u(g, n, 0.0, 2 * math.pi)
    s = torch.sqrt(1.0 - cz * cz)
    return torch.stack([s * torch.cos(ph), s * torch.sin(ph), cz])


def _plummer(g, n):
    """G = M = a = 1, equal masses, radii up to 10, speeds from the distribution function by
    rejection (Aarseth, Henon and Wielen 1974), as generators.plummer."""
    X = _u(g, n, 1e-9, (1.0 + 0.01) ** -1.5)
    r = 1.0 / torch.sqrt(X ** (-2.0 / 3.0) - 1.0)
    q = torch.empty(0, device=DEV, dtype=F64)
    while q.numel() < n:
        c, h = _u(g, 4 * n + 64), _u(g, 4 * n + 64, 0.0, 0.1)
        q = torch.cat([q, c[h < c * c * (1.0 - c * c) ** 3.5]])
    pos = _iso(g, n) * r
    vel = _iso(g, n) * (q[:n] * math.sqrt(2.0) * (1.0 + r * r) ** -0.25)
    pos -= pos.mean(dim=1, keepdim=True)
    vel -= vel.mean(dim=1, keepdim=True)
    m = torch.full((n,), 1.0 / n, device=DEV, dtype=F64)
    w = (1.0 + (pos * pos).sum(dim=0)) ** -1.5  # the smooth sphere's pull
    return m, [p.clone() for p in pos], [v.clone() for v in vel], [-(p * w) for p in pos]


def _mix(g, n):
    """Half disc, half a cluster of 1e-3 solar masses and scale radius 0.05 AU on a circular orbit
    at 5 AU, as generators.disc_plummer_mix."""
    nd = n // 2
    G = generators.reference_G()
    md, pd, vd, ad = _disc(g, nd)
    mp, pp, vp, ap = _plummer(g, n - nd)
    a, M, R = 0.05, 1e-3 * generators.MSUN_KG, 5.0
    mu = G * generators.MSUN_KG
    vs, vc = math.sqrt(G * M / a), math.sqrt(mu / R)
    pos = [torch.cat([p, q * a + (R if k == 0 else 0.0)]) for k, (p, q) in enumerate(zip(pd, pp))]
    vel = [torch.cat([p, q * vs + (vc if k == 1 else 0.0)]) for k, (p, q) in enumerate(zip(vd, vp))]
    acc = [torch.cat([p, q * (G * M / (a * a)) - (mu / (R * R) if k == 0 else 0.0)])
           for k, (p, q) in enumerate(zip(ad, ap))]
    return torch.cat([md, mp * M]), pos, vel, acc


def _bodies(case, seed):
    """(m, pos, vel, acc, G, eps2, dt) of a single system."""
    g = _gen(seed)
    if case["dist"] == "plummer":
        return (*_plummer(g, case["n"]), 1.0, 1e-6, 1e-3)
    make = _mix if case["dist"] == "mix" else _disc
    return (*make(g, case["n"]), generators.reference_G(), 1e-22, 1.0 / 24)


def _ensemble_counts(case):
    """Log-uniform counts, the same for every seed: evenly spread in a scrambled order."""
    k, lo, hi = case["systems"], math.log(case["lo"]), math.log(case["hi"])
    return [int(math.exp(lo + (hi - lo) * (((i * 0.6180339887498949) % 1.0)))) for i in range(k)]


def _ensemble(case, seed):
    g = _gen(seed)
    counts = _ensemble_counts(case)
    parts = [_plummer(g, c) for c in counts]
    m = torch.cat([p[0] for p in parts])
    pos, vel, acc = ([torch.cat([p[i][k] for p in parts]) for k in range(3)] for i in (1, 2, 3))
    return counts, m, pos, vel, acc


def _policy(g):
    """An opening network as training leaves one: the logarithm of a monopole's relative error as
    a linear trend of the features (force over weakest acceleration, distance over cell size,
    spread) through the two ReLU layers, with small random weights beside it."""
    W1 = 0.01 * torch.randn(8, 32, generator=g, device=DEV)
    W2 = 0.01 * torch.randn(32, 32, generator=g, device=DEV)
    b1, b2 = (0.01 * torch.randn(32, generator=g, device=DEV) for _ in range(2))
    w3 = 0.01 * torch.randn(32, generator=g, device=DEV)
    trend = torch.tensor([0.0, 0.43, 0.0, 0.0, 0.0, 0.8, -0.48, 0.0], device=DEV)
    W1[:, 0], W1[:, 1] = trend, -trend
    W2[:, 0], W2[:, 1] = 0.0, 0.0
    W2[0, 0] = W2[1, 1] = 1.0
    w3[0], w3[1] = 1.0, -1.0
    b3 = torch.full((1,), -0.42, device=DEV)
    return torch.cat([W1.ravel(), b1, W2.ravel(), b2, w3, b3]).contiguous()


def _train_inputs(case, seed):
    g = _gen(seed)
    scale = torch.tensor([0.5, 0.2, 0.3, 0.2, 0.3, 0.4, 0.5, 0.2], device=DEV)
    X = scale * torch.randn(TRAIN_ROWS, 8, generator=g, device=DEV) + 0.5 * scale
    trend = torch.tensor([0.0, 0.25, 0.0, 0.0, 0.0, 0.8, -0.48, 0.0], device=DEV)
    Y = X @ trend - 0.6 + 0.05 * torch.randn(TRAIN_ROWS, generator=g, device=DEV)
    idx = torch.randint(TRAIN_ROWS, (case["rows"],), generator=g, device=DEV).to(torch.int32)
    p = 0.25 * torch.randn(NET, generator=g, device=DEV)
    m = 1e-3 * torch.randn(NET, generator=g, device=DEV)
    v = 1e-5 * (0.1 + torch.rand(NET, generator=g, device=DEV))
    return X.contiguous(), Y.contiguous(), idx, p, m, v


# -- the cases --------------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case, "ctx": lib.Context(0)}
    if kind == "train":
        s["X"], s["Y"], s["idx"], s["p"], s["m"], s["v"] = _train_inputs(case, seed)
        s["grad"] = torch.zeros(NET, device=DEV)
        s["loss"] = torch.zeros(1, device=DEV)
        s["step"] = 99
        return s
    if kind == "ensemble":
        counts, s["m"], s["pos"], s["vel"], s["acc"] = _ensemble(case, seed)
        s["vh"] = [torch.zeros_like(v) for v in s["vel"]]
        s["batch"] = lib.Batch(s["ctx"], counts)
        s["batch"].set_config(lib.PAIR_CONFIGS + 2)  # kept from a tuning run of such ensembles
        s["graph"] = s["batch"].graph(s["m"], s["pos"], s["vel"], s["vh"], s["acc"], 1.0, 1e-6,
                                      1e-3, 1)
        return s
    s["m"], s["pos"], s["vel"], s["acc"], s["G"], s["eps2"], s["dt"] = _bodies(case, seed)
    if kind == "energy":
        s["out"] = torch.zeros(4, dtype=F64, device=DEV)
        return s
    s["vh"] = [torch.zeros_like(v) for v in s["vel"]]
    if kind == "bh":
        s["tree"] = lib.BHTree(s["ctx"], case["n"], theta=case["theta"])
        s["tree"].set_records(lib.build_mask_for(case["opening"], case["precision"]))
        if case["opening"] == "learned":
            s["tree"].set_policy(_policy(_gen(seed + 77)), -4.25, case["theta"], 2 ** 31 - 1)
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "train":
        s["step"] += 1
        lib.mlp_loss_grad(ctx, s["p"], s["X"], s["Y"], s["idx"], s["idx"].numel(), s["grad"],
                          s["loss"])
        lib.mlp_adam(ctx, s["p"], s["m"], s["v"], s["grad"], 2e-3, 0.9, 0.999, 1e-8, s["step"])
        return {"loss": s["loss"], "grad": s["grad"], "p": s["p"], "m": s["m"], "v": s["v"]}
    if kind == "energy":
        ctx.energy(s["m"], *s["pos"], *s["vel"], s["G"], s["out"])
        return s["out"]
    if kind == "ensemble":
        s["graph"].launch()
        return {"pos": s["pos"], "vel": s["vel"], "acc": s["acc"]}
    ctx.kick_drift(s["vh"], s["vel"], s["pos"], s["acc"], s["dt"])
    if kind == "bh":
        c = s["case"]
        s["tree"].build(s["m"], *s["pos"], s["G"])
        s["tree"].accel(*s["pos"], *s["acc"], s["G"], s["eps2"], c["opening"], c["precision"])
    else:
        ctx.naive_accel(s["m"], *s["pos"], *s["acc"], s["G"], s["eps2"], s["case"]["precision"])
    ctx.kick(s["vel"], s["vh"], s["acc"], s["dt"])
    return {"pos": s["pos"], "vel": s["vel"], "acc": s["acc"]}


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows = case["rows"]  # forward 2 x 1,312 multiply-adds, backward twice that
        return {"bytes": rows * 40.0 + NET * 4 * 7, "flops": rows * 6.0 * (8 * 32 + 32 * 32 + 32)}
    if kind == "energy":
        n = case["n"]
        return {"bytes": n * 56.0, "flops": n * (n - 1) / 2 * 12.0}
    if kind == "ensemble":
        # mean of a log-uniform count's first and second moments
        lo, hi = case["lo"], case["hi"]
        w = math.log(hi / lo)
        n1, n2 = (hi - lo) / w, (hi * hi - lo * lo) / (2 * w)
        return {"bytes": case["systems"] * n1 * 152.0, "flops": case["systems"] * n2 * 20.0}
    n = case["n"]
    if kind == "naive":
        return {"bytes": n * 152.0, "flops": n * float(n) * 20.0}
    # monopoles a body accepts: about 28 log2(n) / theta^2 * 0.45 on these systems, 20 flop each
    cells = min(float(n), 28.0 * 0.45 * math.log2(n) / case["theta"] ** 2)
    return {"bytes": n * 152.0, "flops": n * cells * 20.0}


# -- results in 64 bits -----------------------------------------------------------------------


def _direct(m, pos, G, eps2):
    """All-pairs accelerations, chunked over targets."""
    n = m.numel()
    out = [torch.empty_like(m) for _ in range(3)]
    rows = max(1, (1 << 26) // n)
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d = [p[None, :] - p[a:b, None] for p in pos]
        den = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps2
        w = m[None, :] / (den * torch.sqrt(den))
        w[torch.arange(b - a, device=DEV), torch.arange(a, b, device=DEV)] = 0.0
        for k in range(3):
            out[k][a:b] = (w * d[k]).sum(dim=1) * G
    return out


def _octree(m, pos):
    """The octree of the Barnes-Hut rule: per node the mass, centre of mass, edge, the body of a
    leaf (else -1) and the children (-1 where empty). Box: the bodies' and the origin's bounds as a
    cube; octants by strict midpoint comparisons (ties: lower x, lower y, upper z)."""
    lo = [min(0.0, float(p.min())) for p in pos]
    hi = [max(0.0, float(p.max())) for p in pos]
    edge = max(h - l for l, h in zip(lo, hi))
    lo = [l - (edge - (h - l)) / 2 for l, h in zip(lo, hi)]
    n = m.numel()
    ids = torch.arange(n, device=DEV)
    corner = [torch.full_like(m, l) for l in lo]
    cell = torch.zeros(n, dtype=torch.int64, device=DEV)
    nodes = {"mass": [m.sum()[None]], "edge": [torch.full((1,), edge, device=DEV, dtype=F64)],
             "body": [torch.full((1,), 0 if n == 1 else -1, dtype=torch.int64, device=DEV)],
             "parent": [torch.full((1,), -1, dtype=torch.int64, device=DEV)],
             "oct": [torch.zeros(1, dtype=torch.int64, device=DEV)]}
    for k in range(3):
        nodes["c%d" % k] = [(m * pos[k]).sum()[None] / m.sum()]
    total = 1
    while n > 1 and ids.numel() > 0 and len(nodes["mass"]) < 60:
        octant = torch.zeros_like(cell)
        for k in range(3):
            mid = corner[k] + edge / 2
            p = pos[k][ids]
            up = p >= mid if k == 2 else p > mid
            octant |= up.to(torch.int64) << k
            corner[k] = torch.where(up, mid, corner[k])
        edge = edge / 2
        key, inv, cnt = torch.unique(cell * 8 + octant, return_inverse=True, return_counts=True)
        mass = torch.zeros(key.numel(), device=DEV, dtype=F64).index_add_(0, inv, m[ids])
        nodes["mass"].append(mass)
        for k in range(3):
            s = torch.zeros_like(mass).index_add_(0, inv, m[ids] * pos[k][ids])
            nodes["c%d" % k].append(s / mass)
        nodes["edge"].append(torch.full_like(mass, edge))
        first = torch.zeros_like(key).scatter_reduce_(0, inv, ids, "amax", include_self=False)
        nodes["body"].append(torch.where(cnt == 1, first, -1))
        nodes["parent"].append(torch.div(key, 8, rounding_mode="floor"))
        nodes["oct"].append(key % 8)
        keep = cnt[inv] > 1
        cell, ids = (inv + total)[keep], ids[keep]
        corner = [c[keep] for c in corner]
        total += key.numel()
    t = {k: torch.cat(v) for k, v in nodes.items()}
    t["child"] = torch.full((total, 8), -1, dtype=torch.int64, device=DEV)
    at = torch.arange(1, total, device=DEV)
    t["child"][t["parent"][1:], t["oct"][1:]] = at
    return t


def _barnes_hut(m, pos, G, eps2, theta):
    """Accelerations under the per-body rule edge / distance < theta, breadth first."""
    t = _octree(m, pos)
    n = m.numel()
    out = [torch.zeros_like(m) for _ in range(3)]
    for a in range(0, n, 16384):
        b = torch.arange(a, min(n, a + 16384), device=DEV)
        node = torch.zeros_like(b)
        while b.numel() > 0:
            d = [t["c%d" % k][node] - pos[k][b] for k in range(3)]
            d2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            body = t["body"][node]
            take = ((body >= 0) & (body != b)) | ((body < 0) & (t["edge"][node] / torch.sqrt(d2) < theta))
            den = (d2 + eps2)[take]
            w = t["mass"][node[take]] / (den * torch.sqrt(den)) * G
            for k in range(3):
                out[k].index_add_(0, b[take], w * d[k][take])
            go = (body < 0) & ~take
            kids = t["child"][node[go]]
            b = b[go][:, None].expand(-1, 8)
            ok = kids >= 0
            b, node = b[ok], kids[ok]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        X, Y, idx, p, m, v = (t.double() if t.is_floating_point() else t.long()
                              for t in _train_inputs(case, seed))
        X, Y = X[idx], Y[idx]
        q = p.clone().requires_grad_(True)
        W1, b1, W2, b2, w3, b3 = torch.split(q, [256, 32, 1024, 32, 32, 1])
        h = torch.relu(X @ W1.view(8, 32) + b1)
        h = torch.relu(h @ W2.view(32, 32) + b2)
        loss = ((h @ w3 + b3 - Y) ** 2).mean()
        g, = torch.autograd.grad(loss, q)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        mh, vh = m / (1 - 0.9 ** 100), v / (1 - 0.999 ** 100)
        return {"loss": loss.detach()[None], "grad": g,
                "p": p - 2e-3 * mh / (torch.sqrt(vh) + 1e-8), "m": m, "v": v}
    if kind == "ensemble":
        counts, m, pos, vel, acc = _ensemble(case, seed)
        G, eps2, dt = 1.0, 1e-6, 1e-3
    else:
        m, pos, vel, acc, G, eps2, dt = _bodies(case, seed)
    if kind == "energy":
        n = case["n"]
        ek = (0.5 * m * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2)).sum()
        ep = torch.zeros((), device=DEV, dtype=F64)
        rows = max(1, (1 << 26) // n)
        for a in range(0, n, rows):
            b = min(n, a + rows)
            d = [p[None, :b] - p[a:b, None] for p in pos]
            r = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
            w = torch.tril((m[None, :b] * m[a:b, None] / r), diagonal=a - 1)
            ep -= torch.where(torch.isfinite(w), w, 0.0).sum() * G
        return torch.stack([ek, ep, ek + ep, 2.0 * ek / ep.abs()])
    vh = [v + a * (dt / 2) for v, a in zip(vel, acc)]
    pos = [p + v * dt for p, v in zip(pos, vh)]
    if kind == "bh" and case["opening"] != "theta":
        return {"pos": pos, "vel": [None] * 3, "acc": [None] * 3}
    if kind == "bh":
        acc = _barnes_hut(m, pos, G, eps2, case["theta"])
    elif kind == "naive":
        acc = _direct(m, pos, G, eps2)
    else:
        parts, at = [], 0
        for c in counts:
            parts.append(_direct(m[at:at + c], [p[at:at + c] for p in pos], G, eps2))
            at += c
        acc = [torch.cat([p[k] for p in parts]) for k in range(3)]
    return {"pos": pos, "vel": [v + a * (dt / 2) for v, a in zip(vh, acc)], "acc": acc}
