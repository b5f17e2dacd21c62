"""Measured cases: FMM solves as a program calls them, over the range of sizes,
precisions and options of this library's workloads.

A case is one pass of one use:

* ``solve``      a solver kept between solves, new points and strengths on the
                 device each time (tree, passes, evaluation, fields on the device);
* ``strengths``  a fixed tree with new strengths each time, as an iterative
                 solver applies it (one graph launch per application);
* ``bases``      a fixed tree and precomputed target bases, new strengths;
* ``oneshot``    ``engine.solve`` on host arrays: create, solve, copy out;
* ``served``     a batch of the mixed request stream through ``engine.Server``.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from wbfmm_b200 import engine
from wbfmm_b200 import workloads as W

LAP, HELM = engine.LAPLACE, engine.HELMHOLTZ
DEV = "cuda"
CUTOFF2 = 1e-12       # pairs closer than 1e-6 are one point (self term)


def _case(name, use, problem, n, depth, **kw):
    c = dict(name=name, use=use, problem=problem, n=n, depth=depth, nt=0, order=14, k=0.0,
             fp32=False, points="cube", dipoles=False, grad=True, skip_empty=False,
             sparse=False, requests=0)
    c.update(kw)
    return c


def listed():
    return [
        # the serving stream's smallest request as a plain FP64 solve: latency
        _case("laplace_1e3_fp64", "solve", LAP, 1000, 2),
        # an iterative solver's matrix product on a small fixed tree
        _case("laplace_1e4_strengths_fp32", "strengths", LAP, 10000, 2, fp32=True),
        # the simplest call there is: one solve of host arrays
        _case("helmholtz_2e4_oneshot_fp64", "oneshot", HELM, 20011, 3, order=8, k=8.0),
        # the reference's own test size: separate sources and targets, order 12
        _case("laplace_2e4_targets_fp64", "solve", LAP, 20000, 4, nt=20000, order=12),
        # boundary-element matrix product at fixed targets, potential only
        _case("helmholtz_1e5_bases_fp64", "bases", HELM, 100003, 4, order=8, k=10.0, grad=False),
        # ordinary single-precision solves of the serving orders, volume and surface points
        _case("helmholtz_1e5_fp32", "solve", HELM, 100000, 4, k=10.0, fp32=True, skip_empty=True),
        _case("laplace_3e5_fp32", "solve", LAP, 300000, 4, fp32=True, skip_empty=True),
        # the large cube of the library's benchmark: single precision at a quarter
        # of its points and a level less, and the plain FP64 form whole
        _case("helmholtz_cube_2e5_fp32", "solve", HELM, 249989, 5, order=6, k=8.0, fp32=True),
        _case("helmholtz_cube_1e6_fp64", "solve", HELM, 1000000, 6, order=6, k=8.0),
        # surface scattering: monopoles and dipoles on a sphere, targets on another
        _case("helmholtz_sphere_fp64", "solve", HELM, 500000, 6, nt=125000, order=6, k=40.0,
              points="sphere", dipoles=True, skip_empty=True),
        # clustered particles with sparse level storage
        _case("laplace_clusters_2e6_fp64", "solve", LAP, 2000000, 7, order=10, points="clusters",
              sparse=True),
        # a batch of the mixed serving stream, device-resident requests
        _case("served_16_fp32", "served", LAP, 300000, 0, fp32=True, skip_empty=True, requests=16),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges; no more work than the largest listed one."""
    use = rng.choice(["solve"] * 7 + ["strengths", "strengths", "bases", "oneshot", "served"])
    problem = rng.choice([LAP, HELM])
    fp32 = rng.random() < 0.5
    if use == "served":
        c = _case("", use, LAP, _logu(rng, 3e4, 3e5), 0, fp32=True, skip_empty=True,
                  requests=rng.randint(4, 16))
    else:
        top = {"solve": 3e5 if fp32 else 8e5, "strengths": 2e5, "bases": 1.5e5, "oneshot": 5e4}[use]
        n = _logu(rng, 1e3, top)
        occ = _logu(rng, 8, 100)              # mean points of a leaf box
        depth = min(5 if problem == HELM else 6, max(2, round(math.log(n / occ, 8))))
        order = rng.randint(6, 16)
        points = rng.choice(["cube", "cube", "sphere", "clusters"])
        if points == "clusters":
            depth += 1
            n = min(n, 200000)
        if depth >= 5:
            order = min(order, 10)
        k = rng.uniform(4.0, 30.0) if problem == HELM else 0.0
        if fp32 and problem == HELM:
            k = max(k, 0.9 * 2 ** depth)      # the FP32 form's wavenumber range
        c = _case("", use, problem, n, depth, order=order, k=round(k, 4), fp32=fp32, points=points,
                  nt=_logu(rng, 1e3, n) if n > 1000 and rng.random() < 0.3 else 0,
                  dipoles=use in ("solve", "oneshot") and n <= 200000 and rng.random() < 0.3,
                  grad=use != "bases" and rng.random() < 0.75,
                  skip_empty=use != "bases" and rng.random() < 0.5,
                  sparse=use == "solve" and rng.random() < 0.2)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
X0, D = (-0.51, -0.51, -0.51), 1.02      # the tree cube of points in [-0.5, 0.5]^3


def _points(gen, kind, n, r=0.45):
    if kind == "sphere":
        v = torch.randn(n, 3, dtype=torch.float64, device=gen.device, generator=gen)
        return r * v / v.norm(dim=1, keepdim=True)
    if kind == "clusters":
        c = torch.rand(8, 3, dtype=torch.float64, device=gen.device, generator=gen) * 0.8 - 0.4
        which = torch.randint(0, 8, (n,), device=gen.device, generator=gen)
        g = torch.randn(n, 3, dtype=torch.float64, device=gen.device, generator=gen)
        return (c[which] + 0.05 * g).clamp_(-0.5, 0.5)
    return torch.rand(n, 3, dtype=torch.float64, device=gen.device, generator=gen) - 0.5


def _orders(case):
    if case["problem"] == LAP:
        return [0] + [case["order"]] * case["depth"]
    return [0] + [W.helmholtz_order(case["k"], D / 2 ** lv, lo=case["order"], hi=60)
                  for lv in range(1, case["depth"] + 1)]


def _inputs(case, seed):
    """Points, strengths, normals and targets of a single solve, on the device."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    n, helm = case["n"], case["problem"] == HELM
    xs = _points(gen, case["points"], n).contiguous()
    q = torch.randn(n * (2 if helm else 1), dtype=torch.float64, device=DEV, generator=gen)
    nrm = dip = None
    if case["dipoles"]:
        # the first half of the sources monopoles, the second half dipoles
        nrm = xs / xs.norm(dim=1, keepdim=True).clamp_min(1e-12)
        dip = torch.randn(q.numel(), dtype=torch.float64, device=DEV, generator=gen)
        half = (n // 2) * (2 if helm else 1)
        q[half:] = 0.0
        dip[:half] = 0.0
    xt = _points(gen, case["points"], case["nt"], 0.49).contiguous() if case["nt"] else xs
    return xs, q, nrm, dip, xt


def _config(case):
    field = engine.POTENTIAL | (engine.GRADIENT if case["grad"] else 0)
    orders = _orders(case)
    return engine.SolverConfig(case["problem"], case["depth"], orders, list(orders), case["k"], X0, D,
                               engine.FP32 if case["fp32"] else engine.FP64, field,
                               skip_empty=case["skip_empty"], leaf_order=case["fp32"],
                               sparse=case["sparse"])


def _requests(case, seed):
    """A batch of the serving stream: sizes evenly spread over log [1e3, n],
    half Laplace and half Helmholtz, cube and sphere."""
    rng = np.random.default_rng(seed)
    m, lo, hi = case["requests"], math.log(1e3), math.log(case["n"])
    for i in range(m):
        n = int(round(math.exp(lo + (hi - lo) * (i + 0.5) / m)))
        yield W.serve_request(rng, n, i % 2 == 0, float(rng.uniform(1.0, 30.0)), (i // 2) % 2 == 0)


def prepare(case, seed):
    use = case["use"]
    if use == "served":
        reqs = []
        for p in _requests(case, seed):
            w = 2 if p.problem == HELM else 1
            d = {"xs": torch.from_numpy(p.xs).to(DEV), "q": torch.from_numpy(p.q).to(DEV),
                 "pot": torch.empty(w * p.nt, dtype=torch.float64, device=DEV),
                 "grad": torch.empty(3 * w * p.nt, dtype=torch.float64, device=DEV)}
            ok = engine.fp32_range_ok(engine.SolverConfig.from_problem(p))
            reqs.append((p, d, engine.FP32 if ok else engine.FP64))
        return {"use": use, "server": engine.Server(slots=6, largest_first=True), "reqs": reqs}
    xs, q, nrm, dip, xt = _inputs(case, seed)
    if use == "oneshot":
        def host(a):
            return None if a is None else a.cpu().numpy()
        o = _orders(case)
        p = W.Problem("oneshot", case["problem"], case["depth"], o, list(o), case["k"], host(xs),
                      host(q), host(xt), host(nrm), host(dip), np.array(X0), D,
                      targets_are_sources=xt is xs)
        if xt is xs:
            p.xt = p.xs
        field = engine.POTENTIAL | (engine.GRADIENT if case["grad"] else 0)
        return {"use": use, "p": p, "precision": engine.FP32 if case["fp32"] else engine.FP64,
                "field": field, "skip_empty": case["skip_empty"]}
    w = 2 if case["problem"] == HELM else 1
    nt = xt.shape[0]
    st = {"use": use, "solver": engine.Solver(_config(case)), "xs": xs, "q": q, "nrm": nrm,
          "dip": dip, "xt": xt, "depth": case["depth"],
          "pot": torch.empty(w * nt, dtype=torch.float64, device=DEV),
          "grad": torch.empty(3 * w * nt, dtype=torch.float64, device=DEV) if case["grad"] else None}
    if use != "solve":                       # the fixed tree
        torch.cuda.synchronize()
        s = st["solver"]
        s.set_sources(xs, nrm, on_device=True)
        s.set_targets(xt, on_device=True)
        s.build_operators()
        if use == "bases":
            s.target_bases()
        s.synchronize()
    return st


def run(st):
    use = st["use"]
    if use == "served":
        srv = st["server"]
        tickets = [srv.submit(p, prec, skip_empty=True, leaf_order=True, device=d,
                              near_fp32=prec == engine.FP64) for p, d, prec in st["reqs"]]
        out = [srv.wait(t) for t in tickets]
        for t in tickets:
            srv.forget(t)
        return out
    if use == "oneshot":
        return engine.solve(st["p"], st["precision"], st["field"], st["skip_empty"])
    s = st["solver"]
    if use == "solve":
        s.set_sources(st["xs"], st["nrm"], on_device=True)
        s.set_strengths(st["q"], st["dip"], on_device=True)
        s.set_targets(st["xt"], on_device=True)
        s.run()
    elif use == "strengths":
        s.set_strengths(st["q"], on_device=True)
        s.run_graph()
    else:
        s.set_strengths(st["q"], on_device=True)
        s.leaf_expansions()
        for lv in range(st["depth"], 2, -1):
            s.upward_pass(lv)
        for lv in range(2, st["depth"] + 1):
            s.downward_pass(lv)
        s.evaluate_bases()
    pot, grad = st["pot"], st["grad"]
    s.field_to_device(pot.data_ptr(), None if grad is None else grad.data_ptr())
    return (pot,) if grad is None else (pot, grad)


# -------------------------------------------------------------------- work
def _box_sum(g):
    """Sum over the 3x3x3 neighbourhood of every cell of a cubic grid."""
    for _ in range(3):
        g = F.pad(g, (0, 0, 0, 0, 1, 1))
        g = (g[:-2] + g[1:-1] + g[2:]).permute(1, 2, 0)
    return g


def _grid(x, x0, width, depth):
    nb = 1 << depth
    o = torch.as_tensor(np.asarray(x0, dtype=np.float64), device=x.device)
    i = ((x - o) / width * nb).floor().long().clamp_(0, nb - 1)
    return torch.bincount((i[:, 0] * nb + i[:, 1]) * nb + i[:, 2],
                          minlength=nb ** 3).double().reshape(nb, nb, nb)


def _coarsen(g):
    n = g.shape[0] // 2
    return g.reshape(n, 2, n, 2, n, 2).sum((1, 3, 5))


def _solve_work(problem, depth, orders, xs, xt, x0, width, grad, dipoles):
    """Bytes (inputs read, fields written) and operations of one solve: leaf
    expansions, shifts of the occupied boxes, the interaction-list pairs of
    occupied boxes by rotation and coaxial translation in the symmetric halves
    of the rotation matrices, leaf evaluation and the near-field pairs."""
    helm = problem == HELM
    w = 2 if helm else 1
    ns, nt = xs.shape[0], xt.shape[0]
    gs, gt = _grid(xs, x0, width, depth), _grid(xt, x0, width, depth)
    pairs = float((gt * _box_sum(gs)).sum()) - (nt if xt is xs else 0)
    p = orders[depth]
    nc = (p + 1) ** 2
    fl = pairs * ((44 if grad else 28) if helm else (20 if grad else 12)) * (1.5 if dipoles else 1.0)
    fl += ns * nc * (8 if helm else 4) + nt * nc * ((24 if helm else 12) if grad else (8 if helm else 4))
    for lv in range(depth, 1, -1):
        s, t = (gs > 0).double(), (gt > 0).double()
        p = orders[lv]
        x = (p + 1) ** 2 + 2 * sum((p + 1 - m) ** 2 for m in range(1, p + 1))
        par = _box_sum(_coarsen(s))
        par = par.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
        fl += float((t * (par - _box_sum(s))).sum()) * (16 if helm else 6) * x
        if lv > 2:
            fl += float(s.sum() + t.sum()) * (12 if helm else 6) * x
        gs, gt = _coarsen(gs), _coarsen(gt)
    by = 8.0 * (ns * (3 + w) + (0 if xt is xs else 3 * nt) + nt * w * (4 if grad else 1))
    if dipoles:
        by += 8.0 * ns * (3 + w)
    return by, fl


def work(case):
    if case["use"] == "served":
        by = fl = 0.0
        for p in _requests(case, 0):
            xs = torch.from_numpy(p.xs).to(DEV)
            b, f = _solve_work(p.problem, p.depth, p.order_s, xs, xs, p.x0, p.D, True, False)
            by += b
            fl += f
        return {"bytes": by, "flops": fl}
    xs, _, _, _, xt = _inputs(case, 0)
    by, fl = _solve_work(case["problem"], case["depth"], _orders(case), xs, xt, X0, D,
                         case["grad"], case["dipoles"])
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------- exact
def _direct(problem, k, xs, q, nrm, dip, xt, grad):
    """Direct sum over all pairs in 64 bits."""
    helm = problem == HELM
    nt = xt.shape[0]
    w = 2 if helm else 1
    qm = q.reshape(-1, w)
    dm = None if dip is None else dip.reshape(-1, w)
    pot = torch.empty(nt, w, dtype=torch.float64, device=xt.device)
    g = torch.empty(nt, 3, w, dtype=torch.float64, device=xt.device) if grad else None
    s = [xs[:, a].contiguous() for a in range(3)]
    nv = None if nrm is None else [nrm[:, a].contiguous() for a in range(3)]

    def cmul(re, im, v):           # sum over sources of (re + i im) v, v complex
        a, b = re @ v, im @ v
        return torch.stack((a[:, 0] - b[:, 1], a[:, 1] + b[:, 0]), 1)

    step = max(1, 12_000_000 // xs.shape[0])
    for i in range(0, nt, step):
        d = [xt[i:i + step, a, None] - s[a] for a in range(3)]
        r2 = d[0] * d[0]
        r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        near = r2 <= CUTOFF2
        ir = r2.rsqrt().masked_fill_(near, 0.0)
        if nv is not None:
            nr = d[0] * nv[0]
            nr.addcmul_(d[1], nv[1]).addcmul_(d[2], nv[2])
        sl = slice(i, i + step)
        if helm:
            kr = r2.mul_(ir).mul_(k)
            ikr = ir / k
            h0r, h0i = torch.sin(kr).mul_(ikr), torch.cos(kr).mul_(ikr).neg_()
            h1r, h1i = torch.addcmul(h0i, h0r, ikr), torch.addcmul(-h0r, h0i, ikr)
            f = cmul(h0r, h0i, qm)
            if dm is not None:
                u = nr * ir
                f -= k * cmul(h1r * u, h1i * u, dm)
            pot[sl] = f
            if grad:
                ar, ai = h1r * ir, h1i * ir
                if dm is not None:
                    dpr, dpi = h0r - 2 * h1r * ikr, h0i - 2 * h1i * ikr
                    c = nr * ir * ir
                    br, bi = (dpr * k - h1r * ir) * c, (dpi * k - h1i * ir) * c
                for a in range(3):
                    v = cmul(ar * d[a], ai * d[a], qm)
                    if dm is not None:
                        v += cmul(br * d[a] + ar * nv[a], bi * d[a] + ai * nv[a], dm)
                    g[sl, a] = -k * v
        else:
            ir3 = ir * ir * ir
            f = ir @ qm
            if dm is not None:
                f += (nr * ir3) @ dm
            pot[sl] = f
            if grad:
                for a in range(3):
                    v = -((ir3 * d[a]) @ qm)
                    if dm is not None:
                        v += (ir3 * nv[a] - 3 * nr * d[a] * ir3 * ir * ir) @ dm
                    g[sl, a] = v
    c = 0.25 / math.pi
    pot = pot.mul_(c).reshape(-1)
    return (pot,) if g is None else (pot, g.mul_(c).reshape(-1))


def exact(case, seed):
    if case["use"] == "served":
        out = []
        for p in _requests(case, seed):
            xs, q = torch.from_numpy(p.xs).to(DEV), torch.from_numpy(p.q).to(DEV)
            out.append(_direct(p.problem, p.k, xs, q, None, None, xs, True))
        return out
    if case["n"] * (case["nt"] or case["n"]) * (2 if case["dipoles"] else 1) > 1.2e11:
        return None                          # the pairs would take too long
    xs, q, nrm, dip, xt = _inputs(case, seed)
    return _direct(case["problem"], case["k"], xs, q, nrm, dip, xt, case["grad"])
