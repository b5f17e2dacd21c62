"""The near field alone: sources and targets in one leaf and its neighbour, so
that no expansion reaches a target.  FP32 terms are formed two at a time and a
tree of few leaves shares a leaf's targets between CTAs; here at lone, odd and
tile-crossing source counts, and at target counts of one and of several shares."""
from __future__ import annotations

import numpy as np
import pytest

from wbfmm_b200 import engine

pytestmark = pytest.mark.gpu


def _direct(problem, k, xs, q, nrm, d, xt):
    r = xt[:, None] - xs[None]
    R = np.linalg.norm(r, axis=2)
    on = R > 1e-6
    R = np.where(on, R, 1.0)
    if problem == engine.LAPLACE:
        G, G1, G2 = 1 / R, -1 / R**2, 2 / R**3
    else:
        e = np.exp(1j * k * R) / (1j * k)
        G, G1 = e / R, e * (1j * k / R - 1 / R**2)
        G2 = e * (-k * k / R - 2j * k / R**2 + 2 / R**3)
    G, G1, G2 = (np.where(on, a, 0.0) / (4 * np.pi) for a in (G, G1, G2))
    u = r / R[..., None]
    pot, grad = G @ q, np.einsum("ts,tsc,s->tc", G1, u, q)
    if d is not None:        # n . grad over the sources (Laplace), the targets (Helmholtz)
        d = -d if problem == engine.LAPLACE else d
        nu = np.einsum("tsc,sc->ts", u, nrm)
        pot = pot + (G1 * nu) @ d
        g = (G2 * nu)[..., None] * u + (G1 / R)[..., None] * (nrm[None] - nu[..., None] * u)
        grad = grad + np.einsum("tsc,s->tc", g, d)
    return pot, grad


# FP32: a term is a dozen operations of half an ulp (6e-8) each, cubed 1/r
# tripling its own: below 2e-6 of the term, and no sum is larger than its terms
@pytest.mark.parametrize("precision,tol", [(engine.FP64, 1e-12), (engine.FP32, 5e-6)])
@pytest.mark.parametrize("problem", [engine.LAPLACE, engine.HELMHOLTZ])
@pytest.mark.parametrize("ns,nt", [(1, 1), (2, 9), (7, 40), (127, 511), (129, 520), (128, 1100),
                                   (301, 3000)])
@pytest.mark.parametrize("dipoles", [False, True])
def test_near(gpu_lib, problem, precision, tol, ns, nt, dipoles):
    rng = np.random.default_rng(ns + nt)
    k = 6.0 if problem == engine.HELMHOLTZ else 0.0
    xs, xt = rng.uniform(0.01, 0.24, (ns, 3)), rng.uniform(0.01, 0.24, (nt, 3))
    xs[:, 0] += 0.255 * (np.arange(ns) % 2)              # the leaf and its neighbour
    same = min(ns, nt) // 2
    xt[:same] = xs[:same]                                # pairs within the cutoff
    shape = (ns, 2) if problem == engine.HELMHOLTZ else (ns, 1)
    q, d = rng.uniform(0.5, 1.0, shape), rng.uniform(0.5, 1.0, shape)
    nrm = rng.standard_normal((ns, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    orders = [0, 8, 8]
    cfg = engine.SolverConfig(problem, 2, orders, list(orders), k, (-0.51,) * 3, 1.02, precision,
                              engine.POTENTIAL | engine.GRADIENT)
    with engine.Solver(cfg) as s:
        s.set_sources(xs, nrm if dipoles else None)
        s.set_strengths(q.ravel(), d.ravel() if dipoles else None)
        s.set_targets(xt)
        s.run()
        pot, grad = s.field()

    def whole(a):
        return a[..., 0] + 1j * a[..., 1] if problem == engine.HELMHOLTZ else a[..., 0]
    P, G = _direct(problem, k, xs, whole(q), nrm, whole(d) if dipoles else None, xt)
    got_p, got_g = np.asarray(pot).ravel(), np.asarray(grad).ravel()
    if problem == engine.HELMHOLTZ:
        got_p, got_g = got_p[0::2] + 1j * got_p[1::2], got_g[0::2] + 1j * got_g[1::2]
    assert np.linalg.norm(got_p - P) <= tol * np.linalg.norm(P)
    assert np.linalg.norm(got_g - G.ravel()) <= tol * np.linalg.norm(G)


# An infinite strength reaches every target of its leaf as an infinity and not
# as a NaN, whichever entry of a run it is (lone ones among them), as in the
# kernel for dipole sources (here of strength zero), whose terms are not paired
@pytest.mark.parametrize("problem", [engine.LAPLACE, engine.HELMHOLTZ])
@pytest.mark.parametrize("ns,nt,depth", [(1, 1, 2), (7, 40, 2), (5, 600, 2), (7, 5000, 3)])
def test_infinite_strength(gpu_lib, problem, ns, nt, depth):
    rng = np.random.default_rng(ns + nt)
    w = 2 if problem == engine.HELMHOLTZ else 1
    xs, xt = rng.uniform(0.01, 0.11, (ns, 3)), rng.uniform(0.01, 0.11, (nt, 3))
    nrm = np.tile([0.0, 0.0, 1.0], (ns, 1))
    orders = [0] + [6] * depth
    cfg = engine.SolverConfig(problem, depth, orders, list(orders), 6.0, (-0.51,) * 3, 1.02,
                              engine.FP32, engine.POTENTIAL | engine.GRADIENT)
    zero = np.zeros(ns * w)
    with engine.Solver(cfg) as s:
        s.set_sources(xs, nrm).set_strengths(zero).set_targets(xt).run()   # no far field
        for i in range(ns):
            q = rng.uniform(0.5, 1.0, ns * w)
            q[i * w] = np.inf
            fields = []
            for dip in (None, zero):
                s.set_strengths(q, dip)
                s.evaluate()
                fields.append(np.concatenate([np.ravel(f) for f in s.field()]))
            assert np.all(np.isinf(fields[1]))
            assert np.array_equal(fields[0], fields[1])


# the argument after the reduction is within half a unit of pi/4 (0.9e-16), the
# series round to about one of 1 (1.5e-16), and CUDA's own values are within 2
# units (2.2e-16): 5e-16
@pytest.mark.parametrize("xmax", [3.2, 1e3, 1e5, 1.6e5])     # (the library's above 1e5)
def test_fp64_sincos(gpu_lib, xmax):
    assert engine.selftest_sincos64(xmax, 200_000) <= 5e-16


# many wavelengths between the points (k r to 2e4 and, where the library's
# sincos takes over, 2.6e5): r is a few roundings off on either side, k r
# times 1e-15, and so is the phase
@pytest.mark.parametrize("k", [3e3, 3e4, 4e5])
def test_near_high_wavenumber(gpu_lib, k):
    rng = np.random.default_rng(5)
    ns, nt = 129, 520
    xs, xt = rng.uniform(0.01, 0.24, (ns, 3)), rng.uniform(0.01, 0.24, (nt, 3))
    xs[:, 0] += 0.255 * (np.arange(ns) % 2)
    q = rng.uniform(0.5, 1.0, (ns, 2))
    cfg = engine.SolverConfig(engine.HELMHOLTZ, 2, [0, 8, 8], [0, 8, 8], k, (-0.51,) * 3, 1.02,
                              engine.FP64, engine.POTENTIAL | engine.GRADIENT)
    with engine.Solver(cfg) as s:
        pot, grad = s.set_sources(xs).set_strengths(q.ravel()).set_targets(xt).run().field()
    P, G = _direct(engine.HELMHOLTZ, k, xs, q[:, 0] + 1j * q[:, 1], None, None, xt)
    tol = 1e-15 * k * np.linalg.norm(xt[:, None] - xs[None], axis=2).max()
    assert np.linalg.norm(pot[0::2] + 1j * pot[1::2] - P) <= tol * np.linalg.norm(P)
    assert np.linalg.norm(grad[0::2] + 1j * grad[1::2] - G.ravel()) <= tol * np.linalg.norm(G)


# FP64 potentials round the sum once per term: as far from the exact sum as a
# plain FP64 sum in the same order (over 4000 terms of one sign the sum's
# roundings are all that counts, and two per term would be sqrt(2) of it; the
# spread of the mean over 256 values is about 5%)
def test_fp64_sum(gpu_lib):
    rng = np.random.default_rng(8)
    ns, nt, k = 4000, 128, 2.0
    xs, xt = rng.uniform(0.01, 0.24, (ns, 3)), rng.uniform(0.01, 0.24, (nt, 3))
    q = rng.uniform(0.5, 1.0, (ns, 2))
    cfg = engine.SolverConfig(engine.HELMHOLTZ, 2, [0, 8, 8], [0, 8, 8], k, (-0.51,) * 3, 1.02,
                              engine.FP64, engine.POTENTIAL)
    with engine.Solver(cfg) as s:
        pot = s.set_sources(xs).set_strengths(q.ravel()).set_targets(xt).run().field()[0]
        order = s.tree(2)[0]

    def terms(T):
        d = xt.astype(T)[:, None] - xs.astype(T)[None, order]
        kr = T(k) * np.sqrt((d * d).sum(2))
        a, b = np.sin(kr) / kr, -np.cos(kr) / kr
        qr, qi = q[order].astype(T).T
        return np.stack((a * qr - b * qi, b * qr + a * qi), 2)

    exact = terms(np.longdouble).sum(1)
    plain = np.cumsum(terms(np.float64), axis=1)[:, -1]
    err = [np.linalg.norm((f - exact).astype(float))
           for f in (4 * np.pi * pot.reshape(nt, 2).astype(np.longdouble), plain)]
    assert err[0] <= 1.2 * err[1]
