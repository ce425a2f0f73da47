"""Training samples on ragged grids and lattices against the numpy oracle: lines shorter and longer than
the filter's 32-cell rows, its blocks of rows and chunks of planes with remainders, a lattice that
leaves no whole march of rows, FP32 and FP64 contexts, and the filtered field's statistics."""
import numpy as np
import pytest

import oracle.closure as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("C,sx,sz,ox,oz", [((3, 2, 1), 1, 1, 0, 0), ((33, 9, 5), 1, 1, 0, 0), ((40, 17, 23), 3, 2, 1, 1),
                                           ((70, 8, 3), 8, 3, 7, 2), ((64, 33, 40), 4, 4, 0, 3)])
def test_samples_match_oracle(ark, port, C, sx, sz, ox, oz, prec):
    p = port.channel_params(*C, re_b=2000.0, seed=8, amp=0.15)
    gp = ark.make_params(*C, vis=p["nu"], sound=p["sound"], rho0=p["rho0"], cfl=p["cfl"], lx=p["lx"], ly=p["ly"], lz=p["lz"],
                         ub=p["ub"], precision=ark.FP64 if prec == "fp64" else ark.FP32)
    with ark.Context(gp) as c, ark.ClosureData(C[0] * C[1] * C[2]) as d:
        c.upload(port.channel_state(p))
        c.step(2)
        c.sync()
        c.closure_sample(d, sx=sx, sz=sz, ox=ox, oz=oz, u_tau=0.05)
        F, T = d.get()
        stats = d.filtered_stats()
        u = [port.interior(n, c.get(n)) for n in ("u1nCon", "u2nCon", "u3nCon")]
    dx = tuple(p[n] / k for n, k in zip(("lx", "ly", "lz"), C))
    tgt, ub = oc.target(u, dx, p["nu"])
    pick = lambda a: a[oz::sz, :, ox::sx]
    Fo, To = pick(oc.features(ub, dx, p["ly"], 0.05, p["nu"])).reshape(-1, oc.NIN), pick(tgt).ravel()
    assert F.shape == Fo.shape
    # a row is FP64 rounded to FP32 (2^-24); an n-th root of an invariant that cancels to FP64 rounding
    # (1e-14 of |A|^n, some fifty operations) is off by at most the n-th root of that
    norm = (np.abs(Fo[:, 1]) + np.abs(Fo[:, 2]) + np.abs(Fo[:, 0]))[:, None]
    root = np.array([1, 2, 2, 3, 3, 4, 6, 1, 1, 1])
    # on the centre row of an odd C2 the height is zero up to its last bit, so its sign (features 7 and 8:
    # -sgn(y) S_12, -sgn(y) W_12) is either one's
    if C[1] % 2:
        mid = pick(np.broadcast_to((np.arange(C[1]) == C[1] // 2)[None, :, None], u[0].shape)).ravel()
        F[mid, 7:9] = Fo[mid, 7:9] = 0.0
    assert np.all(np.abs(F - Fo) <= 2.0**-23 * np.abs(Fo) + 1e-14 ** (1.0 / root) * norm), np.abs(F - Fo).max(axis=0)
    # the target: products of order U^2 cancel against filtered ones (1e-15 each), over 2 |S| nu
    tol = 2.0**-23 * np.abs(To) + 1e-13 / (p["nu"] * np.maximum(Fo[:, 1], 1e-12))
    assert np.all(np.abs(T - To) <= tol), np.abs(T - To).max()
    means = [ub[0], ub[1], ub[2], ub[0] ** 2, ub[1] ** 2, ub[2] ** 2, ub[0] * ub[1], ub[0] * ub[2], ub[1] * ub[2]]
    n = C[0] * C[2]
    for q, a in enumerate(means):
        assert np.all(np.abs(stats[:, q] - a.mean(axis=(0, 2))) <= (4 * n + 40) * 2.0**-53 * (np.abs(a).mean(axis=(0, 2)) + 1e-3)), q
