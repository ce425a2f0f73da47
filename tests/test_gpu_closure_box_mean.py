"""The box filter of the training data rounds as its definition does: the sums of a box along x, y and z in
that order and one correctly rounded quotient by 27.  On a grid of one cell per plane the filtered
field's plane means are its values, so they equal the same operations in numpy bit for bit; velocities of
ordinary size, zeros and ones whose sums are subnormal."""
import numpy as np
import pytest

import oracle.closure as oc

pytestmark = pytest.mark.gpu


def box_mean(u):
    """u (C3, C2, C1): periodic x and z, a solid neighbour in y counts as minus the cell."""
    x = (np.roll(u, 1, 2) + u) + np.roll(u, -1, 2)
    lo, hi = np.roll(x, 1, 1), np.roll(x, -1, 1)
    lo[:, 0], hi[:, -1] = -x[:, 0], -x[:, -1]
    xy = (lo + x) + hi
    return ((np.roll(xy, 1, 0) + xy) + np.roll(xy, -1, 0)) / 27.0


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("scale", [1.0, 0.0, 1e-308])
def test_filtered_values_are_the_rounded_quotients(ark, port, scale, prec):
    if prec == "fp32" and scale:
        scale = 1.0 if scale == 1.0 else 1e-44
    C = (1, 257, 1)
    p = port.channel_params(*C, re_b=2000.0, seed=8, amp=0.15)
    st = port.channel_state(p)
    r = np.random.default_rng(5)
    for n in ("u1nCon", "u2nCon", "u3nCon"):
        st[n][...] = r.normal(0.5, 1.0, st[n].shape) * scale
    gp = ark.make_params(*C, vis=p["nu"], sound=p["sound"], rho0=p["rho0"], cfl=p["cfl"], lx=p["lx"], ly=p["ly"], lz=p["lz"],
                         ub=p["ub"], precision=ark.FP64 if prec == "fp64" else ark.FP32)
    with ark.Context(gp) as c, ark.ClosureData(C[1]) as d:
        c.upload(st)
        c.closure_sample(d, sx=1, sz=1, ox=0, oz=0, u_tau=0.05)
        F, _ = d.get()
        stats = d.filtered_stats()
        u = [port.interior(n, c.get(n)) for n in ("u1nCon", "u2nCon", "u3nCon")]
    assert np.isfinite(F).all()
    for m in range(3):
        want = box_mean(np.asarray(u[m], np.float64))[0, :, 0]
        assert np.array_equal(stats[:, m], want), (m, np.abs(stats[:, m] - want).max())
        # and it is the mean of the definition's three passes, to their nine roundings
        assert np.all(np.abs(want - oc.box_filter(u[m], -1.0)[0, :, 0]) <= 16 * 2.0**-53 * np.abs(u[m]).max() + 1e-320)
