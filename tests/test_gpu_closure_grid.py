"""The eddy viscosity of the learned closure does not depend on how its kernel's blocks are dealt: a state
periodic in z over 12 planes, on that many planes (fewer blocks than fit at once), on eight periods
(several rounds) and on 64 (a block per 128 cells, capped), gives the same values bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C1, C2, P = 64, 20, 12


def nut(ark, port, st, p, net, m):
    gp = ark.make_params(C1, C2, P * m, vis=p["nu"], sound=p["sound"], rho0=p["rho0"], cfl=p["cfl"], lx=p["lx"], ly=p["ly"],
                         lz=p["lz"] * m, ub=p["ub"], precision=ark.FP32)
    tiled = {}
    for n, a in st.items():
        k = np.arange(a.shape[0] + P * (m - 1))
        tiled[n] = np.ascontiguousarray(a[1 + (k - 1) % P])
    with ark.Context(gp) as c:
        c.upload(tiled)
        c.set_closure(net, 0.05)
        c.step(1)
        c.sync()
        return c.get("nut")[1:P * m + 1, 1:C2 + 1, 1:C1 + 1]


def test_eddy_viscosity_does_not_depend_on_the_grid_of_blocks(ark, port):
    p = port.channel_params(C1, C2, P, seed=53)
    st = port.channel_state(p)
    with ark.Mlp(seed=5) as net:
        one = nut(ark, port, st, p, net, 1)
        assert np.any(one)
        for m in (8, 64):
            got = nut(ark, port, st, p, net, m)
            for q in range(m):
                assert np.array_equal(got[P * q:P * (q + 1)].view(np.uint64), one.view(np.uint64)), (m, q)
