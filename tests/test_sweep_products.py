"""FP64 products of the sweeps: every caller names the pipes that take them, and the separate sweep kernels
(the step by its pieces, timed steps, x1 lines chosen by hand) follow the same rule as the captured step.
The step by its pieces equals the oracle bit for bit on both sides of the rule's line."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ark-cpp-mpi_gb300", "csrc")
CELLS = ["roCon", "u1Con", "u2Con", "u3Con", "ronCon", "u1nCon", "u2nCon", "u3nCon"]
FACES = [f"{v}{d}" for d in "123" for v in ("p", "u1", "u2", "u3")]


def test_no_sweep_takes_integer_products_unasked():
    with open(os.path.join(CSRC, "ark_kernels.cuh")) as f:
        text = f.read()
    assert not re.search(r"bool INT\s*=", text)
    sweep = re.search(r"void Launch<T>::sweep\(.*?\n}", text, re.S).group(0)
    assert "int_products(S.g)" in sweep and len(re.findall(r"<T, (?:\d, )?fp64><<<", sweep)) == 3


@pytest.mark.gpu
@pytest.mark.parametrize("C", [(20, 10, 12), (64, 31, 19), (64, 32, 19), (33, 35, 37)])
@pytest.mark.parametrize("px,pz", [(1, 1), (0, 0)])
def test_fp64_step_by_its_pieces_matches_oracle(ark, port, C, px, pz):
    p = port.channel_params(*C, seed=31)
    st = port.channel_state(p)
    o = port.Port(p, periodic_x=bool(px), periodic_z=bool(pz))
    o.load(st)
    o.run(3)
    gp = ark.make_params(*C, vis=p["nu"], sound=p["sound"], rho0=p["rho0"], cfl=p["cfl"], lx=p["lx"], ly=p["ly"], lz=p["lz"],
                         ub=p["ub"], precision=ark.FP64)
    gp.periodic_x, gp.periodic_z = px, pz
    with ark.Context(gp) as c:
        c.upload(st)
        for _ in range(2):
            c.time_step_size()
            c.phase1()
            c.stress_tensor()
            c.use_forces()
            c.phase2()
            c.phase1()
            c.use_forces()
        c.kernel_times(1)  # one step, launch by launch
        out = c.download(CELLS + FACES)
    for n in CELLS + FACES:
        a, b = port.interior(n, out[n]), port.interior(n, o.get(n))
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint64), np.ascontiguousarray(b).view(np.uint64)), n
