"""Small grids (and one of several waves), whose sweeps are cut into chunks of a line and short segments: every interior array
against the oracle bit for bit (FP64), and FP32 with the separate sweeps against the folded ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELLS = ["roCon", "u1Con", "u2Con", "u3Con", "ronCon", "u1nCon", "u2nCon", "u3nCon"]
FACES = [f"{v}{d}" for d in "123" for v in ("p", "u1", "u2", "u3")]


def params(ark, p, px, pz, precision):
    gp = ark.make_params(p["C1"], p["C2"], p["C3"], vis=p["nu"], sound=p["sound"], rho0=p["rho0"], cfl=p["cfl"], lx=p["lx"],
                         ly=p["ly"], lz=p["lz"], ub=p["ub"], precision=precision)
    gp.periodic_x, gp.periodic_z = px, pz
    return gp


def run(ark, p, st, px, pz, precision, steps=4):
    with ark.Context(params(ark, p, px, pz, precision)) as c:
        c.upload(st)
        c.step(steps)
        c.sync()
        return c.download(CELLS + FACES)


# lines shorter than, equal to and longer than a chunk's 31 new positions (C1 + 2 positions a line,
# several lines in one chunk, a line over several chunks), one to three layers, single rows
@pytest.mark.parametrize("px,pz", [(1, 1), (0, 0)])
@pytest.mark.parametrize("C", [(1, 1, 1), (3, 2, 5), (29, 3, 2), (30, 4, 3), (31, 5, 1), (61, 3, 7), (64, 32, 32), (130, 6, 3)])
def test_fp64_small_grids_match_oracle(ark, port, C, px, pz):
    p = port.channel_params(*C, seed=17)
    st = port.channel_state(p)
    st["condition"][0, 1:2, 1:2] = 1.0  # a solid ghost cell, and one in the middle where there is room
    if min(C) > 2:
        st["condition"][2, 2, 2] = 1.0
        for n in CELLS:
            if n[0] == "u":
                st[n][2, 2, 2] = 0.0
    o = port.Port(p, periodic_x=bool(px), periodic_z=bool(pz))
    o.load(st)
    o.run(4)
    out = run(ark, p, st, px, pz, ark.FP64)
    for n in CELLS + FACES:
        a, b = port.interior(n, out[n]), port.interior(n, o.get(n))
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint64), np.ascontiguousarray(b).view(np.uint64)), n


@pytest.mark.parametrize("px,pz", [(1, 1), (0, 1), (1, 0)])
@pytest.mark.parametrize("C", [(5, 3, 2), (30, 4, 9), (48, 20, 24), (70, 33, 5), (150, 10, 31), (256, 5, 3), (96, 64, 200)])
def test_fp32_separate_sweeps_equal_folded_on_small_grids(ark, port, monkeypatch, C, px, pz):
    p = port.channel_params(*C, seed=23)
    st = port.channel_state(p)
    outs = []
    for form in ("0", "5"):
        monkeypatch.setenv("ARK_PHASE2_FUSED", form)
        outs.append(run(ark, p, st, px, pz, ark.FP32))
    for n in CELLS + FACES:
        a, b = (np.ascontiguousarray(port.interior(n, o[n])) for o in outs)
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), n
