"""A run of many steps (graphs of several steps, then single ones) equals the same steps one call at a
time bit for bit: both precisions, from either face generation and level, with averages and with the
learned closure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["roCon", "u1Con", "u2Con", "u3Con", "ronCon", "u1nCon", "u2nCon", "u3nCon"] + [
    f"{v}{d}" for d in "123" for v in ("p", "u1", "u2", "u3")]


@pytest.mark.parametrize("C", [(20, 9, 12), (70, 40, 33)])
@pytest.mark.parametrize("kind", ["fp64", "fp32", "closure"])
def test_many_steps_equal_single_steps(ark, port, C, kind):
    p = port.channel_params(*C, seed=41)
    st = port.channel_state(p)
    gp = ark.make_params(*C, precision=ark.FP64 if kind == "fp64" else ark.FP32)
    with ark.Context(gp) as a, ark.Context(gp) as b, ark.Mlp(seed=2) as net:
        for c in (a, b):
            c.upload(st)
            if kind == "closure":
                c.set_closure(net, 0.05)
            c.set_averaging(True)
        a.step(1)       # start from the other face generation
        a.phase1()      # and, with the pieces, from the other level
        a.step(64 + 11)
        a.step(16)      # the captured chain again
        for n, f in ((1, b.step), (0, None), (75, b.step), (16, b.step)):
            if f is None:
                b.phase1()
            else:
                for _ in range(n):
                    f(1)
        a.sync()
        b.sync()
        assert a.scalars().nstep == b.scalars().nstep == 92 and a.scalars().time == b.scalars().time
        x, y = a.download(FIELDS), b.download(FIELDS)
        for m in "123":
            x[f"averageU{m}"], y[f"averageU{m}"] = a.get(f"averageU{m}"), b.get(f"averageU{m}")
    for n in x:
        u, v = x[n], y[n]
        if not n.startswith("average"):
            u, v = np.ascontiguousarray(port.interior(n, u)), np.ascontiguousarray(port.interior(n, v))
        assert np.array_equal(u.view(np.uint64), v.view(np.uint64)), n
