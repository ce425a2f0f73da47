"""The statistics of a state against the same sums in numpy: rows shorter and longer than a warp, fewer
and more planes than the blocks of a y plane take at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("C", [(1, 1, 1), (3, 1, 9), (33, 5, 8), (70, 3, 130), (96, 64, 20)])
def test_statistics_match_numpy(ark, port, C, prec):
    p = port.channel_params(*C, seed=5)
    st = port.channel_state(p)
    if min(C) > 2:
        st["condition"][2, 2, 2] = 1.0  # a solid cell: out of the profile and the sums
    gp = ark.make_params(*C, precision=ark.FP64 if prec == "fp64" else ark.FP32)
    with ark.Context(gp) as c:
        c.upload(st)
        c.step(2)
        c.sync()
        ro, u1, u2, u3 = (port.interior(n, c.get(n)) for n in ("ronCon", "u1nCon", "u2nCon", "u3nCon"))
        fluid = port.interior("condition", st["condition"]) == 0
        prof, _ = c.mean_profile()
        s, planes, energy = c.sums(), c.plane_stats(), c.kinetic_energy()
    fixed = lambda a: int(np.rint(a[fluid] * 2.0**32).astype(np.int64).sum()) * 2.0**-32
    # integer sums: the same to the last bit (FP32 density comes back as ro0 + its stored deviation, as summed)
    assert s.cells == fluid.sum()
    assert [s.mass, s.momentum1, s.momentum2, s.momentum3] == [fixed(ro), fixed(ro * u1), fixed(ro * u2), fixed(ro * u3)]
    assert s.kinetic == fixed((u1 * u1 + u2 * u2 + u3 * u3) / 2)
    for j in range(C[1]):
        f = fluid[:, j]
        assert prof[j] == (int(np.rint(u1[:, j][f] * 2.0**32).astype(np.int64).sum()) * 2.0**-32) / f.sum()
    # FP64 sums of n terms: each addition and product off by at most 2^-53 of the sum of magnitudes
    n = C[0] * C[2]
    pairs = [u1, u2, u3, u1 * u1, u2 * u2, u3 * u3, u1 * u2, u1 * u3, u2 * u3]
    for q, a in enumerate(pairs):
        bound = 2 * (n + 2) * 2.0**-53 * np.abs(a).mean(axis=(0, 2))
        assert np.all(np.abs(planes[:, q] - a.mean(axis=(0, 2))) <= bound), q
    e = float(((u1 * u1 + u2 * u2 + u3 * u3) / 2).sum()) * gp.lx * gp.ly * gp.lz
    assert abs(energy - e) <= 2 * (n * C[1] + 4) * 2.0**-53 * e
