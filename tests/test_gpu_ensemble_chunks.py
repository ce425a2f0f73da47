"""Small ensembles, whose staged chunks and x2 segments follow the members' total size: every member equals
the same channel advanced alone, bit for bit, for one member, a few of one size and a few of mixed sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ["roCon", "u1Con", "u2Con", "u3Con", "ronCon", "u1nCon", "u2nCon", "u3nCon"] + [
    f"{v}{d}" for d in "123" for v in ("p", "u1", "u2", "u3")]


@pytest.mark.parametrize("sizes", [[(40, 9, 5)], [(64, 24, 48)] * 3, [(32, 32, 32), (96, 40, 31), (128, 64, 24), (33, 17, 64)],
                                   [(128, 64, 64)] * 6])
def test_members_of_small_ensembles_equal_single_contexts(ark, port, sizes):
    ps = [ark.make_params(*C, precision=ark.FP32) for C in sizes]
    sts = [ark.channel_init(p, seed=60 + q) for q, p in enumerate(ps)]
    with ark.Ensemble(ps) as E:
        for q, st in enumerate(sts):
            E.upload(q, st)
        E.step(5)
        E.sync()
        got = [E.download(q, NAMES) for q in range(len(ps))]
    for q, (p, st) in enumerate(zip(ps, sts)):
        with ark.Context(p) as c:
            c.upload(st)
            c.step(5)
            c.sync()
            want = c.download(NAMES)
        for n in NAMES:
            a, b = (np.ascontiguousarray(port.interior(n, x[n])) for x in (got[q], want))
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), (q, n)
