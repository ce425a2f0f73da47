"""Training samples of grids far longer along one axis than a launch's y and z extents reach in tiles (65,535):
the samples at both ends and in the middle equal the ones of a short grid of the same velocities."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_samples_of_a_long_grid(ark, axis):
    n, m = 540_000, 24
    out = []
    for length in (n, m):
        C = [1, 1, 1]
        C[axis] = length
        p = ark.make_params(*C, lx=float(C[0]), ly=float(C[1]), lz=float(C[2]), precision=ark.FP32)
        with ark.Context(p) as c, ark.ClosureData(length) as d:
            st = ark.channel_init(p, seed=1, amp=0.0)
            r = np.random.default_rng(7)
            for name in ("u1nCon", "u2nCon", "u3nCon"):
                a = r.normal(0.0, 1.0, m)  # the same m cells at both ends, and again in the middle
                line = np.zeros(length)
                line[:m] = line[-m:] = line[length // 2 - m // 2:][:m] = a
                shape = [1, 1, 1]
                shape[2 - axis] = length  # host arrays are [k][j][i]
                v = np.zeros(st[name].shape)
                v[1:-1, 1:-1, 1:-1] = line.reshape(shape)
                st[name] = v
            c.upload(st)
            c.closure_sample(d, sx=1, sz=1, ox=0, oz=0, u_tau=0.05)
            out.append(d.get())
    (F, T), (f, t) = out
    assert F.shape[0] == n
    cut = slice(3, m - 3)  # away from the short grid's own ends; feature 9 is the height
    for at in (0, n // 2 - m // 2, n - m):
        for q in range(9) if axis != 1 else range(7):  # (7 and 8 carry the sign of the height)
            np.testing.assert_array_equal(F[at:at + m][cut, q], f[cut, q])
        np.testing.assert_array_equal(T[at:at + m][cut], t[cut])
