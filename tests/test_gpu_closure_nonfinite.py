"""Training samples of a field with NaN or infinite velocities: features and targets show them as the
velocity-gradient algebra does (matrix products, features 1 and 2 the roots of a positive part, which is 0
of a NaN), and every sample away from them is the one of the field without."""
import numpy as np
import pytest

import oracle.closure as oc

pytestmark = pytest.mark.gpu


def expected(u, dx, ly, nu):
    """The numpy oracle's features, with the positive part of a NaN taken as 0."""
    with np.errstate(all="ignore"):
        f = oc.features([oc.box_filter(a, -1.0) for a in u], dx, ly, 0.05, nu)
    f[..., 1:3] = np.where(np.isnan(f[..., 1:3]), 0.0, f[..., 1:3])
    return f


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("m", [0, 1, 2])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_nonfinite_velocities_show_in_samples(ark, port, bad, m, prec):
    C = (16, 12, 10)
    p = port.channel_params(*C, re_b=2000.0, seed=8, amp=0.15)
    gp = ark.make_params(*C, vis=p["nu"], sound=p["sound"], rho0=p["rho0"], cfl=p["cfl"], lx=p["lx"], ly=p["ly"], lz=p["lz"],
                         ub=p["ub"], precision=ark.FP64 if prec == "fp64" else ark.FP32)
    st = port.channel_state(p)
    rows = []
    for broken in (False, True):
        if broken:
            for n in (f"u{m + 1}nCon", f"u{m + 1}Con"):
                st[n][6, 5, 4] = bad
        with ark.Context(gp) as c, ark.ClosureData(C[0] * C[1] * C[2]) as d:
            c.upload(st)
            c.closure_sample(d, sx=1, sz=1, ox=0, oz=0, u_tau=0.05)
            rows.append(d.get())
            u = [port.interior(n, c.get(n)) for n in ("u1nCon", "u2nCon", "u3nCon")]
    (F0, T0), (F, T) = rows
    assert np.isfinite(F0).all() and np.isfinite(T0).all()
    want = expected(u, tuple(p[n] / k for n, k in zip(("lx", "ly", "lz"), C)), p["ly"], p["nu"]).reshape(-1, oc.NIN)
    # the field has one such cell, inside: its 5 x 5 x 5 neighbourhood at most is touched
    touched = ~np.isfinite(want).all(axis=1)
    assert 27 <= touched.sum() <= 125
    if np.isnan(bad):
        assert np.array_equal(np.isnan(F), np.isnan(want))
    else:  # an invariant of infinite entries may come out infinite or NaN, by the order of its terms
        assert np.array_equal(np.isfinite(F), np.isfinite(want))
    assert np.array_equal(F[touched, 1] == 0.0, want[touched, 1] == 0.0) and np.array_equal(F[touched, 2] == 0.0, want[touched, 2] == 0.0)
    assert np.array_equal(F[~touched], F0[~touched])
    assert np.all(np.isfinite(T) & (T >= 0))
