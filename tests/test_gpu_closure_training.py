"""The training kernels at the edges of their tiles (128 samples, 16 per warp) and block counts against
the numpy oracle's FP64 gradient, and a few Adam steps against the same in numpy."""
import numpy as np
import pytest

import oracle.closure as oc

pytestmark = pytest.mark.gpu


def net_and_rows(n, seed):
    r = np.random.default_rng(seed)
    theta, mu, sd = r.normal(0, 0.3, oc.NPARAM), r.normal(0, 1, oc.NIN), r.uniform(0.5, 2.0, oc.NIN)
    x = (r.normal(0, 1, (n, oc.NIN)) * sd + mu).astype(np.float32)
    return theta, mu, sd, x, r.uniform(0, 3, n).astype(np.float32)


def used(mu, sd):
    return np.float32(mu).astype(np.float64), 1.0 / np.float32(1.0 / sd).astype(np.float64)


# one sample, a warp's 16 and one more, a tile and one more, every block twice (608 tiles) and a remainder
@pytest.mark.parametrize("first,count", [(0, 1), (3, 16), (0, 17), (5, 127), (0, 128), (1, 129), (0, 608 * 128 + 1)])
def test_gradient_at_tile_edges(ark, first, count):
    theta, mu, sd, x, t = net_and_rows(first + count + 2, 31)
    with ark.ClosureData(len(t)) as d, ark.Mlp(seed=3) as net:
        d.append(x, t)
        net.set(theta, mu, sd)
        loss, g = net.gradient(d, first, count)
    s = slice(first, first + count)
    lo, go = oc.loss_and_grad(oc.bf16(theta), *used(mu, sd), x[s].astype(np.float64), t[s].astype(np.float64))
    # two-term BF16 operands: 2^-16 per product, which a sum of a few dozen products keeps
    assert abs(loss - lo) <= 2e-5 * lo
    assert np.linalg.norm(g - go) <= 2e-4 * np.linalg.norm(go)


def test_adam_steps_match_numpy(ark):
    batch, nb, lr = 200, 3, 1e-3
    theta, mu, sd, x, t = net_and_rows(batch * nb + 7, 32)
    w = np.float32(theta).astype(np.float64)
    m, v = np.zeros_like(w), np.zeros_like(w)
    for b in range(nb):  # batch b takes samples b, b + nb, ...
        at = b + nb * np.arange(batch)
        _, g = oc.loss_and_grad(oc.bf16(w), *used(mu, sd), x[at].astype(np.float64), t[at].astype(np.float64))
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        w = w - lr * (m / (1 - 0.9 ** (b + 1))) / (np.sqrt(v / (1 - 0.999 ** (b + 1))) + 1e-8)
    with ark.ClosureData(len(t)) as d, ark.Mlp(seed=3) as net:
        d.append(x, t)
        net.set(theta, mu, sd)
        net.train(d, epochs=1, batch=batch, lr=lr)
        got, _, _ = net.get()
    # a step moves a weight by at most about lr times sign-like factors; gradients off by 2e-4 move the
    # nearly cancelling ones by a part of that
    assert np.abs(got - w).max() <= nb * lr
    assert np.linalg.norm(got - w) <= 1e-2 * np.linalg.norm(w - np.float32(theta))
