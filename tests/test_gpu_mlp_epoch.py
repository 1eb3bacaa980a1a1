"""Training's epoch launches where their shape changes: batches below, at and
above a tile of 128 rows, a short last batch with fewer tiles than the
others, one step an epoch - against Adam on the host over the gradients of
the same rows in the same order."""
import numpy as np
import pytest

from transportoptimiser_gb300 import mlp

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1


def _orders(n, epochs, state):
    """Fisher-Yates orders of a splitmix64 stream."""
    out = []
    for _ in range(epochs):
        r = list(range(n))
        for i in range(n - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & M64
            z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & M64
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
            j = (z ^ (z >> 31)) % (i + 1)
            r[i], r[j] = r[j], r[i]
        out.append(np.array(r))
    return out


@pytest.mark.parametrize("n,batch", [(5, 9), (130, 127), (256, 128), (300, 299), (700, 384)])
def test_epochs_match_host_adam(ctx, n, batch):
    f = np.float32
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, mlp.IN)).astype(f)
    t = rng.normal(size=(n, mlp.OUT)).astype(f)
    p = mlp.init_params(3)
    got, curve = mlp.train_raw(p, x, t, epochs=2, batch=batch, lr=1e-3, seed=11, ctx=ctx)
    m, v, b1, b2, step, losses = np.zeros_like(p), np.zeros_like(p), f(0.9), f(0.999), 0, []
    for order in _orders(n, 2, 11):
        total = 0.0
        for s in range(0, n, batch):
            rows = order[s:s + batch]
            g, loss = mlp.grad(p, x[rows], t[rows], ctx)
            total += loss * rows.size
            step += 1
            m = b1 * m + (f(1) - b1) * g
            v = b2 * v + (f(1) - b2) * g * g
            c1, c2 = f(1) - f(float(b1) ** step), f(1) - f(float(b2) ** step)
            p = p - f(1e-3) * (m / c1) / (np.sqrt(v / c2) + f(1e-8))
        losses.append(total / n)
    # the steps differ by a rounding of the bias corrections at most
    np.testing.assert_allclose(got, p, rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(curve, losses, rtol=1e-6)


def test_more_tiles_than_sms_match_host_adam(ctx):
    """A batch of 154 tiles, which are not all at work at once: steps of three
    launches in place of the epoch's one."""
    test_epochs_match_host_adam(ctx, 20000, 19600)
