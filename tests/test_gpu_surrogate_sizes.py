"""The local-linear surrogates at the edges of their launches against the
oracle, bit for bit: every dimension the regression is specialised for and
the general one, fewer samples than a regression takes, grids of one and of
several CTAs."""
import numpy as np
import pytest

from oracle import pyoracle as po
from transportoptimiser_gb300 import simulate_gpu as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sem", [0, 1])
@pytest.mark.parametrize("n,d,R", [(2, 1, 5), (60, 1, 65), (130, 2, 33), (500, 3, 11), (777, 4, 6),
                                   (300, 5, 3)])
def test_rov_surrogate_sizes(ctx, n, d, R, sem):
    rng = np.random.default_rng(n + d)
    pred = rng.uniform(0.05, 0.6, (d, n)).astype(np.float32)
    y = (rng.standard_normal(n) - 1.0).astype(np.float32)
    ysd = np.abs(rng.standard_normal(n)).astype(np.float32)
    m, s = sg.buildSurrogateROVCUDA(pred.astype(np.float64), y.astype(np.float64),
                                    ysd.astype(np.float64), R, sem=sem, ctx=ctx)
    assert np.array_equal(m.astype(np.float32), po.build_surrogate_nd(pred, y, R, sem=sem, clip=1))
    assert np.array_equal(s.astype(np.float32), po.build_surrogate_nd(pred, ysd, R, sem=sem, clip=0))
