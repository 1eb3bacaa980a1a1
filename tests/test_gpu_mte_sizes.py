"""The sparse MTE at the edges of its tiles and layouts against the oracle,
bit for bit: one and two paths a lane, full and ragged tiles, several CTAs an
SM, lists of uneven lengths, both population buffers in shared memory, one of
them in global memory, and lists too long for shared memory."""
import numpy as np
import pytest

from oracle import pyoracle as po
from transportoptimiser_gb300 import simulate_gpu as sg
from transportoptimiser_gb300._capi import MIG_SPARSE_FP32

pytestmark = pytest.mark.gpu


def _model(n, entries, rng):
    """n patches, `entries` origins a destination on average, some far above it."""
    m = np.zeros((n, n), np.float32)
    for k in range(n):
        cnt = n if k % 97 == 5 and entries < n else min(n, int(rng.integers(0, 2 * entries + 1)))
        o = rng.choice(n, cnt, replace=False)
        m[k, o] = rng.uniform(0.001, 1.8 / max(1, min(n, 2 * entries)), cnt).astype(np.float32)
    caps = (50 * rng.integers(4, 101, n)).astype(np.float32)
    return dict(N=n, init_pops=(caps / 2).astype(np.float32), caps=caps, mmm=m[None])


@pytest.mark.parametrize("n,entries,paths,years,sem,jump", [
    (1, 1, 1, 3, 0, 0.0), (3, 2, 33, 18, 1, 0.1), (4, 3, 32, 16, 0, 0.0),
    (41, 6, 65, 17, 1, 0.0), (115, 6, 9700, 5, 0, 0.1), (61, 5, 19999, 4, 1, 0.0),
    (340, 6, 500, 6, 1, 0.0), (340, 6, 9800, 3, 0, 0.1), (430, 8, 9750, 3, 1, 0.0),
    (508, 7, 200, 4, 0, 0.1), (400, 38, 9750, 3, 1, 0.0), (60, 60, 40, 3, 0, 0.0),
    (41, 6, 70, 0, 0, 0.0), (41, 6, 70, 1, 1, 0.1)])
def test_sparse_mte_sizes(ctx, n, entries, paths, years, sem, jump):
    rng = np.random.default_rng(n * 7 + paths)
    m = _model(n, entries, rng)
    params = np.array([0.05, 0.04, 0.02, 0.0, 0.5, 0.3 if jump else 0.0, jump, 0.4], np.float32)
    end, _ = sg.simulateMTECUDA([m], [params], paths, years, seed=9, road=3, sem=sem,
                                migration=MIG_SPARSE_FP32, ctx=ctx)
    ref = po.simulate_mte(paths, years, n, 1.0, params, m["init_pops"], m["caps"], m["mmm"][0],
                          9, 3, 0, sem, threads=8)
    assert np.array_equal(end[:, 0].astype(np.float32), ref)
