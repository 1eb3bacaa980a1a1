"""Host arrays larger than the context's pinned staging buffer (64 MiB) go
through it piece by piece: results against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import pyoracle as po
from transportoptimiser_gb300 import simulate_gpu as sg

pytestmark = pytest.mark.gpu
PARAMS = np.array([0.05, 0.04, 0.02, 0.0, 0.5, 0.0, 0.0, 0.4], np.float32)


def test_download_in_pieces(ctx):
    paths = (64 << 20) // 4 + 777
    m = dict(N=1, init_pops=np.array([30.0], np.float32), caps=np.array([50.0], np.float32),
             mmm=np.array([[[0.9]]], np.float32))
    end, _ = sg.simulateMTECUDA([m], [PARAMS], paths, 1, seed=3, sem=1, ctx=ctx)
    ref = po.simulate_mte(paths, 1, 1, 1.0, PARAMS, m["init_pops"], m["caps"], m["mmm"][0], 3, 0, 0, 1,
                          threads=8)
    assert np.array_equal(end[:, 0].astype(np.float32), ref)


def test_upload_in_pieces(ctx):
    S, n, paths = 19, 958, 8                    # 70 MB of matrices, padded to 960
    rng = np.random.default_rng(1)
    models = []
    for _ in range(S):
        mm = np.zeros((n, n), np.float32)
        mm[np.arange(n), rng.integers(0, n, n)] = rng.uniform(0.1, 1.0, n).astype(np.float32)
        caps = (50 * rng.integers(4, 101, n)).astype(np.float32)
        models.append(dict(N=n, init_pops=(caps / 2).astype(np.float32), caps=caps, mmm=mm[None]))
    end, _ = sg.simulateMTECUDA(models, [PARAMS] * S, paths, 2, seed=3, sem=1, ctx=ctx)
    for s, m in enumerate(models):
        ref = po.simulate_mte(paths, 2, n, 1.0, PARAMS, m["init_pops"], m["caps"], m["mmm"][0], 3, 0, s,
                              1, threads=8)
        assert np.array_equal(end[:, s].astype(np.float32), ref), s
