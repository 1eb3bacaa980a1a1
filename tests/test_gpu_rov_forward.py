"""The forward pass's two-paths-a-lane form where its layout changes course,
bit for bit against the oracle: path counts around a tile of 64, species of
few and many patches (a next-year buffer that does and does not fit beside
the lists in shared memory), empty columns, even and odd list lengths, every
number of controls, and the years around a chunk of 16 draws."""
import numpy as np
import pytest

from oracle import pyoracle as po
from transportoptimiser_gb300 import simulate_gpu as sg
from transportoptimiser_gb300._capi import MIG_SPARSE_FP32

pytestmark = pytest.mark.gpu


def _problem(N, nnz, P, Y, C, sem, S, seed):
    rng = np.random.default_rng(seed)
    species = []
    for s in range(S):
        n = N - 3 * s
        m = np.zeros((n, n))
        for k in range(n):
            m[k, rng.choice(n, size=min(n, int(rng.integers(0, 2 * nnz + 1))), replace=False)] = 1.0
        m *= rng.random((n, n)) / max(nnz, 1)
        mmm = np.stack([m * np.exp(-0.3 * c * (rng.random((n, n)) < 0.4)) for c in range(C)])
        ip = rng.integers(100, 2500, n).astype(np.float32)
        species.append(dict(N=n, params=np.array([0.05, 0.05, 0.05, 0, 0.5, 0.1, 0.2, 0.4], np.float32),
                            init_pops=ip, caps=2 * ip, mmm=mmm.astype(np.float32)))
    unc = np.array([[1, 1, 0.1, 0.2, 0, 0], [1, 1, 0.2, 0.35, 0.1, 0.2]], np.float32)
    return dict(n_paths=P, n_years=Y, dim_res=4, dt=1.0, rrr=7.0, unit_cost=0.5, unit_revenue=1.2,
                seed=9, road=2, sem=sem, species=species,
                flows=np.linspace(0, 100, C).astype(np.float32), uncert=unc.reshape(-1),
                fuel_costs=np.array([0.3], np.float32), fuel_idx=np.array([0], np.int32),
                ore_content=np.array([0.8], np.float32), ore_sd=np.array([0.05], np.float32),
                demand_idx=-1)


@pytest.mark.parametrize("N,nnz,P,Y,C,sem,S", [
    (1, 1, 3, 3, 3, 1, 1), (5, 2, 63, 16, 1, 1, 1), (40, 6, 64, 17, 2, 0, 1), (115, 5, 65, 4, 3, 1, 2),
    (333, 8, 130, 5, 3, 1, 2), (372, 9, 40, 5, 3, 1, 1), (480, 7, 70, 4, 3, 1, 1), (300, 14, 33, 4, 3, 0, 1)])
def test_forward_equals_oracle(ctx, N, nnz, P, Y, C, sem, S):
    pr = _problem(N, nnz, P, Y, C, sem, S, N + P)
    g = sg.simulateROVCUDA(pr, want=("cond_exp", "opt_cont", "adj_pops"), migration=MIG_SPARSE_FP32,
                           ctx=ctx)
    o = po.simulate_rov(pr, threads=8)
    a = np.asarray(g["adj_pops"], np.float32).reshape(Y, S, P)[1:]
    np.testing.assert_array_equal(a, np.asarray(o["adj_pops"], np.float32).reshape(Y, S, P)[1:])
    np.testing.assert_array_equal(g["opt_cont"], o["opt_cont"])
    np.testing.assert_array_equal(np.asarray(g["cond_exp"], np.float32), o["cond_exp"])
