"""Re-simulated paths in tiles of 32 (more tiles of 16 than SMs) and at the
edge to tiles of 16, union lists and the controls' own, more groups than
half-warps, bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_rov_forward import _problem
from transportoptimiser_gb300 import simulate_gpu as sg
from transportoptimiser_gb300._capi import MIG_SPARSE_FP32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nnz,P,Y,C,S", [
    (13, 3, 2500, 4, 3, 2), (13, 3, 2431, 4, 3, 1), (9, 2, 2449, 4, 5, 1), (141, 3, 20, 4, 2, 2),
    (70, 2, 2501, 3, 3, 3)])
def test_resimulated_tiles_equal_oracle(ctx, N, nnz, P, Y, C, S):
    pr = dict(_problem(N, nnz, P, Y, C, 1, S, N + P), algo=6)
    g = sg.simulateROVCUDA(pr, want=("cond_exp", "opt_cont"), migration=MIG_SPARSE_FP32, ctx=ctx)
    o = po.simulate_rov(pr, threads=8)
    np.testing.assert_array_equal(g["opt_cont"], o["opt_cont"])
    np.testing.assert_array_equal(np.asarray(g["cond_exp"], np.float32), o["cond_exp"])
