"""ALGO6's re-simulation in each of its shared-memory layouts - union lists
with the groups' sums, the controls' own lists (more than three controls)
with and without them - and with more groups than the warps hold normals
for, bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_rov_forward import _problem
from transportoptimiser_gb300 import simulate_gpu as sg
from transportoptimiser_gb300._capi import MIG_SPARSE_FP32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nnz,P,Y,C,S", [
    (5, 2, 33, 4, 1, 1), (61, 5, 97, 6, 3, 2), (40, 4, 64, 5, 5, 1), (196, 1, 40, 4, 3, 2),
    (301, 2, 31, 3, 1, 2), (20, 3, 70, 5, 2, 4)])
def test_resimulated_equals_oracle(ctx, N, nnz, P, Y, C, S):
    pr = dict(_problem(N, nnz, P, Y, C, 1, S, N + P), algo=6)
    g = sg.simulateROVCUDA(pr, want=("cond_exp", "opt_cont"), migration=MIG_SPARSE_FP32, ctx=ctx)
    o = po.simulate_rov(pr, threads=8)
    np.testing.assert_array_equal(g["opt_cont"], o["opt_cont"])
    np.testing.assert_array_equal(np.asarray(g["cond_exp"], np.float32), o["cond_exp"])
