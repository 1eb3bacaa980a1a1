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


def _overflowing(others, own, seed):
    """One path whose first patch overflows under control 1, the optimal one
    while valid; where it then falls to zero or stays infinite, the other
    patches decide by the threshold of 1,000.  Their lists are of odd length,
    which are padded, or (own) hold the first patch under control 0 only."""
    m = np.repeat(np.eye(5, dtype=np.float32)[None], 2, axis=0)
    m[:, 4, 4], m[:, 4, 1], m[1, 0, 0] = 0.9, 1e-4, 1e25
    m[0, 1:4, 0] = 1e-30 if own else 0.0
    ip = np.array([1e6, others, others, others, 10], np.float32)
    pr = _problem(5, 1, 1, 7, 2, 1, 1, 0)
    pr["species"][0].update(params=np.array([0.05, 0.05, 0, 1000, 0.5, 0, 0, 5], np.float32),
                            init_pops=ip, caps=2 * ip, mmm=m)
    return dict(pr, algo=6, unit_revenue=10.0, seed=seed)


def _same_where_the_forward_pass_is_finite(ctx, others, own):
    n = 0
    for seed in range(400):
        pr = _overflowing(others, own, seed)
        o = po.simulate_rov(pr, threads=1)
        if not np.isfinite(o["adj_pops"]).all():
            continue
        g = sg.simulateROVCUDA(pr, want=("cond_exp", "opt_cont"), migration=MIG_SPARSE_FP32, ctx=ctx)
        np.testing.assert_array_equal(g["opt_cont"], o["opt_cont"], str(seed))
        np.testing.assert_array_equal(np.asarray(g["cond_exp"], np.float32), o["cond_exp"], str(seed))
        n += 1
    assert n > 100


@pytest.mark.parametrize("own", [False, True])
def test_infinite_patch_leaves_the_others_alone(ctx, own):
    _same_where_the_forward_pass_is_finite(ctx, 5000, own)


def test_infinite_patch_stays_infinite(ctx):
    _same_where_the_forward_pass_is_finite(ctx, 20, False)
