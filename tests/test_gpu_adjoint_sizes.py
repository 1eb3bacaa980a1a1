"""The population sweeps of the frozen-policy sensitivities where their layout
changes course, against the FP64 oracle and its central differences: path
counts around a tile of 64, patch counts around a group of four and where
the next year's rows no longer fit in shared memory beside the others, years
around a checkpoint interval of 10, controls no entry or some entries
distinguish."""
import numpy as np
import pytest

from oracle import pyoracle as po
from transportoptimiser_gb300._capi import TransOptError
from transportoptimiser_gb300.adjoint import FrozenPolicy, theta_from_problem

pytestmark = pytest.mark.gpu


def _problem(N, nnz, P, Y, C, S, seed):
    rng = np.random.default_rng(seed)
    hz = np.linspace(0.0, 0.4, C)
    species, cross = [], []
    for s in range(S):
        x = (rng.integers(0, 3, (N, N)) * (rng.random((N, N)) < 0.6)).astype(np.int32)  # [l][k]
        m = np.zeros((N, N))
        for k in range(N):
            m[k, rng.choice(N, size=min(N, int(rng.integers(0, 2 * nnz + 1))), replace=False)] = 1.0
        m *= rng.random((N, N)) * 1.5 / max(nnz, 1)
        mmm = np.stack([m * np.exp(-x.T * h) for h in hz])
        ip = rng.integers(100, 2500, N).astype(np.float32)
        species.append(dict(N=N, params=np.array([0.05, 0.06, 0.05, 0, 0.5, 0.1, 0.2, 0.4], np.float32),
                            init_pops=ip, caps=2 * ip, mmm=mmm.astype(np.float32)))
        cross.append(x)
    unc = np.array([[1, 1, 0.1, 0.2, 0, 0], [1, 1, 0.2, 0.35, 0.1, 0.2]], np.float32)
    pr = dict(n_paths=P, n_years=Y, dim_res=4, dt=1.0, rrr=7.0, unit_cost=0.5, unit_revenue=1.2,
              seed=9, road=2, sem=1, species=species,
              flows=np.linspace(0, 100, C).astype(np.float32), uncert=unc.reshape(-1),
              fuel_costs=np.array([0.3], np.float32), fuel_idx=np.array([0], np.int32),
              ore_content=np.array([0.8], np.float32), ore_sd=np.array([0.05], np.float32),
              demand_idx=-1)
    ctl = rng.integers(0, C, (Y, P)).astype(np.int32)
    return pr, cross, hz, ctl


@pytest.mark.parametrize("N,nnz,P,Y,C,S", [
    (1, 1, 1, 1, 1, 1), (3, 2, 33, 9, 2, 1), (4, 2, 64, 10, 3, 3), (65, 4, 65, 11, 3, 2),
    (70, 3, 20, 21, 8, 1), (400, 3, 3, 4, 3, 1), (512, 2, 5, 11, 2, 1)])
def test_sweeps_match_fp64(ctx, N, nnz, P, Y, C, S):
    pr, cross, hz, ctl = _problem(N, nnz, P, Y, C, S, N + P)
    th = theta_from_problem(pr, hz)
    out, J = FrozenPolicy(pr, ctl, cross, hz, ctx).jacobian(th)
    np.testing.assert_allclose(out, po.adjoint_forward(pr, ctl, cross, hz, th), rtol=1e-4)
    for i in range(th.size):
        h = 1e-4 * max(abs(th[i]), 1.0)
        d = np.eye(th.size)[i] * h
        fd = (po.adjoint_forward(pr, ctl, cross, hz, th + d) -
              po.adjoint_forward(pr, ctl, cross, hz, th - d)) / (2 * h)
        scale = np.abs(J).max(axis=1)
        assert np.all(np.abs(J[:, i] - fd) <= 2e-3 * np.abs(fd) + 1e-3 * scale), (i, J[:, i], fd)


def _overflow_problem(M, ip, cap):
    pr, _, _, _ = _problem(1, 1, 3, 2, 1, 1, 0)
    M = np.asarray(M, np.float32)
    C, N = M.shape[0], M.shape[1]
    prm = np.array([-0.05, -0.05, 0, 0, 0.5, 0, 0, 0], np.float32)
    pr.update(species=[dict(N=N, params=prm, init_pops=np.array(ip, np.float32),
                            caps=np.array(cap, np.float32), mmm=M)],
              flows=np.zeros(C, np.float32))
    return pr, [np.zeros((N, N), np.int32)], np.zeros(C)


def _end(ctx, pr, cross, hz, ctl):
    ctl = np.repeat(np.array(ctl, np.int32)[:, None], pr["n_paths"], axis=1)
    pr = dict(pr, n_years=ctl.shape[0])
    out, tape = FrozenPolicy(pr, ctl, cross, hz, ctx).forward(theta_from_problem(pr, hz), False)
    return out[1]


def test_overflowing_population_stays_infinite(ctx):
    # 1e20 (1 + 0.05 (1e20 - 1)) overflows; infinite from then on
    pr, cross, hz = _overflow_problem([[[1.0]]], [1e20], [1.0])
    assert _end(ctx, pr, cross, hz, [0, 0, 0]) == np.inf


def test_infinite_patch_leaves_the_others_alone(ctx):
    # the first patch overflows under control 1 and is left behind under
    # control 2; the second receives from it under control 0 only
    M = [[[1, 0], [1e-30, 1]], [[1e25, 0], [0, 1]], [[0, 0], [0, 1]]]
    pr, cross, hz = _overflow_problem(M, [1e6, 500], [1e6, 1000])
    x = 500.0
    for _ in range(3):
        x *= 1 - 0.05 * (1000 - x) / 1000
    np.testing.assert_allclose(_end(ctx, pr, cross, hz, [1, 2, 2]), x, rtol=1e-5)


def test_most_parameters(ctx):
    """Eight processes, species and controls: 40 sensitivities an output."""
    pr, cross, hz, ctl = _problem(4, 2, 5, 3, 8, 8, 1)
    pr["uncert"] = np.tile(np.array([1, 1, 0.1, 0.2, 0.1, 0.2], np.float32), 8)
    th = theta_from_problem(pr, hz)
    assert th.size == 40
    out, J = FrozenPolicy(pr, ctl, cross, hz, ctx).jacobian(th)
    np.testing.assert_allclose(out, po.adjoint_forward(pr, ctl, cross, hz, th), rtol=1e-4)
    for i in range(th.size):
        h = 1e-4 * max(abs(th[i]), 1.0)
        d = np.eye(th.size)[i] * h
        fd = (po.adjoint_forward(pr, ctl, cross, hz, th + d) -
              po.adjoint_forward(pr, ctl, cross, hz, th - d)) / (2 * h)
        scale = np.abs(J).max(axis=1)
        assert np.all(np.abs(J[:, i] - fd) <= 2e-3 * np.abs(fd) + 1e-3 * scale), (i, J[:, i], fd)


def test_processes_and_controls_out_of_range(ctx):
    """Profits of processes that do not exist are refused; under a control that
    does not exist nothing earns or survives."""
    pr, cross, hz, ctl = _problem(4, 2, 5, 3, 2, 1, 1)
    th = theta_from_problem(pr, hz)
    for bad in (dict(fuel_idx=np.array([2], np.int32)), dict(fuel_idx=np.array([-1], np.int32)),
                dict(demand_idx=2), dict(fuel_costs=np.ones(2, np.float32),
                                         fuel_idx=np.array([0, 1], np.int32))):
        with pytest.raises(TransOptError) as e:
            FrozenPolicy(dict(pr, **bad), ctl, cross, hz, ctx).forward(th, False)
        assert e.value.status == 1
    out, _ = FrozenPolicy(pr, np.full_like(ctl, 1 << 30), cross, hz, ctx).forward(th, False)
    assert np.all(out == 0.0)


def test_many_paths_tape(ctx):
    """More (species, tile) pairs than CTAs at work at a time: the sweeps equal
    those of a few paths, and the tape keeps checkpoints by path, not a
    segment's scratch (the free memory before and while it is held)."""
    torch = pytest.importorskip("torch")
    pr, cross, hz, ctl = _problem(64, 2, 30000, 21, 2, 2, 5)
    th = theta_from_problem(pr, hz)
    model = FrozenPolicy(pr, ctl, cross, hz, ctx)
    free = torch.cuda.mem_get_info()[0]
    out, tape = model.forward(th)
    held = free - torch.cuda.mem_get_info()[0]
    S, P, Y = 2, 30000, 21
    paths = 4 * (S * (Y // 10 + 1 + 10) * 64 + S * Y * 2 + Y) + 8 * (1 + S + th.size)
    assert held <= paths * P + (8 << 20), held      # checkpoints and one segment; lists and rounding
    g = model.backward(tape, [1.0, 2.0, -1.0])
    model.free(tape)
    parts = np.zeros_like(g)
    few = np.zeros(3)
    for p0 in range(0, P, 5000):                    # Philox streams are a path's own: masks, not slices
        w = slice(p0, p0 + 5000)
        sub = np.full_like(ctl, 2)                  # no control: nothing earns or migrates
        sub[:, w] = ctl[:, w]
        m = FrozenPolicy(pr, sub, cross, hz, ctx)
        o, t = m.forward(th)
        few += o
        parts += m.backward(t, [1.0, 2.0, -1.0])
        m.free(t)
    np.testing.assert_allclose(out, few, rtol=1e-12)
    np.testing.assert_allclose(g, parts, rtol=1e-9, atol=1e-12)
