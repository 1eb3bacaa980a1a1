"""The regressions of the ROV at the sizes where their kernels change course,
bit for bit against the oracle: groups of a few points, of one tile of
points more or less (512), of more points than shared memory holds; every
number of species; both semantics and both algorithms, with and without the
surfaces; ties (profits all equal: no distance is a number), states that
take few values, species below their thresholds; the cell-grid search above
32,768 paths; few queries and many (more than two tiles of 128 an SM)."""
import ctypes

import numpy as np
import pytest

from oracle import pyoracle as po
from transportoptimiser_gb300 import _capi
from transportoptimiser_gb300 import simulate_gpu as sg

pytestmark = pytest.mark.gpu

#        species bins paths years sem algo patches surfaces kind
CASES = [(1, 16, 130, 5, 0, 4, 40, True, ""), (1, 16, 1700, 4, 0, 4, 12, True, ""),
         (2, 8, 2000, 4, 1, 4, 20, False, ""), (3, 5, 300, 5, 1, 4, 30, False, ""),
         (4, 4, 300, 4, 1, 4, 10, True, ""), (4, 8, 2600, 3, 1, 4, 6, False, ""),
         (2, 11, 200, 5, 1, 6, 16, True, ""), (1, 5, 6, 5, 1, 4, 8, True, ""),
         (2, 5, 3, 4, 1, 4, 8, False, ""), (1, 8, 1536, 4, 1, 4, 9, True, ""),
         (1, 4, 33000, 3, 1, 4, 5, False, ""), (2, 4, 13000, 3, 1, 4, 5, False, ""),
         (2, 6, 400, 5, 1, 4, 12, True, "equal profits"),
         (1, 7, 900, 4, 1, 4, 12, False, "few states"), (2, 7, 700, 4, 1, 4, 12, True, "below"),
         (2, 33, 500, 3, 1, 4, 7, True, "")]


def _problem(S, R, P, Y, sem, algo, N, kind):
    rng = np.random.default_rng(S * 1000 + P)
    species = []
    for _ in range(S):
        m = rng.random((N, N)) * (rng.random((N, N)) < 0.4) + np.eye(N)
        m /= m.sum(0, keepdims=True)
        loss = rng.random((N, N)) * 0.3
        mmm = np.stack([m * np.exp(-loss * c) for c in range(3)]).astype(np.float32)
        ip = rng.integers(100, 2500, N).astype(np.float32)
        prm = np.array([0.05, 0.05, 0.05, 0.0, 0.5, 0.0, 0.0, 0.4], np.float32)
        if kind == "few states":
            prm[[2, 7]] = 0.0
        if kind == "below":
            prm[[3, 5, 6]] = [ip.sum() * 0.8, 0.1, 0.3]
        species.append(dict(N=N, params=prm, init_pops=ip, caps=2 * ip, mmm=mmm))
    unc = np.array([[1, 1, 0.1, 0.2, 0, 0], [1, 1, 0.2, 0.35, 0.1, 0.2], [1, 1, 0.3, 0.5, 0, 0]],
                   np.float32)
    osd = 0.05
    if kind == "equal profits":
        unc[:, [2, 4]] = 0.0
        osd = 0.0
    return dict(n_paths=P, n_years=Y, dim_res=R, dt=1.0, rrr=7.0, unit_cost=0.5, unit_revenue=1.2,
                seed=5, road=3, sem=sem, algo=algo, species=species,
                flows=np.array([0, 50, 100], np.float32), uncert=unc.reshape(-1),
                fuel_costs=np.array([0.3], np.float32), fuel_idx=np.array([0], np.int32),
                ore_content=np.array([0.8], np.float32), ore_sd=np.array([osd], np.float32),
                demand_idx=2 if sem == 1 else -1)


@pytest.mark.parametrize("S,R,P,Y,sem,algo,N,surf,kind", CASES)
def test_regressions_equal_oracle(ctx, S, R, P, Y, sem, algo, N, surf, kind):
    pr = _problem(S, R, P, Y, sem, algo, N, kind)
    want = ("cond_exp", "opt_cont", "unit_profits", "adj_pops") + (("regression",) if surf else ())
    g = sg.simulateROVCUDA(pr, want=want, ctx=ctx)
    o = po.simulate_rov(pr, threads=8)

    def same(a, b):
        np.testing.assert_array_equal(np.asarray(a, np.float32), np.asarray(b, np.float32))
    same(g["opt_cont"], o["opt_cont"])
    same(g["cond_exp"], o["cond_exp"])
    same(g["unit_profits"][P:], o["unit_profits"][P:])
    same(np.reshape(g["adj_pops"], (Y, S, P))[1:], np.reshape(o["adj_pops"], (Y, S, P))[1:])
    if surf:
        same(g["regression"], o["regression"])


def test_year_zero_is_zero(ctx):
    """No kernel writes year 0 of the profits and populations; the call returns
    zeros there whatever an earlier one left in the scratch, also where one
    road of a batch asks for them and the others do not."""
    big = _problem(2, 8, 9000, 12, 1, 4, 40, "")
    sg.simulateROVCUDA(big, ctx=ctx)
    for sem, S in ((0, 1), (1, 2)):
        g = sg.simulateROVCUDA(_problem(S, 6, 500, 5, sem, 4, 9, ""), ctx=ctx)
        assert np.all(g["unit_profits"][:500] == 0.0) and np.all(g["adj_pops"][:S * 500] == 0.0)
        assert np.all(g["adj_pops"][S * 500:] > 0.0)
        sg.simulateROVCUDA(big, ctx=ctx)
    prs, keep = zip(*[sg.rov_ctypes(dict(_problem(2, 6, 500, 5, 1, 4, 9, ""), road=r)) for r in range(3)])
    pops, prof = np.full(5 * 2 * 500, -7.0), np.full(5 * 500, -7.0)
    res = (_capi.RovResult * 3)()
    res[1].adj_pops = _capi.ptr(pops, ctypes.c_double)
    res[2].unit_profits = _capi.ptr(prof, ctypes.c_double)
    assert ctx.lib.to_simulate_rov_batch(ctx.handle, 3, (_capi.RovProblem * 3)(*prs), res) == 0
    assert np.all(pops[:1000] == 0.0) and np.all(pops[1000:] > 0.0)
    assert np.all(prof[:500] == 0.0) and not np.any(prof[500:] == -7.0)
    one = sg.simulateROVCUDA(dict(_problem(2, 6, 500, 5, 1, 4, 9, ""), road=1), ctx=ctx)
    np.testing.assert_array_equal(pops, one["adj_pops"])


@pytest.mark.parametrize("S,R,P,Y,sem,algo,N,surf,kind", [
    (1, 120, 400, 4, 0, 4, 12, True, ""), (4, 11, 300, 3, 1, 4, 6, False, "")])
def test_many_tiles_equal_oracle(ctx, S, R, P, Y, sem, algo, N, surf, kind):
    """More than two tiles an SM for the fewest and the most dimensions."""
    test_regressions_equal_oracle(ctx, S, R, P, Y, sem, algo, N, surf, kind)
