"""The exogenous processes at the edges of their tiles (16 years, four
processes, 32 paths) and with jumps in some of them, and the first period with
a control nobody takes: the valuation against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import pyoracle as po
from transportoptimiser_gb300 import simulate_gpu as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths,years,procs,sem", [(131, 17, 3, 1), (160, 16, 4, 1), (97, 33, 6, 1),
                                                   (2, 4, 3, 1), (200, 15, 5, 0)])
def test_exogenous_processes(ctx, paths, years, procs, sem):
    rng = np.random.default_rng(paths)
    n = 9
    m = rng.random((n, n)) * (rng.random((n, n)) < 0.5) + np.eye(n)
    m /= m.sum(0, keepdims=True)
    mmm = np.stack([m * np.exp(-0.2 * c) for c in range(3)]).astype(np.float32)
    ip = rng.integers(100, 2500, n).astype(np.float32)
    sp = dict(N=n, params=np.array([0.05, 0.05, 0.05, 0.0, 0.5, 0.0, 0.0, 0.4], np.float32),
              init_pops=ip, caps=2 * ip, mmm=mmm)
    unc = np.array([[1 + 0.1 * u, 1, 0.1 + 0.05 * u, 0.2, 0.3 if u % 2 else 0.0, 0.25 if u % 2 else 0.0]
                    for u in range(procs)], np.float32)
    pr = dict(n_paths=paths, n_years=years, dim_res=5, dt=1.0, rrr=7.0, unit_cost=0.5, unit_revenue=1.2,
              seed=8, road=2, sem=sem, algo=4, species=[sp], flows=np.array([0, 50, 100], np.float32),
              uncert=unc.reshape(-1), fuel_costs=np.array([0.3, 0.2], np.float32),
              fuel_idx=np.array([0, 1], np.int32), ore_content=np.array([0.8], np.float32),
              ore_sd=np.array([0.05], np.float32), demand_idx=procs - 1 if sem == 1 else -1)
    g = sg.simulateROVCUDA(pr, want=("cond_exp", "opt_cont", "unit_profits"), ctx=ctx)
    o = po.simulate_rov(pr, threads=8)
    for k in ("unit_profits", "cond_exp", "opt_cont"):
        a, b = np.asarray(g[k], np.float32), np.asarray(o[k], np.float32)
        s = paths if k == "unit_profits" else 0
        np.testing.assert_array_equal(a[s:], b[s:], err_msg=k)
    np.testing.assert_allclose(g["stats"], o["stats"], rtol=1e-9)
