"""A generation whose migration matrices are not sparse: the migration kernel
is then chosen by a trial on the dense form, and the results are those of each
kernel asked for.  One range keeps a packed form, the other outgrows it."""
import numpy as np
import pytest

from transportoptimiser_gb300 import synth
from transportoptimiser_gb300._capi import MIG_AUTO, MIG_SIMT_FP32
from transportoptimiser_gb300.generation import Generation, pack_roads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lam,trial", [(0.2, False), (0.075, True), (0.02, True)])
def test_auto_on_dense_matrices(ctx, lam, trial):
    sc = synth.generation(11, n_roads=2)
    for sp in sc.species:
        sp.lambda_mean = lam
    gen = Generation(sc, max_roads=2, max_patches=512, ctx=ctx)
    packed = pack_roads(sc, sc.roads)
    paths = 40 + int(1000 * lam)                # a shape of its own in the record
    auto = gen.evaluate(packed, gen.opts(paths, 5, seed=4, sem=1, migration=MIG_AUTO))
    line = [l for l in ctx.tuning().splitlines() if f"paths={paths} " in l][-1]
    assert ("simt -1.000" not in line) == trial, line
    ref = gen.evaluate(packed, gen.opts(paths, 5, seed=4, sem=1, migration=MIG_SIMT_FP32))
    # end populations: FP32 sums in one order on both kernels (3xTF32: 1e-5)
    np.testing.assert_allclose(auto[:, :, 2:7], ref[:, :, 2:7], rtol=1e-4, atol=1e-6)
    gen.close()


@pytest.mark.parametrize("lam", [0.075, 0.02])
def test_tuned_shape_builds_its_models_once(ctx, lam):
    """After the trial a generation's species models are built in one pass,
    whichever kernel the record names, with the results of the first."""
    sc = synth.generation(11, n_roads=2)
    for sp in sc.species:
        sp.lambda_mean = lam
    gen = Generation(sc, max_roads=2, max_patches=512, ctx=ctx)
    packed = pack_roads(sc, sc.roads)
    opts = gen.opts(48 + int(1000 * lam), 5, seed=4, sem=1, migration=MIG_AUTO)
    first = gen.evaluate(packed, opts)
    for _ in range(2):
        ctx.profile(True)
        n0 = ctx.kernel_time("species_links")[1]
        again = gen.evaluate(packed, opts)
        n1 = ctx.kernel_time("species_links")[1]
        ctx.profile(False)
        assert n1 - n0 == 1
        assert np.array_equal(again, first, equal_nan=True)      # no ROV, no penalty: NaN
    gen.close()
