"""The single-road species model's N x N outputs against the oracle where its
route or layout changes: types labelled a CTA each, blocks too many for that
(one CTA, type by type), capacities that are no multiple of four."""
import numpy as np
import pytest

from oracle import pyoracle as po
from transportoptimiser_gb300 import simulate_gpu as sg
from transportoptimiser_gb300 import synth

pytestmark = pytest.mark.gpu
TYPES = [synth.PRIMARY, synth.MARGINAL, synth.OTHER, 5, synth.CLEAR]


@pytest.mark.parametrize("side,tile,res,habitable,cap,sem", [
    (64, 8, 6, 64, 701, 1), (96, 12, 8, 96, 1024, 0), (100, 4, 90, 18, 1022, 1), (33, 33, 4, 33, 64, 0)])
def test_species_model_dense_outputs(ctx, side, tile, res, habitable, cap, sem):
    rng = np.random.default_rng(side)
    base = synth.habitat_map(side, side, tile, [0.35, 0.25, 0.15, 0.15, 0.1], TYPES, rng)
    grid = np.asarray(base).reshape(side, side).copy()
    grid[habitable:] = synth.CLEAR
    grid[:, habitable:] = synth.CLEAR
    sp = synth.default_species(3, np.array([0.0, 0.5, 1.0]), TYPES[:4], threshold=0.0)
    road = synth.random_road(side, side, 12, rng)
    sc = synth.Scene(W=side, H=side, res=res, base_map=grid.reshape(-1), species=[sp], n_controls=3,
                     flows=np.array([0.0, 0.5, 1.0]), seed=1)
    hab = sc.hab_map(road)
    ref = po.species_model(sc, sp, road, sem=sem, max_patches=2048, hab=hab)
    got = sg.createSpeciesModel(hab, sc.pop_map(sp, hab), side, side, res, sp.habitats, road.colmajor(),
                                road.G, sp.hazard, sp.lambda_mean, sem=sem, max_patches=cap, ctx=ctx)
    assert got["N"] == ref["N"] > 0 and got["n_transitions"] == ref["n_transitions"]
    for k in ("area", "cap", "pop", "cx", "cy", "type", "crossings"):
        assert np.array_equal(got[k], ref[k]), k
    # FP64 exp differs from the host's in the last bits
    for k in ("trans", "surv"):
        np.testing.assert_allclose(got[k], ref[k], rtol=1e-12, atol=0)
    np.testing.assert_allclose(got["mmm"], ref["mmm"], rtol=1e-6, atol=1.1e-5)


def test_species_model_holds_its_own_patches_only(ctx):
    """The outputs own their memory: nothing of max_patches' size stays alive."""
    sc = synth.mte_road(0)
    sp, road = sc.species[0], sc.roads[0]
    hab = sc.hab_map(road)
    m = sg.createSpeciesModel(hab, sc.pop_map(sp, hab), sc.W, sc.H, sc.res, sp.habitats, road.colmajor(),
                              road.G, sp.hazard, sp.lambda_mean, sem=1, max_patches=2000, ctx=ctx)
    N, C = m["N"], len(sp.hazard)
    for k, shape in (("crossings", (N, N)), ("trans", (N, N)), ("surv", (C, N, N)), ("mmm", (C, N, N))):
        assert m[k].base is None and m[k].flags.owndata and m[k].shape == shape, k
