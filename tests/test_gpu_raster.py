"""Device road rasterisation on the spans whose arithmetic has special cases
(vertical and horizontal spans, endpoints on grid lines and corners, spans
towards smaller x, zero-length and long spans, points outside the grid),
where the crossing lists come out of order or tie, against the host cells."""
import numpy as np
import pytest

from transportoptimiser_gb300 import synth
from transportoptimiser_gb300.generation import Generation, pack_roads, pack_segments

pytestmark = pytest.mark.gpu

SPECIAL = [
    [(3.5, 4.5), (3.5, 180.2)], [(7.5, 180.2), (7.5, 4.5)], [(2.2, 7.0), (190.9, 7.0)],
    [(190.9, 33.3), (2.2, 33.3)], [(5.0, 5.0), (9.0, 13.0), (9.0, 13.0), (60.0, 60.0)],
    [(199.0, 199.0), (0.0, 0.0)], [(0.0, 0.0), (199.0, 199.0)], [(38.5, 1.5), (1.5, 38.5)],
    [(100.0, 50.0), (100.0 + 1e-12, 150.0)], [(100.0 + 1e-12, 150.0), (100.0, 20.0)],
    [(-30.3, 40.7), (260.1, 90.2)], [(20.0, -50.0), (21.0, 240.0)], [(12.0, 12.0), (12.0, 12.0)],
]


@pytest.mark.parametrize("sem", [0, 1])
@pytest.mark.parametrize("n", [1, 5, 70])
def test_special_spans_equal_host_cells(ctx, sem, n):
    sc = synth.generation(9, n_roads=0)
    rng = np.random.default_rng(n)
    roads = []
    for i in range(n):
        pts = np.array(SPECIAL[(i + n) % len(SPECIAL)], np.float64)
        segs = np.column_stack([pts[:-1], pts[1:]])
        roads.append(synth.Road(points=pts, segments=segs))
        if i % 3 == 2:
            roads[-1] = synth.random_road(sc.W, sc.H, int(rng.integers(2, 65)), rng)
    gen = Generation(sc, max_roads=n, max_patches=512, ctx=ctx)
    opts = gen.opts(32, 3, seed=3, sem=sem, migration=3)
    a = gen.evaluate(pack_roads(sc, roads, sem=sem), opts)
    b = gen.evaluate_segments(pack_segments(roads), opts)
    np.testing.assert_array_equal(a, b)
    f = gen.features(pack_segments(roads))          # cells of corrected semantics
    cells = [len(synth.road_cells(rd, sc.W, sc.H, sem=1)) for rd in roads]
    np.testing.assert_allclose(f[:, 2] * sc.W, cells, rtol=1e-6)
    gen.close()
