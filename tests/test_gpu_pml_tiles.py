"""PML update in each of its plane tiles (32 x 16, 16 x 32 and 8 x 64 cells,
chosen per slab by the fewest tiles) with ragged last tiles, against the C
oracle in FP64.  The slabs of the first room (7 x 30, 61 x 30 and 61 x 7 cells)
take the three shapes, one tile or two of them; those of the second (12 x 17,
130 x 17, 130 x 12) take them with several tiles; the third room is below every
tile.

Tolerances, from the arithmetic: a step rounds each PML value about five times
at its own size, and the leapfrog carries an error of step t on to step T with a
factor of T - t at most: 5 * 2^-24 * sqrt(sum (T - t)^2) = 5 * 2^-24 * T^1.5 / sqrt(3)
= 8e-5 for random signs and T = 60; doubled for the rooms' part in FP32.  In
FP64 the field readout's rounding to float32: 1e-6.
"""
import numpy as np
import pytest

import ard_gb300 as A
from oracle import oracle as O

pytestmark = pytest.mark.gpu

T = 60


@pytest.mark.parametrize("extent", [(61, 7, 30), (130, 12, 17), (9, 6, 7)])
@pytest.mark.parametrize("precision", [A.PREC_F32, A.PREC_F64])
def test_pml_tile_shapes(extent, precision):
    dh, c0 = 0.1, 343.0
    dt = float(np.float32(0.5 * dh / (c0 * np.sqrt(3.0))))
    w, h, d = extent
    flat = O.make_flat_scene([(0, 0, 0) + extent], [], [], dict(dh=dh, dt=dt, c0=c0, pml_layers=5))
    # sources along the room, so that the field reaches every slab in T steps
    flat["sources"] = [(x, h // 2, d // 2, 0) for x in range(min(8, w // 2), w, 20)][:8]
    series = (1e6 * np.random.default_rng(w).standard_normal((len(flat["sources"]), T))).astype(np.float32)
    sim = A.Simulation(A.scene_from_flat(flat), precision=precision, max_steps=T)
    ref = O.OracleSim(flat, "f64")
    for i, s in enumerate(series):
        sim.set_source_series(i, s)
        ref.set_source_series(i, s)
    sim.run(T)
    ref.step(T)
    tol = 1.6e-4 if precision == A.PREC_F32 else 1e-6
    slabs = [i for i, p in enumerate(flat["partitions"]) if p[0] != 0]
    assert len(slabs) == 6
    for i in slabs:
        want = ref.field(i)[0]
        size = np.sqrt(np.mean(want ** 2))
        assert size > 0
        assert np.sqrt(np.mean((sim.field(i) - want) ** 2)) < tol * size, (i, want.shape)
