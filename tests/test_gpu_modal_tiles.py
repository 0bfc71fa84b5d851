"""Modal update at the edges of its tiles (32 kx x 32 ky x the planes of one kz
parity) against the C oracle in FP64: extents below, at and just above a tile,
an odd depth (the odd parity one plane short), the smallest partition, and up
to eight sources and recorders in one partition.

Tolerances, from the arithmetic: every step adds a few roundings per mode
(the expansion's nine products, the recurrence's five operations) to values
of the field's own size, about 10 units in the last place of the working
precision over T = 40 steps with random signs and no growth (the recurrence's
gain is below one): 40 * 10 * 2^-24 = 2.4e-5 in FP32; in FP64 the oracle's own
transforms round as well: 1e-11.
"""
import numpy as np
import pytest

import ard_gb300 as A
from helpers import rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu

T = 40


@pytest.mark.parametrize("extent,points", [((6, 6, 6), 1), ((31, 33, 7), 3), ((32, 32, 32), 2), ((33, 64, 9), 8),
                                           ((65, 30, 50), 5), ((100, 7, 13), 4)])
@pytest.mark.parametrize("precision", [A.PREC_F32, A.PREC_F64])
def test_modal_tile_edges(extent, points, precision):
    dh, c0 = 0.1, 343.0
    dt = float(np.float32(0.5 * dh / (c0 * np.sqrt(3.0))))
    rng = np.random.default_rng(sum(extent) + points)
    flat = O.make_flat_scene([(0, 0, 0) + extent], [], [], dict(dh=dh, dt=dt, c0=c0, pml_layers=5))
    cells = set()
    while len(cells) < 2 * points:
        cells.add(tuple(int(rng.integers(0, n)) for n in extent))
    cells = sorted(cells)
    rng.shuffle(cells)
    flat["sources"] = [tuple(int(v) for v in c) + (0,) for c in cells[:points]]
    flat["recorders"] = [tuple(int(v) for v in c) + (0,) for c in cells[points:]]
    series = (1e6 * rng.standard_normal((points, T))).astype(np.float32)
    sim = A.Simulation(A.scene_from_flat(flat), precision=precision, max_steps=T)
    ref = O.OracleSim(flat, "f64")
    for i in range(points):
        sim.set_source_series(i, series[i])
        ref.set_source_series(i, series[i])
    sim.run(T)
    ref.step(T)
    tol = 2.4e-5 if precision == A.PREC_F32 else 1e-11
    field = ref.field(0)[0]
    # rounding is set by the field's size, which a recorder far from the sources does not reach
    off = sim.recorders(f64=True) - ref.recorders()
    assert np.sqrt(np.mean(off ** 2)) < tol * np.sqrt(np.mean(field ** 2))
    # the field readout is float32
    assert rel_l2(sim.field(0), field) < max(tol, 1e-6)
