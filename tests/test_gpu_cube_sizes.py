"""The recorders' neighbourhoods against the whole field of the same step (the
dense transform of the same modes, a path of its own), at extents around the
row kernel's chunk of 128 kx, its 32 rows, the 8-term rounds of the ky and kz
sums, row pitches with padding, and the smallest partition a cube fits into.

Tolerance: both sides sum the same modes in the context's precision, the cube
is stored as float.  FP64: one float rounding, 2^-24 = 6e-8 of the value, 1e-7 of
the largest.  FP32: three chained sums of at most 131 terms on either side, a
few roundings of 6e-8 each with random signs on values of the field's size:
sqrt(2 * 3 * 131) * 6e-8 = 1.7e-6 of the field, 1e-5 of the largest with margin."""
import numpy as np
import pytest

import ard_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [A.PREC_F32, A.PREC_F64])
@pytest.mark.parametrize("dims", [(12, 12, 12), (128, 33, 13), (129, 31, 40), (131, 64, 17), (30, 128, 34), (15, 65, 32)])
def test_neighbourhoods_match_the_field(precision, dims):
    w, h, d = dims
    dh, c0 = 0.1, 343.0
    dt = float(np.float32(0.5 * dh / (c0 * np.sqrt(3.0))))
    recs = [(6, 6, 6), (w - 5, h - 5, d - 5), (w // 2, h // 2, d // 2)]
    recs = [tuple(min(max(c, 6), n - 5) for c, n in zip(r, dims)) for r in recs]   # the scene builder's margin
    scene = A.build_scene([(0, 0, 0, w, h, d)], [(w // 3, h // 3, d // 3)], recs, dh, dt, c0, 5)
    T = 24
    sim = A.Simulation(scene, precision=precision, max_steps=T)
    sim.set_source_series(0, (1e6 * np.random.default_rng(5).standard_normal(T)).astype(np.float32))
    sim.record_neighbourhoods(True)
    sim.run(T)
    cubes = sim.neighbourhoods(t0=T - 1, nt=1)[0].reshape(len(recs), 10, 10, 10)
    field = np.asarray(sim.field(0), dtype=np.float64).reshape(d, h, w)
    tol = (1e-5 if precision == A.PREC_F32 else 1e-7) * np.abs(field).max()
    assert tol > 0
    for r in range(len(recs)):
        x, y, z, part = scene.recorders[r]
        q = scene.partitions[part]
        x, y, z = x - q[2], y - q[3], z - q[4]
        want = field[z - 5:z + 5, y - 5:y + 5, x - 5:x + 5]
        assert np.abs(cubes[r] - want).max() <= tol, (dims, r)
