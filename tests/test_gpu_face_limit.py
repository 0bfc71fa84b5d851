"""Fused face transforms at the limit of their dispatch rule, against the C
oracle in FP64: the largest faces, faces whose longest side is the one that the
slabs run along, and a context of unlike partitions whose largest regions of
shared memory come from different faces.

Tolerances as for the modal update, whose roundings are of the same number: a
step adds about ten units in the last place of the field's size with random
signs, 40 * 10 * 2^-24 = 2.4e-5 for T = 40 in FP32; in FP64 the field readout
is float32: 1e-6.
"""
import numpy as np
import pytest

import ard_gb300 as A
from oracle import oracle as O

pytestmark = pytest.mark.gpu

T = 40


@pytest.mark.parametrize("precision,air", [
    (A.PREC_F32, [(0, 0, 0, 136, 136, 12)]),
    (A.PREC_F32, [(0, 0, 0, 40, 137, 40)]),
    (A.PREC_F32, [(0, 0, 0, 14, 140, 12)]),
    (A.PREC_F32, [(0, 0, 0, 132, 132, 20), (132, 0, 0, 300, 12, 20)]),
    (A.PREC_F64, [(0, 0, 0, 88, 88, 12)]),
    (A.PREC_F64, [(0, 0, 0, 38, 90, 40)]),
    (A.PREC_F64, [(0, 0, 0, 12, 95, 12)]),
])
def test_fused_faces_at_their_limit(precision, air):
    dh, c0 = 0.1, 343.0
    dt = float(np.float32(0.5 * dh / (c0 * np.sqrt(3.0))))
    rng = np.random.default_rng(air[0][4])
    flat = O.make_flat_scene(air, [], [], dict(dh=dh, dt=dt, c0=c0, pml_layers=5))
    flat["sources"] = [(b[0] + b[3] // 2, b[1] + b[4] // 3, b[2] + b[5] // 2, i) for i, b in enumerate(air)]
    series = (1e6 * rng.standard_normal((len(air), T))).astype(np.float32)
    sim = A.Simulation(A.scene_from_flat(flat), precision=precision, max_steps=T)
    assert "faces fused" in sim.layout
    ref = O.OracleSim(flat, "f64")
    for i, s in enumerate(series):
        sim.set_source_series(i, s)
        ref.set_source_series(i, s)
    sim.run(T)
    ref.step(T)
    tol = 2.4e-5 if precision == A.PREC_F32 else 1e-6
    for i in range(len(air)):
        want = ref.field(i)[0]
        assert np.sqrt(np.mean((sim.field(i) - want) ** 2)) < tol * np.sqrt(np.mean(want ** 2))
