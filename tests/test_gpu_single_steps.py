"""Single steps by one-step graphs against direct launches of the same kernels:
the same results bit for bit, from either parity, across the hand-over from
the first directly launched steps, mixed with longer runs, with the recorders'
neighbourhoods switched on in between, and again after a reset."""
import numpy as np
import pytest

import ard_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [A.PREC_F32, A.PREC_F64])
@pytest.mark.parametrize("runs", [[1] * 11, [3, 1, 33, 2, 1, 40], [37, 1, 1]])
def test_single_step_graphs_match_direct_launches(precision, runs):
    dh, c0 = 0.1, 343.0
    dt = float(np.float32(0.5 * dh / (c0 * np.sqrt(3.0))))
    scene = A.build_scene([(0, 0, 0, 20, 20, 16), (20, 4, 0, 14, 13, 16)], [(6, 7, 8)], [(12, 10, 8), (27, 11, 9)],
                          dh, dt, c0, 5)
    T = sum(runs) + 6
    series = (1e6 * np.random.default_rng(3).standard_normal(T)).astype(np.float32)
    got = []
    for graphs in (True, False):
        sim = A.Simulation(scene, precision=precision, max_steps=T, use_graphs=graphs)
        sim.set_source_series(0, series)
        out = []
        for rep in range(2):
            for n in runs:
                sim.run(n)
            sim.record_neighbourhoods(True)
            for _ in range(6):
                sim.Update()
            out += [sim.recorders(f64=True), sim.neighbourhoods(t0=sum(runs), nt=6)]
            out += [sim.field(p) for p in range(len(scene.partitions))]
            sim.record_neighbourhoods(False)
            sim.reset()
        got.append(out)
    for a, b in zip(*got):
        assert np.array_equal(a, b)
