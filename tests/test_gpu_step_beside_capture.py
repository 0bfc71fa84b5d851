"""Steps of a context while the caller captures a CUDA graph of its own on
another stream, from the capturing thread and from a second one: they run, with
the results of steps taken without a capture, and the caller's graph is whole.
Single steps pass from direct launches to one-step graphs on the way (the fifth
and sixth step of a context), a longer run captures the many-step graph."""
import threading

import numpy as np
import pytest

import ard_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threaded", [False, True])
@pytest.mark.parametrize("runs", [[1] * 8, [2, 37]])
def test_steps_while_another_stream_is_captured(runs, threaded):
    import torch
    dh, c0 = 0.1, 343.0
    dt = float(np.float32(0.5 * dh / (c0 * np.sqrt(3.0))))
    scene = A.build_scene([(0, 0, 0, 20, 20, 16), (20, 4, 0, 14, 13, 16)], [(6, 7, 8)], [(12, 10, 8)], dh, dt, c0, 5)
    T = sum(runs)
    series = (1e6 * np.random.default_rng(5).standard_normal(T)).astype(np.float32)
    sims = [A.Simulation(scene, max_steps=T) for _ in range(2)]
    for s in sims:
        s.set_source_series(0, series)
    x = torch.ones(8, device="cuda")
    torch.cuda.synchronize()
    failed = []

    def steps():
        try:
            for n in runs:
                sims[0].run(n)
        except Exception as e:   # raised below, after the capture has ended
            failed.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = x + 1
        if threaded:
            t = threading.Thread(target=steps)
            t.start()
            t.join()
        else:
            steps()
        y = y + 1
    assert not failed, failed
    graph.replay()
    torch.cuda.synchronize()
    assert bool((y == 3).all())
    for n in runs:
        sims[1].run(n)
    assert np.array_equal(sims[0].recorders(f64=True), sims[1].recorders(f64=True))
