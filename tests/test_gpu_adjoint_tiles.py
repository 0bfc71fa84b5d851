"""The adjoint's modal update at the edges of its tiles (32 kx x 32 ky x the
planes of one kz parity) against the FP64 autograd tape: extents just below and
above a tile, an odd depth (the odd parity one plane short), and up to eight
sources and recorders, whose injection and read-out change places.  The rows are
padded (no extent along x is a multiple of four), where the reference's arithmetic
divides by the squared frequency.

Tolerances: the library returns float gradients, so in FP64 their rounding
(2^-24 of each value; 1e-7 for the series, 1e-6 for the pressure that a dense
transform maps back).  In FP32 a forward and a backward run of T = 24 steps each
round a value about ten times a step with random signs, and the forward's error
enters the residuals: 2 * 24 * 10 * 2^-24 = 2.9e-5 of the gradient's size.
"""
import numpy as np
import pytest

import ard_gb300 as A
from oracle import oracle as O
from oracle.tape_oracle import TapeOracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T = 24


def rel(a, b):
    a = np.asarray(a, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("extent,points", [((33, 34, 9), 8), ((31, 8, 7), 3), ((65, 33, 11), 5)])
def test_adjoint_modal_tile_edges(extent, points):
    dh, c0 = 0.1, 343.0
    dt = float(np.float32(0.5 * dh / (c0 * np.sqrt(3.0))))
    rng = np.random.default_rng(sum(extent))
    flat = O.make_flat_scene([(0, 0, 0) + extent], [], [], dict(dh=dh, dt=dt, c0=c0, pml_layers=5))
    cells = set()
    while len(cells) < 2 * points:   # off the shell, which the interfaces force
        cells.add(tuple(int(rng.integers(3, n - 3)) for n in extent))
    cells = sorted(cells)
    rng.shuffle(cells)
    flat["sources"] = [tuple(int(v) for v in c) + (0,) for c in cells[:points]]
    flat["recorders"] = [tuple(int(v) for v in c) + (0,) for c in cells[points:]]
    series = rng.standard_normal((points, T)).astype(np.float32)
    p0 = rng.standard_normal(extent[::-1]).astype(np.float32)
    s_t = torch.tensor(series, dtype=torch.float64, requires_grad=True)
    p_t = torch.tensor(p0, dtype=torch.float64, requires_grad=True)
    rec = TapeOracle(flat).run(s_t, T, p0={0: p_t})
    target = (0.5 * rec.detach().numpy()[::-1]).astype(np.float32)
    (0.5 * ((rec - torch.tensor(target, dtype=torch.float64)) ** 2).sum()).backward()
    for precision, arithmetic, tol_s, tol_p in ((A.PREC_F64, A.ARITH_ACCURATE, 1e-7, 1e-6),
                                                (A.PREC_F64, A.ARITH_REFERENCE, 1e-7, 1e-6),
                                                (A.PREC_F32, A.ARITH_ACCURATE, 2.9e-5, 2.9e-5)):
        sim = A.Simulation(A.scene_from_flat(flat), precision=precision, arithmetic=arithmetic, max_steps=T, adjoint=True)
        for i, s in enumerate(series):
            sim.set_source_series(i, s)
        sim.set_initial_pressure(0, p0)
        g = sim.adjoint(T, target)
        assert rel(g["grad_source"], s_t.grad.numpy()) < tol_s
        assert rel(sim.initial_pressure_grad(0), p_t.grad.numpy()) < tol_p
