"""Rounding of the fused face transforms where it is amplified: the fifth of the
random scenes grows (the scheme is unstable at its interfaces), so that the noise
that a transform puts into quiet cells in the first hundred steps stands beside
the signal later.  FP32 against FP64 contexts, geometric mean over the recorders
and over amplitudes of the source, which round differently.

Bound, from 32 amplitudes with a spread of 1.3 for one: full-length products
give 1.6e-5 over 1000 steps; half-length products added from the low modes up,
whose sums leave the rounding of loud cells in their mirror cells, 3.4e-5.  The
bound is the geometric middle, 2.3e-5, which the mean of eight (spread 1.1) does
not cross from either side.
"""
import numpy as np
import pytest

import ard_gb300 as A
from ard_gb300 import configs

pytestmark = pytest.mark.gpu

T = 1000


def test_rounding_does_not_leak_into_quiet_cells():
    cfg = configs.config("c2", steps=T)
    sc = cfg["scenes"][4]
    scene = A.build_scene(sc["air"], sc["sources"], sc["recorders"], float(np.float32(cfg["h"])), cfg["dt"], cfg["c0"],
                          cfg["pml"])
    sims = [A.Simulation([scene], max_steps=T, precision=p) for p in (A.PREC_F32, A.PREC_F64)]
    assert all("faces fused" in s.layout for s in sims)
    errors = []
    for k in range(8):
        rec = []
        for s in sims:
            s.reset()
            for j, series in enumerate(sc["series"]):
                s.set_source_series(j, np.asarray(series[:T], np.float32) * np.float32(1 + 0.03137 * k))
            s.run(T)
            rec.append(s.recorders(f64=True))
        errors += list(np.linalg.norm(rec[0] - rec[1], axis=0) / np.linalg.norm(rec[1], axis=0))
    assert np.exp(np.mean(np.log(errors))) < 2.3e-5
