"""The 2D fused predictor on narrow grids, against the oracle.

Short lines are swept a thread a line, longer ones a warp a line; the line
between the two depends on the rows of a block as well.  Sizes on both sides,
lines shorter than a warp's segments, and rows that leave the last block partly
filled; small dt, the range of a time step and dt far beyond it.  The predictor
is linear in its inputs at each dt: 1e-12 of each field's range.
"""
import numpy as np
import pytest

from oracle import Oracle
from simplevofsolver_b200 import DROPLET2D_ENV, Solver, droplet2d, physical_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,uniform", [(4, 4, True), (5, 4096, False), (16, 2047, True), (33, 4096, False),
                                           (41, 8, False), (42, 8, False), (48, 16, False), (64, 30, True),
                                           (64, 4097, True), (65, 64, False), (96, 1024, False), (128, 2050, True)])
def test_predictor(gpu_available, nx, ny, uniform):
    ic = droplet2d(nx, ny, uniform=uniform, noise=1e-2, nsub=2)
    phys = physical_params(DROPLET2D_ENV)
    kw = dict(uy_walls=(0.1, -0.1), t_walls=(0.5, -0.5))
    g, o = Solver(ic, phys, **kw), Oracle(ic, phys, **kw)
    for rk, dt in ((0, 1e-6), (1, 1e-3), (0, 50.0)):
        g.fluid_predict_field(rk, dt)
        o.predict(rk, dt)
        for k in ("ux", "uy", "t"):
            a, b = g.field(k), o.field(k)
            assert np.abs(a - b).max() <= 1e-12 * max(np.abs(b).max(), 1e-300), (dt, k)
    g.close()
