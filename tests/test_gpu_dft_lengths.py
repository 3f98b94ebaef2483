"""One step on stretched grids at the longest y transforms, against the oracle.

The column transforms run 4, 2 and 1 columns per block (up to 1024, 2048 and
from 4096 points), the x solves 1, 2 and 8 lines per warp; the x sizes leave
the last tile of columns partly filled.  Tolerance as for every grid shape:
1e-12 of each field's range, p and psi modulo their mean.
"""
import numpy as np
import pytest

from oracle import Oracle
from simplevofsolver_b200 import DROPLET2D_ENV, Solver, droplet2d, physical_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(41, 16), (9, 512), (11, 1024), (7, 2048), (37, 4096), (6, 8192)])
def test_dft_length(gpu_available, nx, ny):
    ic = droplet2d(nx, ny, uniform=False, noise=1e-3)
    phys = physical_params(DROPLET2D_ENV)
    kw = dict(add_buoyancy=True, t_walls=(0.5, -0.5))
    g, o = Solver(ic, phys, **kw), Oracle(ic, phys, **kw)
    assert g.integrate() == o.run(1)[0]
    for k in ("ux", "uy", "p", "psi", "t", "vof"):
        a, b = g.field(k), o.field(k)
        if k in ("p", "psi"):  # the halo rows' wall cells keep the previous call's values
            a, b = ((v - v[1:-1, 1:-1].mean())[1:-1, 1:-1] for v in (a, b))
        r = float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))
        assert r <= 1e-12, (k, r)
    g.close()
