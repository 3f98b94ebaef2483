"""One step on grids whose kernels take each of their launch shapes.

The right-hand side, geometry and vof advection kernels choose the planes a
block walks from the grid (march_planes_even / march_planes_uneven); these
grids lead the advection to blocks of 1, 2, 4 and 8 planes, with x sizes that
leave the last tile ragged, and the Poisson x solves (cline_solve.cuh) to
blocks of 1, 2, 4 and 8 lines, with the last block and the last chunk of rows
partly filled.  Compared with the oracle within 1e-12 of each
field's range (p and psi modulo their mean), as every grid shape is.
"""
import numpy as np
import pytest

from oracle import Oracle3D
from simplevofsolver_b200 import DROPLETS3D_ENV, Solver3D, droplets3d, physical_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(33, 16, 8), (8, 8, 4), (64, 64, 64), (61, 64, 128), (200, 64, 128),
                                      (50, 128, 256), (70, 128, 512)])
def test_depth(gpu_available, nx, ny, nz):
    ic = droplets3d(nx, ny, nz, ndrops=4 if nx > 8 else 0, radii=(0.1, 0.15), seed=nz)
    phys = physical_params(DROPLETS3D_ENV)
    g, o = Solver3D(ic, phys), Oracle3D(ic, phys)
    assert g.integrate() == o.run(1)[0]
    for k in ("ux", "uy", "uz", "p", "psi", "t", "vof"):
        a, b = g.field(k), o.field(k)
        if k in ("p", "psi"):
            a, b = ((v - v[1:-1, 1:-1, 1:-1].mean())[..., 1:-1] for v in (a, b))
        r = float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))
        assert r <= 1e-12, (k, r)
    g.close()
