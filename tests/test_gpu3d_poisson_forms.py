"""The two forms of the 3D Poisson solve's x lines.

Whole lines on chip (k_cline_solve) and the kernel that streams lines in
chunks (k3_pois_x) evaluate the same expressions a row: their results are the
same bits in both storage types.  A grid takes one of them by its size;
SVOF3_POISSON_LINES forces one at a solver's creation.
"""
import os

import numpy as np
import pytest

from oracle import Oracle3D
from simplevofsolver_b200 import DROPLETS3D_ENV, Solver3D, droplets3d, physical_params

pytestmark = pytest.mark.gpu


def solver(ic, whole, precision):
    os.environ["SVOF3_POISSON_LINES"] = "1" if whole else "0"
    try:
        return Solver3D(ic, physical_params(DROPLETS3D_ENV), precision=precision)
    finally:
        del os.environ["SVOF3_POISSON_LINES"]


# divergent velocities: x lines of one ky, kz each, 64 lines a streaming block
# up to 75775 lines and 128 from there on
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_dc"])
@pytest.mark.parametrize("nx,ny,nz", [(4, 8, 4), (61, 64, 32), (33, 16, 128), (97, 64, 64), (1001, 8, 4),
                                      (17, 256, 1024)])
def test_poisson_forms_agree(gpu_available, nx, ny, nz, precision):
    ic = droplets3d(nx, ny, nz, ndrops=0, urms=0.0, seed=1)
    rng = np.random.default_rng(nx)
    for k in ("ux", "uy", "uz"):
        getattr(ic, k)[..., 1:-1] = rng.uniform(-1.0, 1.0, getattr(ic, k)[..., 1:-1].shape)
    out = []
    for whole in (False, True):
        g = solver(ic, whole, precision)
        g.fluid_compute_potential_dft(1, 1e-2)
        out.append((g.field("psi"), g.health()["small_pivots"]))
        g.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
    assert np.abs(out[0][0]).max() > 0.0
    if "fp64" == precision and nx * ny * nz < 1 << 20:
        o = Oracle3D(ic, physical_params(DROPLETS3D_ENV))
        o.potential(1, 1e-2)
        a, b = ((v - v[1:-1, 1:-1, 1:-1].mean())[..., 1:-1] for v in (out[0][0], o.field("psi")))
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
