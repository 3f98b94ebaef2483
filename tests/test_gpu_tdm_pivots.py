"""The predictor's Thomas pivots and sweeps, computed by segments, against the
oracle.  In 3D a line has 8 lanes, 16 from 321 cells, and beyond 1150 cells a
kernel of its own.

A segment starts from a guess some rows ahead; where the guess has not met the
true recurrence the rows are run again.  Small dt (the two meet at once), the
range of a time step and dt far beyond it (they meet late or not at all), on
lines shorter than a warp's segments, of odd length and long.  The predictor
is linear in its inputs at each dt, so the parity tolerance of the entry
points holds: 1e-12 of each field's range.
"""
import numpy as np
import pytest

from oracle import Oracle, Oracle3D
from simplevofsolver_b200 import (DROPLET2D_ENV, DROPLETS3D_ENV, Solver, Solver3D, droplet2d, droplets3d,
                                  physical_params)

pytestmark = pytest.mark.gpu


def close(g, o, names):
    for k in names:
        a, b = g.field(k), o.field(k)
        assert np.abs(a - b).max() <= 1e-12 * max(np.abs(b).max(), 1e-300), k


@pytest.mark.parametrize("dt", [1e-6, 1e-2, 50.0])
@pytest.mark.parametrize("nx,ny,uniform", [(4, 8, True), (5, 8, False), (37, 16, False), (1024, 8, True), (1501, 8, False)])
def test_predictor_2d(gpu_available, nx, ny, uniform, dt):
    ic = droplet2d(nx, ny, uniform=uniform, noise=1e-2)
    phys = physical_params(DROPLET2D_ENV)
    kw = dict(t_walls=(0.5, -0.5))
    g, o = Solver(ic, phys, **kw), Oracle(ic, phys, **kw)
    g.fluid_predict_field(0, dt)
    o.predict(0, dt)
    close(g, o, ("ux", "uy", "t"))
    g.close()


@pytest.mark.parametrize("dt", [1e-6, 1e-2, 50.0])
@pytest.mark.parametrize("nx,uniform", [(4, True), (61, False), (600, False), (1300, False)])
def test_predictor_3d(gpu_available, nx, uniform, dt):
    ic = droplets3d(nx, 8, 8, uniform=uniform, ndrops=0, seed=2)
    phys = physical_params(DROPLETS3D_ENV)
    g, o = Solver3D(ic, phys), Oracle3D(ic, phys)
    g.fluid_predict_field(0, dt)
    o.predict(0, dt)
    close(g, o, ("ux", "uy", "uz", "t"))
    g.close()


@pytest.mark.parametrize("nx,ny,nz", [(65, 256, 512), (320, 128, 128), (321, 16, 1024), (1001, 4, 2048),
                                      (1300, 64, 64)])
def test_predictor_3d_large(gpu_available, nx, ny, nz):
    ic = droplets3d(nx, ny, nz, ndrops=0, seed=3)
    phys = physical_params(DROPLETS3D_ENV)
    kw = dict(uy_walls=(0.1, -0.1), t_walls=(0.5, -0.5))
    g, o = Solver3D(ic, phys, **kw), Oracle3D(ic, phys, **kw)
    for dt in (1e-3, 0.2):
        g.fluid_predict_field(0, dt)
        o.predict(0, dt)
        close(g, o, ("ux", "uy", "uz", "t"))
    g.close()
