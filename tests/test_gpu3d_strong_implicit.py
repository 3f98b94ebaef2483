"""3D grids of many x lines, from weak to strong implicit x.

There the table kernel judges each substep whether its lines go to k3_xlines or
to k3_xsolve (segments that have to be run again too often).  Whichever it
takes, the fields are the bits that either kernel forced for all substeps
(SVOF3_PREDICT_LINES) gives: single predictors at time steps on both sides of
the line, whole steps (graphs) and fixed steps.
"""
import os

import numpy as np
import pytest

from simplevofsolver_b200 import Solver3D, droplets3d, physical_params

pytestmark = pytest.mark.gpu

FIELDS = ("ux", "uy", "uz", "t", "p", "vof")


def solvers(ic, phys, precision):
    out = []
    for force in (None, "0", "1"):
        if force:
            os.environ["SVOF3_PREDICT_LINES"] = force
        try:
            out.append(Solver3D(ic, phys, uy_walls=(0.1, -0.1), t_walls=(0.5, -0.5), precision=precision))
        finally:
            os.environ.pop("SVOF3_PREDICT_LINES", None)
    return out


def same(ss, names=FIELDS):
    for k in names:
        a = [s.field(k) for s in ss]
        assert np.array_equal(a[0], a[1]) and np.array_equal(a[0], a[2]), k


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nz,re,stretch", [(64, 128, 128, 20, 3.5), (161, 64, 128, 20, 3.5), (321, 128, 64, 20, 3.5),
                                                 (200, 128, 128, 20, 2.0), (100, 128, 128, 500, 1.5)])
def test_any_form_gives_the_same_bits(gpu_available, nx, ny, nz, re, stretch, precision):
    ic = droplets3d(nx, ny, nz, ndrops=2, radii=(0.1, 0.15), stretch=stretch, seed=2, nsub=2)
    phys = physical_params({"Ra": float(re) ** 2, "Pr": 1.0, "We": 20.0, "coef_dt_adv": 0.5, "coef_dt_dif": 0.95})
    ss = solvers(ic, phys, precision)
    for dt in (1e-7, 1e-5, 1e-4, 1e-2, 1.0):
        for rk in range(3):
            for s in ss:
                s.fluid_predict_field(rk, dt)
        same(ss, ("ux", "uy", "uz", "t"))
    for s in ss:
        s.close()
    ss = solvers(ic, phys, precision)
    dts = [s.run(2) for s in ss]
    assert np.array_equal(dts[0], dts[1]) and np.array_equal(dts[0], dts[2])
    same(ss)
    for s in ss:
        s.integrate_fixed(0.5 * float(dts[0][-1]))
    same(ss)
    for s in ss:
        s.close()
