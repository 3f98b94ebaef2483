"""The two forms of the 3D predictor's x lines.

Whole lines on chip, in segments over a warp's lanes (k3_xlines), and the
kernel that streams lines in chunks, a lane a line (k3_xsolve), evaluate the
same expressions a row: their results are the same bits in both storage types,
whatever the coefficients, also where segments have to be run again from the
right-hand side.  SVOF3_PREDICT_LINES forces one at a solver's creation.

The FP32 sweeps of the mixed path are also compared with the oracle.  Their
bound: increments and coefficients rounded to FP32, and an FP32 elimination of
an M-matrix T whose inverse has norm at most 1 (rows 1 + |l| + |u|, -l, -u),
with a backward error of at most 16 roundings a row of T: 2^-24 (2 + 16 ||T||)
times the largest increment, ||T|| <= 1 + 2 pf max|Laplacian diagonal|.
"""
import os

import numpy as np
import pytest

from oracle import Oracle3D
from simplevofsolver_b200 import Solver3D, droplets3d, physical_params

pytestmark = pytest.mark.gpu


def solver(ic, phys, whole, **kw):
    os.environ["SVOF3_PREDICT_LINES"] = "1" if whole else "0"
    try:
        return Solver3D(ic, phys, **kw)
    finally:
        del os.environ["SVOF3_PREDICT_LINES"]


def physical(re):
    return physical_params({"Ra": float(re) ** 2, "Pr": 1.0, "We": 20.0, "coef_dt_adv": 0.5, "coef_dt_dif": 0.95})


# Re 20 and strong clustering: segments that do not meet at the first try
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("re,stretch", [(500, 1.5), (20, 2.5)])
@pytest.mark.parametrize("nx", [4, 61, 320, 321, 600, 1001])
def test_predictor_forms_agree(gpu_available, nx, re, stretch, precision):
    ic, phys = droplets3d(nx, 8, 8, ndrops=0, stretch=stretch, seed=2), physical(re)
    kw = dict(uy_walls=(0.1, -0.1), t_walls=(0.5, -0.5), precision=precision)
    a = solver(ic, phys, False, **kw)
    b = solver(ic, phys, True, **kw)
    for dt in (1e-6, 1e-3, 1e-2, 50.0):
        a.fluid_predict_field(0, dt)
        b.fluid_predict_field(0, dt)
        for k in ("ux", "uy", "uz", "t"):
            assert np.array_equal(a.field(k), b.field(k)), (dt, k)
    a.close()
    b.close()


@pytest.mark.parametrize("dt", [1e-6, 1e-3, 1e-2, 50.0])
@pytest.mark.parametrize("nx", [61, 320, 321, 600, 1001, 2400])
def test_mixed_predictor_vs_oracle(gpu_available, nx, dt):
    ic, phys = droplets3d(nx, 8, 8, ndrops=0, seed=2), physical(500)
    kw = dict(uy_walls=(0.1, -0.1), t_walls=(0.5, -0.5))
    g, o = Solver3D(ic, phys, precision="mixed", **kw), Oracle3D(ic, phys, **kw)
    names = ("ux", "uy", "uz", "t")
    before = {k: o.field(k).copy() for k in names}
    g.fluid_predict_field(0, dt)
    o.predict(0, dt)
    lap = 4.0 / np.diff(ic.xf).min() ** 2  # at least the largest diagonal
    norm = 1.0 + 2.0 * 0.5 * (8.0 / 15.0) * dt * max(phys["m_dif"], phys["t_dif"]) * lap
    for k in names:
        b = o.field(k)
        bound = 2.0 ** -24 * (2.0 + 16.0 * norm) * np.abs(b - before[k])[1:-1, 1:-1].max()
        assert np.abs(g.field(k) - b).max() <= bound + 1e-12 * np.abs(b).max(), k
    g.close()
