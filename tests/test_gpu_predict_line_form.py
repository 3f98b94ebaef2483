"""The 2D predictor's line-streaming form on the grids that take it, and at
its remainders.

Grids of 2^19 cells and more with rows of more than 768 cells stream their
lines (k_predict_rhs, _xsolve, _update); all others run the fused kernel
(SVOF_PREDICT_LINES forces one).  Against the oracle on grids that the rule
leads there; bit for bit against the fused form on long rows of odd length and
on numbers of rows that leave the last block of 32 lines partly filled.
"""
import os

import numpy as np
import pytest

from oracle import Oracle
from simplevofsolver_b200 import DROPLET2D_ENV, Solver, droplet2d, physical_params

pytestmark = pytest.mark.gpu

WALLS = dict(uy_walls=(0.1, -0.1), t_walls=(0.5, -0.5))


def solver(ic, lines=None):
    if lines is not None:
        os.environ["SVOF_PREDICT_LINES"] = lines
    try:
        return Solver(ic, physical_params(DROPLET2D_ENV), **WALLS)
    finally:
        os.environ.pop("SVOF_PREDICT_LINES", None)


# the predictor is linear in its inputs at a given dt: 1e-12 of each field's range
@pytest.mark.parametrize("nx,ny,uniform", [(1024, 512, True), (1024, 515, True), (769, 1024, False), (1501, 512, False)])
def test_predictor_vs_oracle(gpu_available, nx, ny, uniform):
    ic = droplet2d(nx, ny, uniform=uniform, noise=1e-2, nsub=2)
    g, o = solver(ic), Oracle(ic, physical_params(DROPLET2D_ENV), **WALLS)
    for rk, dt in ((0, 1e-4), (1, 1e-4), (0, 1e-2)):
        g.fluid_predict_field(rk, dt)
        o.predict(rk, dt)
        for k in ("ux", "uy", "t"):
            a, b = g.field(k), o.field(k)
            assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), (rk, dt, k)
    g.close()


def test_step_vs_oracle(gpu_available):
    ic = droplet2d(1024, 512, noise=1e-2)
    g, o = solver(ic), Oracle(ic, physical_params(DROPLET2D_ENV), **WALLS)
    assert g.integrate() == o.run(1)[0]
    for k in ("ux", "uy", "t", "vof", "p"):
        a, b = g.field(k), o.field(k)
        if "p" == k:
            a, b = ((v - v[1:-1, 1:-1].mean())[1:-1] for v in (a, b))
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), k
    g.close()


@pytest.mark.parametrize("nx,ny,uniform", [(1024, 37, True), (1024, 515, True), (769, 8, False), (1025, 16, False),
                                           (1501, 128, False)])
def test_forms_are_bit_identical(gpu_available, nx, ny, uniform):
    ic = droplet2d(nx, ny, uniform=uniform, noise=1e-2, nsub=2)
    out = []
    for lines in ("0", "1"):
        s = solver(ic, lines)
        out.append((s.run(3), {k: s.field(k) for k in ("ux", "uy", "t", "p", "vof", "srcux_a", "srcuy_a", "srct_a")}))
        s.close()
    assert np.array_equal(out[0][0], out[1][0])
    for k, a in out[0][1].items():
        assert np.array_equal(a, out[1][1][k]), k
