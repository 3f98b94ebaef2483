"""The initial pressure and temperature of a rollout are the caller's to change.

``Rollout.p0`` / ``.t0`` (2D and 3D) are arrays in the restart layout: an edit
in place and an assignment both reach the next forward pass, whose outputs are
the bits of a rollout of a solver made with those fields.
"""
import copy

import numpy as np
import pytest

from simplevofsolver_b200 import (DROPLET2D_ENV, DROPLETS3D_ENV, Solver, Solver3D, droplet2d, droplets3d,
                                  physical_params)

pytestmark = pytest.mark.gpu

DTS = [1e-3, 2e-3]


def make(three):
    from simplevofsolver_b200.adjoint import Rollout, Rollout3D
    if three:
        ic, phys = droplets3d(17, 8, 16, ndrops=2, radii=(0.15, 0.2), seed=3), physical_params(DROPLETS3D_ENV)
        return ic, lambda c: Rollout3D(Solver3D(c, phys, add_buoyancy=True), DTS, 2)
    ic, phys = droplet2d(32, 20, noise=1e-2), physical_params(DROPLET2D_ENV)
    return ic, lambda c: Rollout(Solver(c, phys, add_buoyancy=True), DTS, 2)


def forward(ic, r):
    import torch
    xs = [torch.tensor(getattr(ic, k)[..., 1:-1], dtype=torch.float64, device="cuda")
          for k in (("ux", "uy", "uz", "vof") if hasattr(ic, "uz") else ("ux", "uy", "vof"))]
    return [o.cpu().numpy() for o in r.forward(*xs, 0.1)]


@pytest.mark.parametrize("three", [False, True])
@pytest.mark.parametrize("how", ["edited", "assigned"])
def test_initial_fields_can_be_changed(gpu_available, three, how):
    ic, rollout = make(three)
    rng = np.random.default_rng(5)
    changed = copy.deepcopy(ic)
    for a in (changed.p, changed.t):
        a[..., 1:-1] = rng.uniform(-1e-2, 1e-2, a[..., 1:-1].shape)
    r = rollout(ic)
    before = forward(ic, r)
    if how == "edited":
        r.p0[..., 1:-1] = changed.p[..., 1:-1]
        r.t0[..., 1:-1] += changed.t[..., 1:-1]
    else:
        r.p0, r.t0 = changed.p, changed.t
    got = forward(ic, r)
    want = forward(ic, rollout(changed))
    for a, b, c in zip(got, want, before):
        assert np.array_equal(a, b)
    assert not np.array_equal(got[0], before[0])
