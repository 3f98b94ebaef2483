"""The tensors a rollout takes as its initial fields: on either device, of
another precision, strided, with leading dimensions of length one or
broadcasting to the field's shape, as assignment to an array takes them; a
shape that fits neither is a ValueError.
"""
import numpy as np
import pytest

from simplevofsolver_b200 import (DROPLET2D_ENV, DROPLETS3D_ENV, Solver, Solver3D, droplet2d, droplets3d,
                                  physical_params)

pytestmark = pytest.mark.gpu


def make(three):
    import torch
    from simplevofsolver_b200.adjoint import Rollout, Rollout3D
    if three:
        ic = droplets3d(18, 8, 16, ndrops=2, radii=(0.15, 0.2), seed=3)
        r = Rollout3D(Solver3D(ic, physical_params(DROPLETS3D_ENV)), [1e-3], 1)
    else:
        ic = droplet2d(32, 20, noise=1e-2)
        r = Rollout(Solver(ic, physical_params(DROPLET2D_ENV)), [1e-3], 1)
    names = ("ux", "uy", "uz", "vof") if three else ("ux", "uy", "vof")
    # (values of 24 bits, so that every form below holds the same ones)
    xs = [torch.tensor(getattr(ic, k)[..., 1:-1], dtype=torch.float32, device="cuda").double() for k in names]
    return r, xs


def run(r, xs):
    return [o.cpu().numpy() for o in r.forward(*xs, 0.1)]


FORMS = {"host": lambda a: a.cpu(), "fp32": lambda a: a.float(), "grad": lambda a: a.clone().requires_grad_(True),
         "strided": lambda a: a.repeat_interleave(2, -1)[..., ::2], "transposed": lambda a: a.mT.contiguous().mT,
         "leading": lambda a: a[None]}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("three", [False, True])
def test_forms(gpu_available, form, three):
    if three and "leading" == form:
        pytest.skip("3D fields were never taken with leading dimensions")
    r, xs = make(three)
    want = run(r, xs)
    for a, b in zip(run(r, [FORMS[form](x) for x in xs]), want):
        assert np.array_equal(a, b)


def test_broadcast(gpu_available):
    r, xs = make(False)
    row = [x[:1] for x in xs]
    for a, b in zip(run(r, row), run(r, [x.expand(20, -1).contiguous() for x in row])):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("three", [False, True])
@pytest.mark.parametrize("cut", [lambda x: x[..., :-1], lambda x: x[..., 1:, :], lambda x: x[None].expand(2, *x.shape)])
def test_other_shapes_are_refused(gpu_available, three, cut):
    r, xs = make(three)
    with pytest.raises(ValueError):
        run(r, [cut(xs[0])] + xs[1:])
