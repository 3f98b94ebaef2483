"""load_interior_device puts a CUDA tensor where load_interior puts an array,
halo and wall update included, and refuses what is not a contiguous float64
CUDA tensor of the field's restart shape, leaving the field as it was.
"""
import numpy as np
import pytest

from simplevofsolver_b200 import (DROPLET2D_ENV, DROPLETS3D_ENV, FIELDS, Solver, Solver3D, droplet2d,
                                  droplets3d, interior_shape, interior_shape3d, lib, physical_params)

pytestmark = pytest.mark.gpu


def make(three):
    """two solvers with moving, heated walls, and the restart shapes of their fields"""
    if three:
        ic, kw = droplets3d(9, 8, 4, ndrops=0, seed=1), dict(uy_walls=(0.1, -0.2), uz_walls=(0.3, 0.), t_walls=(1., -1.))
        shapes = {k: interior_shape3d(k, 9, 8, 4) for k in ("ux", "uy", "uz", "p", "t", "vof")}
        return [Solver3D(ic, physical_params(DROPLETS3D_ENV), **kw) for _ in range(2)], shapes
    ic, kw = droplet2d(16, 9), dict(uy_walls=(0.1, -0.2), t_walls=(1., -1.))
    shapes = {k: interior_shape(k, 16, 9) for k in ("ux", "uy", "p", "t", "vof")}
    return [Solver(ic, physical_params(DROPLET2D_ENV), **kw) for _ in range(2)], shapes


@pytest.mark.parametrize("three", [False, True])
def test_same_as_from_the_host(gpu_available, three):
    import torch
    (a, b), shapes = make(three)
    rng = np.random.default_rng(3)
    for k, shape in shapes.items():
        x = rng.uniform(0.0, 1.0, shape)
        a.load_interior(k, x)
        b.load_interior_device(k, torch.from_numpy(x).cuda())
        assert np.array_equal(a.field(k), b.field(k)), k
        assert np.array_equal(b.interior(k)[..., 1:-1], x[..., 1:-1]), k


@pytest.mark.parametrize("three", [False, True])
def test_refusals(gpu_available, three):
    import torch
    (a, _), shapes = make(three)
    good = torch.ones(shapes["uy"], dtype=torch.float64, device="cuda")
    wide = torch.ones(shapes["uy"][:-1] + (2 * shapes["uy"][-1],), dtype=torch.float64, device="cuda")
    before = a.field("uy")
    for bad in (good.cpu(), good.float(), good[..., :-1].contiguous(), good[None], wide[..., ::2], good.cpu().numpy()):
        with pytest.raises(ValueError):
            a.load_interior_device("uy", bad)
    assert np.array_equal(a.field("uy"), before)
    a.load_interior_device("uy", good)
    assert not np.array_equal(a.field("uy"), before)


def test_count_is_checked_at_the_c_entry(gpu_available):
    import torch
    (a, _), shapes = make(False)
    x = torch.ones(shapes["p"], dtype=torch.float64, device="cuda")
    assert 0 != lib().svof_load_interior_device(a._h, FIELDS["p"], x.data_ptr(), x.numel() - 1)
    assert 0 != lib().svof_load_interior_device(a._h, FIELDS["p"], None, x.numel())
    assert 0 != lib().svof_load_interior_device(None, FIELDS["p"], x.data_ptr(), x.numel())
    assert not np.any(a.interior("p"))
