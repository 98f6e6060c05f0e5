"""Tile widths of the counter-scheduled relaxation (32 pixels per warp down to 1 for small scans): the bits of
the flattened kernel (no counter), for rasters whose edges cut tiles and for scans without a raster."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from spammm_b200 import _lib, gpu

pytestmark = pytest.mark.gpu


def _grid():
    rng = np.random.default_rng(1)
    atoms = np.zeros((9, 4), np.float32)
    atoms[:, :2] = rng.uniform(-2.5, 2.5, (9, 2))
    atoms[:, 3] = rng.uniform(-0.3, 0.3, 9)
    prm = np.stack([np.full(9, 3.3), rng.uniform(2e-3, 3e-3, 9), np.full(9, -1.8), np.zeros(9)], 1).astype(np.float32)
    n, o = (60, 56, 40), (-6.0, -5.6, 0.5)
    vec = (np.array([*o, 0], np.float32), np.array([0.2, 0, 0, 0], np.float32), np.array([0, 0.2, 0, 0], np.float32),
           np.array([0, 0, 0.2, 0], np.float32))
    g = gpu.grid_build(1, atoms, prm, n, *vec, [-0.05, 0, 0, 0], [0, 0, 0, 0])
    return g, O.dinv_axis_aligned(np.array(n) * 0.2, np.array(o), n)


@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 5), (17, 23), (41, 37), (61, 53), (103, 59), (137, 101), (149, 131)])
@pytest.mark.parametrize("raster", [True, False])
@pytest.mark.parametrize("radial", [False, True])
def test_widths_give_the_flattened_bits(cuda, nx, ny, raster, radial):
    grid, dinv = _grid()
    xs, ys = np.linspace(-3, 3, nx), np.linspace(-2.5, 2.5, ny)
    pts = np.zeros((nx * ny, 4), np.float32)
    pts[:, 0], pts[:, 1], pts[:, 2] = np.repeat(xs, ny), np.tile(ys, nx), 6.0
    stiff, d0 = ([-0.02, -0.02, -0.03, -1.0], [0, 0, -1.0, 1.0]) if radial else ([-0.0156, -0.0156, -1.25, 0], [0] * 4)
    kw = dict(dinv=dinv, dTip=[0, 0, -0.1, 0], tipC=[0, 0, 1, -0.1], stiffness=stiff, dpos0=d0,
              relax_params=[0.5, 0.1, 0, 0], nz=5, max_iter=200, f2conv=1e-9, raster_ny=ny if raster else 0)
    p = torch.from_numpy(pts).cuda()
    for polish in (False, True):
        P = _lib.make_scan_params(polish=polish, **kw)
        for fn in (gpu.relax_strokes, gpu.relax_pp):
            a, b = fn(grid, P, p), fn(grid, P, p, dynamic=False)
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
        assert torch.equal(gpu.relax_strokes_tilted(grid, P, p), gpu.relax_strokes_tilted(grid, P, p, dynamic=False))


def _same(a, b):
    """The same values, NaN at the same places."""
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a, nan=0.0), torch.nan_to_num(b, nan=0.0))


@pytest.mark.parametrize("max_iter", [0, 1, 3, 40])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("polish", [False, True])
def test_values_that_are_not_finite_spread_as_in_the_general_loop(cuda, max_iter, value, polish):
    """The axis-aligned loop leaves out products with zeros; a component of the field, or the surface bias, that is
    not finite must still reach what it reaches through them."""
    grid, dinv = _grid()
    pts = np.zeros((40 * 31, 4), np.float32)
    pts[:, 0], pts[:, 1], pts[:, 2] = np.repeat(np.linspace(-3, 3, 40), 31), np.tile(np.linspace(-2.5, 2.5, 31), 40), 6.0
    kw = dict(dinv=dinv, dTip=[0, 0, -0.1, 0], tipC=[0, 0, 1, -0.1], stiffness=[-0.0156, -0.0156, -1.25, 0],
              dpos0=[0] * 4, relax_params=[0.5, 0.1, 0, 0], nz=5, max_iter=max_iter, f2conv=1e-9, raster_ny=31,
              polish=polish)
    p = torch.from_numpy(pts).cuda()
    for c in range(4):
        g = grid.clone()
        g[:, 20:30, 25:40, c] = value
        P = _lib.make_scan_params(**kw)
        for fn in (gpu.relax_strokes, gpu.relax_pp):
            a, b = fn(g, P, p), fn(g, P, p, dynamic=False)
            assert _same(a[0], b[0]) and _same(a[1], b[1]), (fn.__name__, c)
        assert _same(gpu.relax_strokes_tilted(g, P, p), gpu.relax_strokes_tilted(g, P, p, dynamic=False)), c
    P = _lib.make_scan_params(surfFF=[value, 0, 0, 0], **kw)
    a, b = gpu.relax_pp(grid, P, p), gpu.relax_pp(grid, P, p, dynamic=False)
    assert _same(a[0], b[0]) and _same(a[1], b[1])
