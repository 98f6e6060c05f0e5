"""Amplitude df as one filter per direction (df_amp_z_kernel, df_amp_tile_kernel) against the FP64
oracle's node-by-node form.

The outputs are float32 roundings of FP64 values: 2^-24 relative, taken as 2e-7.  The FP64 values
differ by the rounding of j + u shift (half an ulp of up to 600 samples, 6e-14 of a sample difference)
and of sums of 18-72 terms (1e-14), both divided by the spacing: 1e-11 max|F| / dr in all.
"""
import numpy as np
import pytest

from oracle import oracle as O
from spammm_b200 import gpu

pytestmark = pytest.mark.gpu


def _check(shape, spacing, direction, amp, dtype, out_iz=None):
    rng = np.random.default_rng(sum(shape))
    F = rng.standard_normal(shape + (4,)).astype(dtype)
    got = gpu.df_amp_dir(F, spacing, direction, amp, out_iz=out_iz).cpu().numpy()
    ref = O.compute_df_amp_dir(F.astype(np.float64), spacing, direction, amp)
    if out_iz is not None:
        ref = ref[:, :, out_iz]
    dr = np.min(spacing)
    np.testing.assert_allclose(got, ref, rtol=2e-7, atol=1e-11 * np.abs(F).max() / dr)


@pytest.mark.parametrize("nz", [2, 3, 31, 32, 33, 63, 64, 65, 130, 480, 512, 513])
@pytest.mark.parametrize("amp", [0.0, 0.04, 1.0, 7.3])
def test_z_columns(cuda, nz, amp):
    """Column lengths around the warp, the table and the padded buffer (nz + reach of the taps > 512:
    clamped taps; 513: the three-dimensional kernel), reaches below one sample to beyond the column."""
    _check((3, 5, nz), 0.1, (0., 0., 1.), amp, np.float32)
    _check((3, 3, nz), (0.2, 0.3, 0.05), (0., 0., -2.), amp, np.float64)


@pytest.mark.parametrize("shape", [(1, 5, 7), (4, 8, 32), (5, 9, 33), (13, 17, 41), (9, 2, 64)])
@pytest.mark.parametrize("direction", [(0.2, 0.1, 1.0), (0.0, 1.0, 0.0), (0.0, -0.7, 0.7)])
@pytest.mark.parametrize("amp", [0.03, 0.5, 1.7])
def test_tilted_tiles(cuda, shape, direction, amp):
    """Tiles with remainders, one to three active axes (axis 0 of length 1 only where it is inactive)."""
    if shape[0] < 2 and direction[0] != 0.0:
        shape = (2,) + shape[1:]
    _check(shape, (0.1, 0.12, 0.11), direction, amp, np.float64)
    _check(shape, 0.1, direction, amp, np.float32)


def test_tilted_heights_and_reach(cuda):
    """A height list (one tile of all heights), tiles shrunk by a long reach, and a reach that fits no tile."""
    _check((7, 9, 70), 0.1, (0.3, 0.0, 1.0), 0.8, np.float32, out_iz=[69, 0, 12, 33])
    _check((40, 30, 20), 0.1, (1.0, 0.3, 0.2), 1.5, np.float32)
    _check((12, 10, 40), 0.1, (1.0, 1.0, 1.0), 6.0, np.float64)


def test_height_outside_the_volume_is_nan(cuda):
    F = np.random.default_rng(0).standard_normal((4, 5, 12, 4)).astype(np.float32)
    for d in ((0., 0., 1.), (0.1, 0., 1.)):
        got = gpu.df_amp_dir(F, 0.1, d, 0.5, out_iz=[-1, 3, 12]).cpu().numpy()
        assert np.isnan(got[..., [0, 2]]).all() and np.isfinite(got[..., 1]).all()


@pytest.mark.parametrize("heights", [[17], [0, 39], list(range(0, 40, 4))])
def test_tilted_height_list_of_a_large_volume(cuda, heights):
    """Short lists are evaluated node by node, longer ones and the whole volume from tiles."""
    F = np.random.default_rng(2).standard_normal((260, 250, 40, 4)).astype(np.float32)
    d = (0.2, 0.1, 1.0)
    got = gpu.df_amp_dir(F, 0.1, d, 1.0, out_iz=heights).cpu().numpy()
    ref = gpu.df_amp_dir(F, 0.1, d, 1.0).cpu().numpy()[:, :, heights]
    np.testing.assert_allclose(got, ref, rtol=2e-7, atol=1e-11 * np.abs(F).max() / 0.1)


def _linear_without_zero_weights(F, coords):
    """Linear interpolation with clamped indices; a corner of weight zero is not read."""
    f = np.floor(coords)
    out = np.zeros(F.shape)
    for c in np.ndindex(2, 2, 2):
        w = np.prod([np.where(c[d], coords[d] - f[d], 1.0 - (coords[d] - f[d])) for d in range(3)], axis=0)
        v = F[tuple(np.clip(f[d].astype(int) + c[d], 0, F.shape[d] - 1) for d in range(3))]
        out += np.where(w == 0.0, 0.0, v * w)
    return out


def test_long_reach_across(cuda):
    """A reach of nine samples in the plane: node by node where tiles would stage hundreds of points per output."""
    _check((64, 64, 100), 0.1, (1.0, 1.0, 0.0), 1.25, np.float32)
    _check((64, 64, 40), 0.1, (1.0, 1.0, 0.0), 1.25, np.float32)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("direction", [(0., 0., 1.), (0., 0., -1.), (0.2, 0., 1.), (0.3, 0.2, 1.), (0., 1., 0.)])
@pytest.mark.parametrize("amp", [0.1, 0.37])
def test_samples_that_are_not_finite(cuda, value, direction, amp, monkeypatch):
    """They reach the outputs that they reach node by node: the same NaN, infinities and finite values."""
    rng = np.random.default_rng(7)
    F = rng.standard_normal((9, 8, 40, 4)).astype(np.float32)
    for x, y, z, c in ((4, 4, 20, 2), (0, 0, 0, 2), (8, 7, 39, 2), (2, 6, 5, 0), (6, 2, 33, 1), (4, 1, 12, 3)):
        F[x, y, z, c] = value
    monkeypatch.setattr(O, "_linear_nearest", _linear_without_zero_weights)
    with np.errstate(invalid="ignore"):
        ref = O.compute_df_amp_dir(F.astype(np.float64), 0.1, direction, amp)
    got = gpu.df_amp_dir(F, 0.1, direction, amp).cpu().numpy()
    np.testing.assert_allclose(got, ref, rtol=2e-7, atol=1e-9)
