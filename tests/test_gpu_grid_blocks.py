"""Force grids of 256 atoms or more: blocks of 16^3 nodes whose distant atoms are interpolated from 8^3
Chebyshev points (build_cell, grid_build.cu), against the FP64 pair sums.

Bound per channel: 1e-5 S (S the sum of the atoms' contribution magnitudes) + the float32 node-coordinate
term of test_gpu_scale.py.  A pair term errs by up to 2e-6 (rsqrt.approx to the 13th power) or, for Morse
(direct sums), 4e-6 (the float32 exponent of up to 40); the interpolation adds at most 1e-6 of an LJ atom's
force at the node.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from spammm_b200 import gpu
from spammm_b200.batch import AFMBatch, BatchItem
from test_gpu_scale import pos_term

pytestmark = pytest.mark.gpu

NONE = ([0, 0, 0, 0], [0, 0, 0, 0])
ON = ([-0.05, 0, 0, 0], [0, 0, 0, 0])
OFF = ([0, -0.1, 0.1, 0], [0, 1.8, 3.6, 0])
BOTH = ([-0.05, 0.2, -0.1, 0.05], [0, -0.7, 1.8, 3.6])


def _system(na, kind, extent, seed=3):
    rng = np.random.default_rng(seed + na)
    atoms = np.zeros((na, 4), np.float32)
    atoms[:, :2] = rng.uniform(-extent, extent, (na, 2))
    atoms[:, 2] = rng.uniform(-3.0, 0.5, na)
    atoms[:, 3] = rng.uniform(-0.8, 0.8, na)
    R0, E0 = rng.uniform(3.0, 3.5, na), rng.uniform(2e-3, 3e-3, na)
    prm = (np.stack([2 * E0 * R0 ** 6, E0 * R0 ** 12], 1) if kind == 0
           else np.stack([R0, E0, np.full(na, -1.8), np.zeros(na)], 1))
    return atoms, prm.astype(np.float32)


def _check(kind, atoms, prm, n, p0, dA, dB, dC, sites, tol_sum=1e-5, tol_rel=2e-5):
    p0, dA, dB, dC = (np.array([*v, 0], np.float32) for v in (p0, dA, dB, dC))
    Qs, QZs = (np.array(v, np.float32) for v in sites)
    g = gpu.grid_build(kind, atoms, prm, n, p0, dA, dB, dC, Qs, QZs).cpu().numpy().reshape(-1, 4).astype(np.float64)
    iz, iy, ix = (a.reshape(-1, 1) for a in np.meshgrid(*(np.arange(k) for k in n[::-1]), indexing="ij"))
    q = (p0.astype(np.float64) + ix * dA.astype(np.float64) + iy * dB.astype(np.float64) + iz * dC.astype(np.float64))[:, :3]
    pick = np.random.default_rng(0).permutation(len(q))[:60000]
    edge = np.flatnonzero((ix[:, 0] % 16 == 15) & (iy[:, 0] % 16 == 0) & (iz[:, 0] % 16 == 15))
    pick = np.unique(np.concatenate([pick, edge, [0, len(q) - 1]]))
    q, g = np.ascontiguousarray(q[pick]), g[pick]
    a64, p64 = atoms.astype(np.float64), prm.astype(np.float64)
    ref = O.pair_fe(kind, a64, p64, q, Qs, QZs)
    cap = np.minimum(1.0, 100.0 / np.abs(ref[:, 3]))[:, None]
    ref, S = ref * cap, O.pair_fe_abs(kind, a64, p64, q, Qs, QZs) * cap
    err = np.abs(g - ref)
    bad = err > tol_sum * S + tol_rel * np.abs(ref) + pos_term(q, a64, ref)
    assert not bad.any(), f"{bad.sum()} values out of bound, worst err/S {(err / S).max():.2e}"


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("na", [31, 32, 33, 255, 256, 257, 600])
@pytest.mark.parametrize("sites", [ON, OFF, BOTH], ids=["on", "off", "both"])
def test_against_pair_sums(cuda, kind, na, sites):
    """Both sides of the atom count where blocks begin (256), further gathers; ragged boxes."""
    atoms, prm = _system(na, kind, 12.0)
    _check(kind, atoms, prm, (97, 65, 81), (-12.0, -5.0, -4.0), (0.1, 0, 0), (0, 0.1, 0), (0, 0, 0.1), sites)


@pytest.mark.parametrize("kind,na", [(k, na) for k in (0, 1) for na in (31, 32, 57, 120, 255)] + [(1, 256), (1, 600)])
def test_molecules_and_morse_are_summed_directly(cuda, kind, na):
    """Below 256 atoms, and for Morse at any size, a node's bits are those of its own pair sums."""
    _same_in_any_box(kind, na, 0.0625 if kind else 0.125, (70, 61, 66))


@pytest.mark.parametrize("na,n,h", [(300, (200, 15, 66), 0.125), (511, (15, 200, 66), 0.125), (300, (90, 61, 66), 0.75)])
def test_thin_and_coarse_boxes_are_summed_directly(cuda, na, n, h):
    """Grids where blocks do not pay: fewer columns than a block's and not many atoms, or nodes half an Angstrom apart."""
    _same_in_any_box(0, na, h, n)


def _same_in_any_box(kind, na, h, n):
    """The box around a node does not matter (dyadic spacings, so that both boxes have the same node coordinates)."""
    atoms, prm = _system(na, kind, 6.0)
    cut = (5, 3, 7)
    vec = [np.array(v, np.float32) for v in ((h, 0, 0, 0), (0, h, 0, 0), (0, 0, h, 0))]
    Qs, QZs = (np.array(v, np.float32) for v in BOTH)
    p0 = np.array([-4.5, -3.75, -1.0, 0], np.float32)
    whole = gpu.grid_build(kind, atoms, prm, n, p0, *vec, Qs, QZs)
    p1 = p0 + np.array([*(h * c for c in cut), 0], np.float32)
    part = gpu.grid_build(kind, atoms, prm, tuple(a - c for a, c in zip(n, cut)), p1, *vec, Qs, QZs)
    assert torch.equal(whole[cut[2]:, cut[1]:, cut[0]:], part)


@pytest.mark.parametrize("n", [(1, 1, 1), (15, 16, 17), (33, 2, 64), (200, 3, 31)])
def test_small_and_thin_boxes(cuda, n):
    atoms, prm = _system(300, 0, 14.0)
    _check(0, atoms, prm, n, (-10.0, -8.0, 3.0), (0.1, 0, 0), (0, 0.1, 0), (0, 0, 0.1), ON)


@pytest.mark.parametrize("kind", [0, 1])
def test_spacings_and_skew_cells(cuda, kind):
    """Uneven spacings, a 60-degree cell with a tilted axis, coarse nodes (Morse: near everywhere)."""
    atoms, prm = _system(400, kind, 15.0)
    _check(kind, atoms, prm, (70, 50, 60), (-14.0, -9.0, 1.0), (0.05, 0, 0), (0, 0.16, 0), (0, 0, 0.1), ON)
    _check(kind, atoms, prm, (90, 80, 50), (-8.0, -8.0, 2.0), (0.1, 0, 0.01), (0.05, 0.0866, -0.01), (0, 0, 0.12), BOTH)
    _check(kind, atoms, prm, (40, 40, 30), (-14.0, -14.0, 1.0), (0.35, 0, 0), (0, 0.35, 0), (0, 0, 0.35), ON)


@pytest.mark.parametrize("h", [0.02, 0.03, 0.05, 0.08, 0.1])
@pytest.mark.parametrize("sites", [NONE, ON], ids=["none", "on"])
def test_fine_spacings(cuda, h, sites):
    """Nine half-edges of a block are 1.4 to 6.8 A here: the core of the LJ law must not be interpolated.  Bound: a
    pair term's 2e-6 and the interpolation's 1e-6, of the terms' magnitudes."""
    atoms, prm = _system(300, 0, 6.0)
    n = (160, 160, 128)
    _check(0, atoms, prm, n, (-80 * h, -80 * h, 3.0), (h, 0, 0), (0, h, 0), (0, 0, h), sites, tol_sum=3e-6, tol_rel=0.0)


def test_laws_of_another_shape(cuda):
    """Atoms without a minimum (no attraction, no repulsion, signs turned) and charges alone, on fine nodes."""
    atoms, prm = _system(320, 0, 9.0)
    prm[0::5, 0] = 0.0
    prm[1::5, 1] = 0.0
    prm[2::5] *= -1.0
    prm[3::5] = 0.0
    for h in (0.03, 0.1):
        _check(0, atoms, prm, (96, 96, 64), (-48 * h, -48 * h, 3.4), (h, 0, 0), (0, h, 0), (0, 0, h), ON, tol_sum=3e-6,
               tol_rel=0.0)


@pytest.mark.parametrize("column,value", [("x", np.inf), ("x", 1e30), ("q", np.nan), ("q", np.inf), ("c6", np.nan),
                                          ("c6", np.inf), ("c12", np.nan), ("c12", np.inf)])
def test_values_that_are_not_finite_as_in_direct_sums(cuda, column, value):
    """One atom's coordinate, charge or parameter, far from the box and in it: NaN where the plain sum has NaN, finite
    elsewhere."""
    for at in (3, 200):
        atoms, prm = _system(300, 0, 9.0)
        atoms[at, :3] = (30.0, 2.0, 1.0) if at == 3 else (0.5, 0.5, 4.0)
        {"x": atoms[:, 0], "q": atoms[:, 3], "c6": prm[:, 0], "c12": prm[:, 1]}[column][at] = value
        vec = [np.array([*v, 0], np.float32) for v in ((-3, -3, 3), (0.125, 0, 0), (0, 0.125, 0), (0, 0, 0.125))]
        Qs, QZs = (np.array(v, np.float32) for v in ON)
        g = gpu.grid_build(0, atoms, prm, (48, 48, 40), *vec, Qs, QZs)
        # the direct sums of a subset small enough for them, with the same atom
        keep = np.r_[0:150] if at == 3 else np.r_[100:250]
        d = gpu.grid_build(0, atoms[keep], prm[keep], (48, 48, 40), *vec, Qs, QZs)
        assert torch.equal(torch.isfinite(g), torch.isfinite(d))
        assert torch.equal(torch.isnan(g), torch.isnan(d))


def test_atoms_that_are_not_finite_stay_in_the_sum(cuda):
    """A NaN coordinate is near every block: every node is NaN, as in the plain sum."""
    atoms, prm = _system(264, 0, 8.0)
    atoms[40, 0] = np.nan
    g = gpu.grid_build(0, atoms, prm, (40, 20, 20), *(np.array([*v, 0], np.float32) for v in
                       ((-20, -20, 5), (0.1, 0, 0), (0, 0.1, 0), (0, 0, 0.1))), np.array(ON[0], np.float32),
                       np.array(ON[1], np.float32))
    assert bool(torch.isnan(g).all())


@pytest.mark.parametrize("na", [31, 32, 120, 300])
@pytest.mark.parametrize("layout", [0, 1])
def test_batch_slabs_equal_the_full_grid(cuda, na, layout):
    """A slab's nodes come from the same blocks as the full grid's, whatever box and launch shape."""
    rng = np.random.default_rng(na)
    items = []
    for m, (n, cx) in enumerate((((150, 141, 130), 0.0), ((128, 160, 96), 1.3))):
        atoms, prm = _system(na - 5 * m, 0, 4.0 + na / 60.0, seed=m)
        xs = (cx - 1.5 + 0.25 * np.arange(12)).astype(np.float32)
        items.append(BatchItem(atoms=atoms, params=prm, origin=np.array([-0.05 * n[0], -0.05 * n[1], -5.0]), step=0.1,
                               ngrid=n, xs=xs, ys=xs[:9].copy(), z_top=4.0 + rng.uniform(0, 0.1), nz=8))
    b = AFMBatch(items)
    shape = type(b.shape)(*b.shape.key())
    for ty, zb in ((4, 8), (2, 16), (8, 8)):
        shape.gb_ty, shape.gb_zb, shape.grid_layout = ty, zb, layout
        b.set_shape(shape)
        b.grid.fill_(float("nan"))
        b.build_grids()
        for i, it in enumerate(items):
            p0, dA, dB, dC = it.spec(0, b.probe, b.dtip).vectors()
            full = gpu.grid_build(0, it.atoms, it.params, it.ngrid, p0, dA, dB, dC, b.probe.tipQs, b.probe.tipQZs)
            full = b.slab_of_full(i, full)
            assert torch.equal(b.slab(i), full), f"molecule {i}, gb_ty={ty}"
            assert torch.equal(b.slab(i, 1), torch.roll(full, -1, dims=2))
