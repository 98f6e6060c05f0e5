"""Node-major gradients through a grid build (spm_adjoint_grid_params_nodes) against the state-major gather.

Both sum float32 pair derivatives of about 1e-6 relative error in FP64; the node-major form rounds the same
products w*ubar to a multiple of 2^-42 of their largest: 5e-6 of the column's norm bounds the difference of
sums whose terms cancel by up to a factor of five."""
import numpy as np
import pytest
import torch

from spammm_b200 import _lib, gpu

pytestmark = pytest.mark.gpu


def _case(kind, na, nxy, nz, seed, n=(70, 66, 60), step=0.2, spread=6.0, sites=([-0.05, 0.1, 0, 0], [0, 1.2, 0, 0])):
    rng = np.random.default_rng(seed)
    atoms = np.zeros((na, 4), np.float32)
    atoms[:, :2] = rng.uniform(-4, 4, (na, 2))
    atoms[:, 2] = rng.normal(0, 0.1, na)
    atoms[:, 3] = rng.uniform(-0.3, 0.3, na)
    R0, E0 = rng.uniform(3.0, 3.5, na), rng.uniform(2e-3, 3e-3, na)
    prm = (np.stack([2 * E0 * R0 ** 6, E0 * R0 ** 12], 1) if kind == 0
           else np.stack([R0, E0, np.full(na, -1.8), np.zeros(na)], 1)).astype(np.float32)
    o = np.array([-step * n[0] / 2, -step * n[1] / 2, 2.0])
    L = np.array(n) * step
    dinv = [np.array([1 / L[d] if c == d else 0 for c in range(3)] + [-o[d] / L[d] + 0.5 / n[d]], np.float32) for d in range(3)]
    P = _lib.make_scan_params(dinv=dinv, tipC=[0, 0, 1, -0.1], nz=nz)
    m = nxy * nz
    PP = np.zeros((m, 4), np.float32)
    PP[:, :2] = np.repeat(rng.uniform(-spread, spread, (nxy, 2)), nz, 0) + rng.normal(0, 0.03, (m, 2))
    PP[:, 2] = 8.0 - 0.1 * np.tile(np.arange(nz), nxy) + rng.normal(0, 0.02, m)
    PP[:, 3] = 5
    ub = rng.normal(0, 1e-3, (m, 4)).astype(np.float32)
    ub[rng.random(m) < 0.1] = 0
    dk = rng.normal(0, 1, (m, 4)).astype(np.float32)
    vec = (np.array([*o, 0]), [step, 0, 0, 0], [0, step, 0, 0], [0, 0, step, 0])
    grid = torch.empty((n[2], n[1], n[0], 4), device="cuda")
    return (kind, atoms, prm, *vec, *sites, grid, P, PP, ub, dk)


def _both(args, monkeypatch):
    out = []
    monkeypatch.setattr(gpu, "NODES_MIN_ATOMS", 1)
    monkeypatch.setattr(gpu, "NODES_MIN_STATES", 1)
    for limit in (1 << 62, 0):
        monkeypatch.setattr(gpu, "NODES_MIN_PAIRS", limit)
        out.append(gpu.adjoint_grid_params(*args))
    return out


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("na,nxy,nz", [(1, 1, 1), (3, 7, 5), (38, 300, 12), (65, 97, 33), (257, 40, 9), (300, 11, 64)])
def test_matches_state_major(cuda, kind, na, nxy, nz, monkeypatch):
    """Atom counts around the CTA's slots, scans around a warp; the raster crosses the grid's seam."""
    a, b = _both(_case(kind, na, nxy, nz, seed=na + nz, spread=8.0), monkeypatch)
    assert torch.equal(a[1], b[1])
    for c in range(6):
        d, s = (a[0][:, c] - b[0][:, c]).norm(), a[0][:, c].norm()
        assert d <= 5e-6 * s, f"column {c}: {float(d / s):.1e}"


def test_repeats_bit_for_bit_and_ignores_the_scratch(cuda, monkeypatch):
    args = _case(0, 38, 200, 20, seed=5)
    monkeypatch.setattr(gpu, "NODES_MIN_PAIRS", 0)
    monkeypatch.setattr(gpu, "NODES_MIN_STATES", 1)
    a = gpu.adjoint_grid_params(*args)
    junk = torch.full((40 << 20,), 3.7e5, device="cuda")  # what the next scratch may be made of
    del junk
    b = gpu.adjoint_grid_params(*args)
    assert torch.equal(a[0], b[0])


def test_no_weight_and_weights_that_are_not_finite(cuda, monkeypatch):
    args = list(_case(0, 38, 50, 20, seed=7))
    monkeypatch.setattr(gpu, "NODES_MIN_PAIRS", 0)
    monkeypatch.setattr(gpu, "NODES_MIN_STATES", 1)
    ub = args[12]
    args[12] = np.zeros_like(ub)
    assert torch.count_nonzero(gpu.adjoint_grid_params(*args)[0]) == 0
    for v in (np.nan, np.inf):
        args[12] = ub.copy()
        args[12][33, 2] = v
        assert not torch.isfinite(gpu.adjoint_grid_params(*args)[0]).any()


@pytest.mark.parametrize("n_state", [(1 << 20) + 1, (1 << 22) + 12345])
def test_every_state_on_one_node(cuda, n_state, monkeypatch):
    """Like-signed adjoints of equal size on one node: 64-bit sums in units of 2^-42 would wrap beyond 2^21 states."""
    args = list(_case(0, 9, 2, 1, seed=3))
    n, o, step = (70, 66, 60), np.array([-7.0, -6.6, 2.0]), 0.2
    PP = np.zeros((n_state, 4), np.float32)
    PP[:, :3], PP[:, 3] = o + step * np.array([31, 33, 24]), 5
    ub = np.tile(np.array([[0.0019, -0.00195, 0.0018, 0.0011]], np.float32), (n_state, 1))
    args[11], args[12], args[13] = PP, ub, np.zeros_like(ub)
    a, b = _both(tuple(args), monkeypatch)
    for c in range(6):
        d, s = float((a[0][:, c] - b[0][:, c]).norm()), float(a[0][:, c].norm())
        assert d <= 5e-6 * s, f"column {c}: {d / max(s, 1e-300):.1e}"


def test_gather_where_the_node_sums_do_not_fit(cuda, monkeypatch):
    """The scratch of the node sums (32 bytes per grid node) cannot be had: the gather's gradients, as before."""
    args = _case(0, 38, 200, 20, seed=5)
    ref, nodes = _both(args, monkeypatch)
    empty, refused = torch.empty, []

    def short(*a, **k):
        t = empty(*a, **k)
        if t.numel() * t.element_size() > 8_000_000:
            refused.append(t.numel())
            raise torch.OutOfMemoryError("no memory")
        return t

    monkeypatch.setattr(torch, "empty", short)
    got = gpu.adjoint_grid_params(*args)
    assert refused and torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
    assert not torch.equal(nodes[0], ref[0])
