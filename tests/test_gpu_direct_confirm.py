"""Convergence of the grid-free relaxation: every state reported converged has an FP64 force below the
threshold, whether FP64 confirmed it or the float32 force lay below by more than its error bound."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from spammm_b200 import _lib, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na", [1, 9, 38, 120, 256, 257])
@pytest.mark.parametrize("k_rad", [-1.0, -20.0])
@pytest.mark.parametrize("turned", [False, True])
def test_converged_states_are_converged_in_fp64(cuda, na, k_rad, turned):
    rng = np.random.default_rng(na)
    atoms = np.zeros((na, 4), np.float32)
    r = 0.8 * np.sqrt(na)
    atoms[:, :2] = rng.uniform(-r, r, (na, 2))
    atoms[:, 3] = rng.uniform(-0.3, 0.3, na)
    cMs = np.stack([rng.uniform(3.2, 3.5, na), rng.uniform(2e-3, 3e-3, na), np.full(na, -1.8), np.zeros(na)], 1)
    cMs = cMs.astype(np.float32)
    nxy, nz, f2 = 23, 25, 1e-8
    pts = np.zeros((nxy * nxy, 4), np.float32)
    x = np.linspace(-4, 4, nxy)
    pts[:, 0], pts[:, 1], pts[:, 2] = np.repeat(x, nxy), np.tile(x, nxy), 10.6
    c, s = (np.cos(0.1), np.sin(0.1)) if turned else (1.0, 0.0)
    R = np.array([[c, 0, -s], [0, 1, 0], [s, 0, c]], np.float32)
    stiff, d0, Qs, QZs = [-0.03, -0.03, -0.03, k_rad], [0, 0, -4.0, 4.0], [0, -0.1, 0.1, 0], [0, 1.8, 3.6, 0]
    P = _lib.make_scan_params(tipA=R[0], tipB=R[1], tipC=[*R[2], -0.1], stiffness=stiff, dpos0=d0,
                              relax_params=[0.5, 0.1, 0.02, 0.5], nz=nz, max_iter=400, f2conv=f2)
    _, PP = gpu.relax_direct_morse(atoms, cMs, pts, P, Qs, QZs)
    PP = PP.cpu().numpy()
    ok = PP[..., 3] > 0
    assert ok.mean() > 0.9
    step = (R[2] * np.float32(-0.1)).astype(np.float32)
    tip = np.zeros(PP.shape[:2] + (3,), np.float32)
    tip[:, 0] = pts[:, :3]
    for i in range(1, nz):
        tip[:, i] = tip[:, i - 1] + step
    q, t = PP[ok][:, :3].astype(np.float64), tip[ok].astype(np.float64)
    F = O.pair_fe(1, atoms.astype(np.float64), cMs.astype(np.float64), q, Qs, QZs)[:, :3]
    R64, k, l = R.astype(np.float64), np.asarray(np.float32(stiff), np.float64), np.asarray(d0, np.float64)
    d = (q - t) @ R64.T
    n = np.linalg.norm(d, axis=1, keepdims=True)
    G = F + ((d - l[:3]) * k[:3] + d * (k[3] * (n - l[3]) / n)) @ R64
    # the kernel's FP64 sum and this one differ by rounding only
    assert (np.sum(G * G, 1)).max() < float(np.float32(f2)) * (1 + 1e-9)


@pytest.mark.parametrize("na", [9, 38])
def test_stretched_frames(cuda, na):
    """The same with a tip frame of length eight (as accepted as any): its spring is rounded at 32 A and its error
    multiplied by eight."""
    rng = np.random.default_rng(na)
    atoms = np.zeros((na, 4), np.float32)
    r = 0.8 * np.sqrt(na)
    atoms[:, :2] = rng.uniform(-r, r, (na, 2))
    cMs = np.stack([rng.uniform(3.2, 3.5, na), rng.uniform(2e-3, 3e-3, na), np.full(na, -1.8), np.zeros(na)], 1)
    cMs = cMs.astype(np.float32)
    nxy, nz, f2 = 41, 12, 1e-8
    pts = np.zeros((nxy * nxy, 4), np.float32)
    x = np.linspace(-4, 4, nxy)
    pts[:, 0], pts[:, 1], pts[:, 2] = np.repeat(x, nxy), np.tile(x, nxy), 10.6
    c, s = 8.0 * np.cos(0.1), 8.0 * np.sin(0.1)
    R = np.array([[c, 0, -s], [0, 8.0, 0], [s, 0, c]], np.float32)
    stiff, d0 = [-0.03 / 64, -0.03 / 64, -0.03 / 64, -20.0 / 64], [0, 0, -0.5, 32.0]
    P = _lib.make_scan_params(tipA=R[0], tipB=R[1], tipC=[*R[2], -0.0125], stiffness=stiff, dpos0=d0,
                              relax_params=[0.5, 0.1, 0.02, 0.5], nz=nz, max_iter=1000, f2conv=f2)
    _, PP = gpu.relax_direct_morse(atoms, cMs, pts, P, [0, 0, 0, 0], [0, 0, 0, 0])
    PP = PP.cpu().numpy()
    ok = PP[..., 3] > 0
    assert ok.mean() > 0.3
    step = (R[2] * np.float32(-0.0125)).astype(np.float32)
    tip = np.zeros(PP.shape[:2] + (3,), np.float32)
    tip[:, 0] = pts[:, :3]
    for i in range(1, nz):
        tip[:, i] = tip[:, i - 1] + step
    q, t = PP[ok][:, :3].astype(np.float64), tip[ok].astype(np.float64)
    F = O.pair_fe(1, atoms.astype(np.float64), cMs.astype(np.float64), q, [0] * 4, [0] * 4)[:, :3]
    R64, k, l = R.astype(np.float64), np.asarray(np.float32(stiff), np.float64), np.asarray(d0, np.float64)
    d = (q - t) @ R64.T
    n = np.linalg.norm(d, axis=1, keepdims=True)
    G = F + ((d - l[:3]) * k[:3] + d * (k[3] * (n - l[3]) / n)) @ R64
    assert (np.sum(G * G, 1)).max() < float(np.float32(f2)) * (1 + 1e-9)
