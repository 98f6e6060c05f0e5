"""Grid-free relaxation: the order of the atom sums, and with it every bit of the result, is the same at both
lane counts per pixel that a molecule takes (half as many from some scan size on)."""
import numpy as np
import pytest
import torch

from spammm_b200 import _lib, gpu

pytestmark = pytest.mark.gpu


# pixels on both sides of the scan sizes at which the molecule's lane count halves
@pytest.mark.parametrize("na,few,many", [(17, 4800, 9600), (32, 4800, 9600), (33, 2400, 4800), (38, 2400, 4800), (64, 2400, 4800),
                                         (65, 1200, 2400), (101, 1200, 2400), (128, 1200, 2400)])
@pytest.mark.parametrize("sites", [0, 1, 2])
def test_scan_size_does_not_change_bits(cuda, na, few, many, sites):
    rng = np.random.default_rng(na)
    atoms = np.zeros((na, 4), np.float32)
    r = 0.8 * np.sqrt(na)
    atoms[:, :2] = rng.uniform(-r, r, (na, 2))
    atoms[:, 3] = rng.uniform(-0.3, 0.3, na)
    cMs = np.stack([rng.uniform(3.2, 3.5, na), rng.uniform(2e-3, 3e-3, na), np.full(na, -1.8), np.zeros(na)], 1)
    pts = np.zeros((many, 4), np.float32)
    pts[:, :2], pts[:, 2] = rng.uniform(-4, 4, (many, 2)), 11.0
    Qs, QZs = [0, -0.1 * (sites > 0), 0.1 * (sites > 1), 0], [0, 1.8, 3.6, 0]
    P = _lib.make_scan_params(tipC=[0, 0, 1, -0.1], stiffness=[-0.03, -0.03, -0.03, -20.0], dpos0=[0, 0, -4.0, 4.0],
                              relax_params=[0.5, 0.1, 0.02, 0.5], nz=6, max_iter=300, f2conv=1e-8)
    a = gpu.relax_direct_morse(atoms, cMs.astype(np.float32), pts[:few], P, Qs, QZs)
    b = gpu.relax_direct_morse(atoms, cMs.astype(np.float32), pts, P, Qs, QZs)
    for x, y in zip(a, b):
        assert torch.equal(x, y[:few])
