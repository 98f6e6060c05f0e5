"""Batch gradients through blocks with a far field (32 to 256 atoms) against the state-major gather.

Float32 pair derivatives of about 1e-6 relative error on both sides, FP64 sums: 5e-6 of the column's norm, as
for the node-major form without blocks."""
import numpy as np
import pytest
import torch

from spammm_b200 import _lib, gpu, synthetic
from spammm_b200.batch import AFMBatch

pytestmark = pytest.mark.gpu


def _items(kind, counts, seed):
    """One molecule per atom count, on grids that end inside a block of 16 nodes."""
    out = []
    for k, na in enumerate(counts):
        out += synthetic.batch_molecules(1, seed=seed + k, kind=kind, natoms=(na, na), side=(9, 11), zside=(9, 11),
                                         npx=(20 + k, 20 + k), nzs=(10 + k, 10 + k))
    return out


def _grads(items, kind, chunk=1024):
    shape = _lib.BatchShape(*_lib.lib().spm_batch_default_shape().key())
    shape.adj_chunk = chunk  # small units: enough of them for the blocks
    b = AFMBatch(items, kind=kind, shape=shape)
    rng = np.random.default_rng(4)
    for i, it in enumerate(b.items):
        b.set_target(i, rng.normal(0.0, 0.05, (len(it.xs), len(it.ys), it.nz)))
    b.forward_adjoint()
    torch.cuda.synchronize()
    return b


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("counts", [(31, 32, 33), (65, 128, 200), (255, 256, 257)])
def test_matches_state_major(cuda, kind, counts, monkeypatch):
    monkeypatch.setattr(gpu, "NODES_MIN_PAIRS", 1 << 62)
    b = _grads(_items(kind, counts, seed=sum(counts)), kind)
    for i, it in enumerate(b.items):
        spec = it.spec(b.kind, b.probe, b.dtip)
        p0, dA, dB, dC = spec.vectors()
        atoms, prm = it.atoms.astype(np.float32), it.params.astype(np.float32)
        grid = gpu.grid_build(kind, atoms, prm, spec.ngrid, p0, dA, dB, dC, spec.tipQs, spec.tipQZs)
        a, c = b._rows(i, "state")
        ref, _ = gpu.adjoint_grid_params(kind, atoms, prm, p0, dA, dB, dC, spec.tipQs, spec.tipQZs, grid,
                                         spec.scan_params(b.probe.stiffness), b.PPs[a:c], b.ubar[a:c], b.dk[a:c])
        got = b.grad_of(i)
        for j in range(6):
            d, s = float((got[:, j] - ref[:, j]).norm()), float(ref[:, j].norm())
            assert d <= 5e-6 * s, f"{len(it.atoms)} atoms, column {j}: {d / max(s, 1e-300):.1e}"


def test_repeats_and_unit_counts(cuda):
    """The same bits call after call (the adjoint grid is left cleared); more or fewer units per molecule than
    lattice cells group the same sums differently."""
    items = _items(0, (40, 64, 90, 120), seed=3)
    b = _grads(items, 0)
    first = b.grad.clone()
    b.forward_adjoint()
    torch.cuda.synchronize()
    assert torch.equal(first, b.grad)
    for chunk in (2048,):
        torch.testing.assert_close(_grads(items, 0, chunk).grad, first, rtol=1e-6, atol=1e-7 * float(first.abs().max()))
