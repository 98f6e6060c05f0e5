"""Batches with a radial tip bond, or without FIRE, take the z-synchronised kernel's general form: the bits of the
per-molecule relaxation, as the plain form's."""
import numpy as np
import pytest
import torch

from spammm_b200 import _lib, gpu, synthetic
from spammm_b200.batch import AFMBatch, ProbeSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radial,fire", [(0.0, True), (-1.25, True), (0.0, False)])
@pytest.mark.parametrize("polish", [False, True])
@pytest.mark.parametrize("layout,regs", [(0, 4), (1, 2), (0, 0)])
def test_general_form_matches_per_molecule(cuda, radial, fire, polish, layout, regs):
    items = synthetic.batch_molecules(3, seed=5, natoms=(10, 40), side=(5, 9), zside=(8, 14), npx=(6, 22), nzs=(8, 16))
    k = np.array([-0.0156, -0.0156, -0.3 if radial else -1.25, radial], np.float32)
    d0 = np.array([0, 0, -1.0, 1.0] if radial else [0] * 4, np.float32)
    b = AFMBatch(items, probe=ProbeSpec(stiffness=k, dpos0=d0, max_iter=300, f2conv=1e-8))
    shape = _lib.BatchShape(*b.shape.key())
    shape.rx_sync, shape.grid_layout, shape.rx_regs = 1, layout, regs
    b.set_shape(shape)
    b.set_relax_options(polish=polish)
    if not fire:
        b.scan_params.flags &= ~_lib.SPM_FLAG_FIRE
    b.build_grids()
    b.relax()
    torch.cuda.synchronize()
    for i, it in enumerate(b.items):
        spec = it.spec(b.kind, b.probe, b.dtip)
        p0, dA, dB, dC = spec.vectors()
        grid = gpu.grid_build(0, it.atoms.astype(np.float32), it.params.astype(np.float32), spec.ngrid, p0, dA, dB, dC,
                              spec.tipQs, spec.tipQZs)
        P = spec.scan_params(k)
        P.flags = b.scan_params.flags
        FEs, PPs = gpu.relax_pp(grid, P, torch.as_tensor(spec.points, device="cuda"))
        inside = ~torch.isnan(b.fes(i)).any(-1)  # a probe that leaves its slab stops there
        assert inside.float().mean() > 0.5
        assert torch.equal(b.fes(i)[inside], FEs[inside]) and torch.equal(b.pps(i)[inside], PPs[inside]), i
