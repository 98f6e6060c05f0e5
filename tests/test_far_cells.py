"""spm_batch_prepare's prefix of far-field lattice cells (block_off), on the CPU."""
import ctypes

import numpy as np
import pytest

from spammm_b200 import _lib
from spammm_b200.batch import BatchItem, BatchPlan


def _item(na, n, x0, npx, z_top):
    xs = (x0 + 0.1 * np.arange(npx)).astype(np.float32)
    return BatchItem(atoms=np.zeros((na, 4), np.float32), params=np.ones((na, 2), np.float32),
                     origin=np.array([-0.05 * n[0], -0.05 * n[1], -4.0]), step=0.1, ngrid=n, xs=xs, ys=xs[:7].copy(),
                     z_top=z_top, nz=12)


@pytest.mark.parametrize("nas", [(31, 32), (255, 256, 10), (600, 40, 33, 256)])
def test_block_prefix_covers_each_box(nas):
    items = [_item(na, (150 + 7 * i, 131, 120 + i), -1.0 + 0.37 * i, 20 + i, 5.0 - 0.2 * i) for i, na in enumerate(nas)]
    plan = BatchPlan(items)
    plan.prepare(_lib.lib().spm_batch_default_shape())
    at = 0
    for j in range(plan.n):
        D = plan.mols[j]
        assert D.block_off == at
        if D.n_atoms < 256:
            continue
        cells = 1
        for lo, n in ((D.x_lo, D.nx_slab), (D.y_lo, D.ny_slab), (D.z_lo, D.nz_slab)):
            cells *= len({i // 32 for i in range(lo, lo + n)})
        at += cells
    assert ctypes.sizeof(_lib.BatchMol) % 8 == 0


@pytest.mark.parametrize("na,n,step,far", [(300, (40, 15, 64), 0.1, False), (300, (40, 16, 64), 0.1, True),
                                           (511, (15, 40, 64), 0.1, False), (512, (15, 15, 64), 0.1, True),
                                           (600, (40, 40, 40), 0.5, True), (600, (40, 40, 40), 0.55, False),
                                           (255, (64, 64, 64), 0.1, False), (256, (64, 64, 64), 0.1, True)])
def test_which_grids_take_blocks(na, n, step, far):
    xs = (np.arange(4) * step).astype(np.float32)
    plan = BatchPlan([BatchItem(atoms=np.zeros((k, 4), np.float32), params=np.ones((k, 2), np.float32),
                                origin=np.array([-1.5 * step, -1.5 * step, 0.0]), step=step, ngrid=n, xs=xs, ys=xs,
                                z_top=step * 30, nz=2) for k in (na, 4)])
    plan.prepare(_lib.lib().spm_batch_default_shape())
    assert (plan.mols[1].block_off > 0) == far
