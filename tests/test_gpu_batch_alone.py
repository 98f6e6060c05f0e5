"""A molecule's forward and gradients are the same bits alone and among others: nothing is chosen by what else
the batch holds."""
import numpy as np
import pytest
import torch

from spammm_b200 import _lib, synthetic
from spammm_b200.batch import AFMBatch

pytestmark = pytest.mark.gpu


def _run(items, targets, kind, chunk):
    shape = _lib.BatchShape(*_lib.lib().spm_batch_default_shape().key())
    shape.adj_chunk = chunk
    b = AFMBatch(items, kind=kind, shape=shape)
    for i, t in enumerate(targets):
        b.set_target(i, t)
    b.forward_adjoint()
    torch.cuda.synchronize()
    return b


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("chunk", [1024, 16384])
def test_gradients_do_not_depend_on_the_rest_of_the_batch(cuda, kind, chunk):
    items = []
    for k, na in enumerate((20, 40, 64, 90, 120, 200, 270)):
        items += synthetic.batch_molecules(1, seed=7 + k, kind=kind, natoms=(na, na), side=(9, 11), zside=(9, 11),
                                           npx=(20 + k, 20 + k), nzs=(10 + k, 10 + k))
    rng = np.random.default_rng(1)
    targets = [rng.normal(0.0, 0.05, (len(it.xs), len(it.ys), it.nz)) for it in items]
    b = _run(items, targets, kind, chunk)
    for i, it in enumerate(items):
        one = _run([it], [targets[i]], kind, chunk)
        assert torch.equal(b.fes(i), one.fes(0)) and torch.equal(b.loss_of(i), one.loss_of(0)), i
        assert torch.equal(b.grad_of(i), one.grad_of(0)), i
