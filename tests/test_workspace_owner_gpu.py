"""Captured batches own their scratch: two of them replayed at once on two streams give what each gives alone
(bit for bit, all sums have a fixed order), and a batch that is dropped leaves no scratch behind."""
import gc

import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib
from jscc_recon_spect_cylinder_gb300.batched import BatchedScOsem

pytestmark = pytest.mark.gpu


def _batch(V, bins, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = (torch.rand((bins, V), generator=g, device="cuda") + 0.05).to(torch.bfloat16)
    perm = torch.randperm(bins, generator=torch.Generator().manual_seed(seed))
    b = BatchedScOsem(A, list(perm.chunk(2)), A.float().sum(0), n)
    b.set_projections(torch.rand((n, bins), generator=g, device="cuda") + 0.5)
    b.splits = {(k, blk[2]): 4 for k in "fb" for blk in b.blocks}  # K splits: partial products in the scratch
    x = torch.rand((n, V), generator=g, device="cuda") + 0.2
    b.set_images(x)
    b.capture()
    return b, x


def test_two_graphs_at_once():
    made = [_batch(4096, 2048, 16, 1), _batch(7200, 3000, 40, 2)]
    alone = []
    for b, x in made:
        b.set_images(x)
        alone.append(b.iterate(30).clone())
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in made]
    for (b, x), s in zip(made, streams):
        with torch.cuda.stream(s):
            b.set_images(x)
    torch.cuda.synchronize()
    for _ in range(30):
        for (b, _), s in zip(made, streams):
            with torch.cuda.stream(s):
                b.iterate()
    torch.cuda.synchronize()
    for (b, _), ref in zip(made, alone):
        assert torch.equal(b.X, ref)


def test_dropped_batch_leaves_nothing():
    _batch(1024, 256, 8, 3)  # the eager call's buffer of this stream, at its largest below
    del_b, _ = _batch(4096, 2048, 16, 4)
    del del_b, _
    gc.collect()
    _lib.workspace.clear()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    for seed in range(4):
        b, x = _batch(4096 + 1024 * seed, 2048, 16, seed)
        b.iterate()
    del b, x
    gc.collect()
    torch.cuda.synchronize()
    assert not _lib.workspace._kept
    _lib.workspace.clear()
    assert torch.cuda.memory_allocated() <= before
