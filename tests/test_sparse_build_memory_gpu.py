"""The sparse builder on a list whose events are mostly dropped: rows are held for the kept events and one
block of candidates at a time, not for every candidate; the rows equal those of one block."""
import pytest
import torch

import jscc_recon_spect_cylinder_gb300.process_list_plane_sparse as psp
from jscc_recon_spect_cylinder_gb300 import compton_sparse_ops as cso, synthetic

pytestmark = pytest.mark.gpu
ARGS = (1.0, 1.0, 0.662, 0.08, 0.47, 0.05, 0.60)


def _list(n_ev, grid):
    g = torch.Generator(device="cuda").manual_seed(n_ev)
    scat = synthetic.cylinder_pixels(120.0, 64, 4, 2.0, device="cuda")
    absb = synthetic.cylinder_pixels(150.0, 64, 4, 2.0, device="cuda")
    n = scat.size(0)
    i1, i2 = (torch.randint(n, (n_ev,), generator=g, device="cuda") for _ in range(2))
    e1 = 0.06 + 0.4 * torch.rand(n_ev, generator=g, device="cuda")
    lst = torch.stack((i1 + 1.0, e1, i2 + 1.0 + n, 0.662 - e1), dim=1)
    A = (torch.rand((n, grid.n_vox), generator=g, device="cuda") + 0.01) * 1e-4
    return lst, A, torch.cat((scat, absb)).float()


def test_dropped_events_hold_no_rows():
    grid = synthetic.polar_grid(100, 360, 100.0)
    lst, A, det = _list(400_000, grid)
    A[4:] = 0.0  # events whose first hit lies elsewhere have no product with the cone
    proj = cso.build_compton_sparse_projector(grid.coor, 4, 1, rotate_num=1).to("cuda")
    rows = psp.build_sparse_rows_from_smeared(A, det, proj, lst[:1000], *ARGS)  # tables
    del rows
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    rows = psp.build_sparse_rows_from_smeared(A, det, proj, lst, *ARGS)
    peak = torch.cuda.max_memory_allocated() - before
    size = rows.numel() * 4
    assert 0 < rows.size(0) < 20_000
    # kept rows, twice while blocks are joined, a block of candidates; every candidate's row: over 5 GB
    assert peak < 2 * size + (3 << 30)


@pytest.mark.parametrize("block", [1, 7, 300, 10_000])
def test_blocks_join(monkeypatch, block):
    grid = synthetic.polar_grid(25, 80, 100.0)
    lst, A, det = _list(700, grid)
    proj = cso.build_compton_sparse_projector(grid.coor, 2, 1, rotate_num=1).to("cuda")
    A[::5] = 0.0
    ref = psp.build_sparse_rows_from_smeared(A, det, proj, lst, *ARGS)
    monkeypatch.setattr(psp, "BUILD_BLOCK_BYTES", block * (proj.coarse_pixel_num + 1) * 4)
    assert ref.size(0) > 0 and torch.equal(psp.build_sparse_rows_from_smeared(A, det, proj, lst, *ARGS), ref)
