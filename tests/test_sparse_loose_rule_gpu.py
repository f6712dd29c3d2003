"""Which kernel takes packed rows of many events: the bulk pipeline from a number of coarse voxels and taps on,
the general kernel below, each against the float64 oracle on both sides of the line.

Tolerance: positive terms, no float32 chain of more than about 300 (a thread's columns, shuffles, warps; a
group's events; groups of a chunk and chunks): 2e-5, as for the other grouped weights."""
import numpy as np
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib, compton_sparse_ops as cso, ops, synthetic
from oracle import sparse as osp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,n_theta,stride,n_ev,n_det,bulk", [
    (22, 92, 4, 250, 40, False), (22, 92, 4, 199, 40, True),        # 506 coarse voxels, 7 taps
    (46, 144, 4, 250, 40, False), (47, 144, 4, 250, 40, True),      # 1,656 and 1,692: 7 taps, 12 to each
    (33, 90, 2, 300, 30, False), (60, 90, 2, 260, 9, True)])        # 3 taps
@pytest.mark.parametrize("grouped", [False, True])
def test_either_side_of_the_line(n_r, n_theta, stride, n_ev, n_det, bulk, grouped):
    grid = synthetic.polar_grid(n_r, n_theta, 30.0)
    proj = cso.build_compton_sparse_projector(grid.coor, stride, 1, rotate_num=1)
    g = torch.Generator().manual_seed(n_r + n_ev)
    A = (torch.rand((n_det, grid.n_vox), generator=g) + 0.05) * 1e-3
    tc = torch.rand((n_ev, proj.coarse_pixel_num), generator=g) ** 3 + 1e-3
    ids = torch.randint(0, n_det, (n_ev,), generator=g, dtype=torch.int32)
    x = torch.rand((grid.n_vox, 1), generator=g) + 0.2
    rows = torch.cat(((ids + 1).float().unsqueeze(1), tc), dim=1)
    tables = cso.tables(proj, "cuda")
    _lib.kernel_timing_collect()
    _lib.kernel_timing_enable(True)
    w = ops.sparse_weight(rows.cuda(), A.cuda(), tables, x.cuda(), grouped=grouped)
    _lib.kernel_timing_enable(False)
    assert ("sparse_group_adjoint" in _lib.kernel_timing_collect()) == bulk
    assert _lib.take_wait_timeout_count() == 0
    op = osp.build_projector(grid.coor.numpy(), theta_stride=stride, z_stride=1, rotate_num=1)
    ref = np.asarray((osp.weight_grouped if grouped else osp.weight_materialize)(rows.numpy(), A.numpy(), x.numpy(), op))
    got = w.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got.ravel() - ref.ravel()) / np.linalg.norm(ref) < 2e-5
