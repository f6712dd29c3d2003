"""The adjoint over several planes of a ring stencil on both sides of the number of groups from which it is
taken (groups times coarse voxels against 250,000), and the gathered taps below, against the float64 oracle.

Tolerance: positive terms, no float32 chain of more than about 300 (56 taps, a thread's columns, a group's
events, groups of a chunk and chunks): 2e-5, as for the other grouped weights."""
import numpy as np
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib, compton_sparse_ops as cso, ops, synthetic
from oracle import sparse as osp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,n_theta,radial,groups", [
    (64, 120, 4, 520), (64, 120, 4, 521), (24, 88, 3, 1450), (12, 2048, 4, 162), (12, 2048, 4, 163), (48, 360, 4, 240)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("grouped", [False, True])
def test_groups(n_r, n_theta, radial, groups, dtype, grouped):
    grid = synthetic.polar_grid(n_r, n_theta, 30.0)
    proj = cso.build_compton_sparse_projector_radial(grid.coor, radial, 4)
    oproj = osp.build_radial_projector(grid.coor.numpy(), radial, 4)
    g = torch.Generator().manual_seed(groups)
    n_ev, vc = groups + 61, proj.coarse_pixel_num
    A = ((torch.rand((groups + 3, grid.n_vox), generator=g) + 0.05) * 1e-3).to(dtype)
    tc = (torch.rand((n_ev, vc), generator=g) ** 3 + 1e-3).to(dtype)
    ids = torch.cat((torch.arange(groups), torch.randint(0, groups, (61,), generator=g)))[torch.randperm(n_ev, generator=g)]
    x = torch.rand((grid.n_vox, 1), generator=g) + 0.2
    rows = torch.cat(((ids + 1).float().unsqueeze(1), tc.float()), dim=1)
    rid, t = ops.split_sparse_rows(rows.cuda(), dtype)
    w = ops.sparse_weight_split(rid, t, A.cuda(), cso.tables(proj, "cuda"), x.cuda(), grouped=grouped)
    assert _lib.take_wait_timeout_count() == 0
    f = osp.weight_grouped if grouped else osp.weight_materialize
    ref = np.asarray(f(rows.numpy(), A.float().numpy(), x.numpy(), oproj)).ravel()
    got = w.cpu().numpy().astype(np.float64).ravel()
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 2e-5
