"""Scatter of coarse rows with neighbours of very different size (a cone's edge), voxel by voxel: a fine
voxel on a coarse sample, and one between two small samples, next to a value 1e9 times larger.

One group, so that no other group's term hides a voxel's error. All terms positive: the shared factor of
the event (its projection) has float32 chains of at most about 300 terms, a voxel's own interpolation a few
roundings: 2e-5 of each voxel, as for the other grouped weights' norms."""
import numpy as np
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib, compton_sparse_ops as cso, ops, synthetic
from oracle import sparse as osp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,n_theta,radial", [(8, 32, 1), (40, 96, 1), (24, 88, 3), (12, 360, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("grouped", [False, True])
def test_steep_neighbours(n_r, n_theta, radial, dtype, grouped):
    grid = synthetic.polar_grid(n_r, n_theta, 30.0)
    if radial > 1:
        proj, oproj = (cso.build_compton_sparse_projector_radial(grid.coor, radial, 4),
                       osp.build_radial_projector(grid.coor.numpy(), radial, 4))
    else:
        proj, oproj = (cso.build_compton_sparse_projector(grid.coor, 4, 1, rotate_num=1),
                       osp.build_projector(grid.coor.numpy(), theta_stride=4, z_stride=1, rotate_num=1))
    g = torch.Generator().manual_seed(n_r * n_theta)
    V, vc = grid.coor.size(0), proj.coarse_pixel_num
    A = ((torch.rand((3, V), generator=g) + 0.05) * 1e-3).to(dtype)
    size = torch.tensor([1.0, 1e-9, 1e-3, 1e-9, 1e-6])[torch.randint(0, 5, (1, vc), generator=g)]
    tc = (size * (torch.rand((1, vc), generator=g) + 0.5)).to(dtype)
    x = torch.rand((V, 1), generator=g) + 0.2
    rows = torch.cat((torch.full((1, 1), 2.0), tc.float()), dim=1)
    rid, t = ops.split_sparse_rows(rows.cuda(), dtype)
    w = ops.sparse_weight_split(rid, t, A.cuda(), cso.tables(proj, "cuda"), x.cuda(), grouped=grouped)
    assert _lib.take_wait_timeout_count() == 0
    f = osp.weight_grouped if grouped else osp.weight_materialize
    ref = f(rows.numpy(), A.float().numpy(), x.numpy(), oproj).ravel()
    got = w.cpu().numpy().astype(np.float64).ravel()
    assert (ref > 0).all()
    assert np.abs(got / ref - 1).max() < 2e-5
