"""Infinite image values in the SC projector of several views: a projection is infinite where one of its
terms is, as in plain arithmetic, and no other lane's columns turn it into NaN. Column counts that leave
lanes of the last columns idle, infinite values at the start and the end of the grid."""
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V,rows,R,first", [(1003, 40, 3, 0), (70, 300, 2, 1), (6017, 9, 5, 0), (33, 3, 20, 0)])
@pytest.mark.parametrize("at", [0, -1])
def test_infinite_voxel(dtype, V, rows, R, first, at):
    g = torch.Generator(device="cuda").manual_seed(V)
    A = (torch.rand(rows * V + first, generator=g, device="cuda") + 0.05).to(dtype)[first:].view(rows, V)
    x = torch.rand((V, 1), generator=g, device="cuda") + 0.2
    x[at] = float("inf")
    tab = torch.arange(1, V + 1, device="cuda").unsqueeze(1).expand(V, R).contiguous()
    f = ops.sc_project(A, x, tab)
    assert torch.equal(f, torch.full_like(f, float("inf")))
    w = ops.sc_weight(A, torch.ones((rows, R), device="cuda"), x, tab, tab)
    assert torch.equal(w, torch.zeros_like(w))  # y / inf
