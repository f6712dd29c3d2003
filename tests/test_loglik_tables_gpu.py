"""poisson_log_likelihood with rotation tables of different row pitches (a column slice of a wider table
beside a contiguous one): the same value and gradient as with contiguous tables."""
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import autograd as ag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 3])
@pytest.mark.parametrize("wide", ["rot", "inv", "both"])
def test_pitches(R, wide):
    V, rows, g = 203, 40, torch.Generator(device="cuda").manual_seed(R)
    A = torch.rand((rows, V), generator=g, device="cuda") + 0.05
    y = torch.poisson(torch.full((rows, R), 3.0, device="cuda"), generator=g)
    rot = torch.stack([torch.randperm(V, generator=g, device="cuda") for _ in range(R)], dim=1)
    inv = torch.argsort(rot, dim=0) + 1
    rot += 1
    x = torch.rand((V, 1), generator=g, device="cuda") + 0.3
    got = []
    for sliced in (False, True):
        a, b = rot, inv
        if sliced and wide != "inv":
            a = torch.cat((rot, rot), dim=1)[:, :R]
        if sliced and wide != "rot":
            b = torch.cat((inv, inv, inv), dim=1)[:, :R]
        xg = x.clone().requires_grad_(True)
        ll = ag.poisson_log_likelihood(xg, sc=(A, y, a, b))
        ll.backward()
        got.append((ll.detach(), xg.grad))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
