"""A second derivative through the one-pass likelihood terms is refused: their gradient is a saved
vector, and following the incoming factor alone would drop the likelihood's own Hessian without a word."""
from __future__ import annotations

import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import autograd as ag, ops


def _sc(monkeypatch):
    A = torch.rand((5, 3), generator=torch.Generator().manual_seed(1)) + 0.1
    y = torch.tensor([[2.0], [0.0], [1.0], [3.0], [1.0]])

    def loglik(sysmat, proj, img, rotmat, rotmat_inv, eps):
        f = sysmat @ img
        return f, sysmat.t() @ (proj / f - 1)

    monkeypatch.setattr(ops, "sc_loglik", loglik)
    return lambda x: ag.SCLogLik.apply(x, A, y, None, None, 0.0)


def _compton(monkeypatch):
    T = torch.rand((5, 3), generator=torch.Generator().manual_seed(2)) + 0.1
    return lambda x: ag.ComptonLogLik.apply(x, (T @ x.detach()).reshape(-1), T.t() @ (1 / (T @ x.detach())), 0.0)


@pytest.mark.parametrize("term", [_sc, _compton])
def test_second_derivative_is_refused(monkeypatch, term):
    ll = term(monkeypatch)
    x = (torch.rand((3, 1), generator=torch.Generator().manual_seed(3)) + 0.5).requires_grad_(True)
    (first,) = torch.autograd.grad(ll(x) ** 2, x)
    (again,) = torch.autograd.grad(ll(x) ** 2, x, create_graph=True)
    assert torch.equal(first, again.detach())  # a graph for the first derivative alone costs nothing
    with pytest.raises(RuntimeError):
        torch.autograd.grad(again.sum(), x)
