"""The strict Compton weight and likelihood of millions of events on grids of a few voxels (more stages of events
than one dimension of a launch takes).

Tolerance: 43 equal blocks of events, added in float32: 1e-5; projections as one block's, 2e-6."""
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _compton, _lib, ops, synthetic

pytestmark = pytest.mark.gpu


def _events(shape, n_ev, model=_lib.CONE_STRICT, repeat=1):
    grid = synthetic.polar_grid(*shape, 100.0, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(n_ev)
    scat = synthetic.cylinder_pixels(120.0, 64, 4, 2.0, device="cuda")
    absb = synthetic.cylinder_pixels(150.0, 64, 4, 2.0, device="cuda")
    n = scat.size(0)
    e1 = 0.06 + 0.4 * torch.rand(8 * n_ev + 256, generator=g, device="cuda")
    i1, i2 = (torch.randint(n, e1.shape, generator=g, device="cuda") for _ in range(2))
    lst = torch.stack((i1 + 1.0, e1, i2 + 1.0 + n, 0.662 - e1), dim=1)
    _, rec, rid = _compton.select_events(lst, torch.cat((scat, absb)).float(), 1.0, 1.0, 0.662, 0.08, 0.47, 0.05, 0.6,
                                         model=model)
    A = (torch.rand((n, grid.n_vox), generator=g, device="cuda") + 0.05) * 1e-4
    x = torch.rand((grid.n_vox, 1), generator=g, device="cuda") + 0.3
    coor = grid.coor.contiguous()
    if model == _lib.CONE_STRICT:  # events that see the grid, with no voxel on their axis
        f, p = (ops.compton_project(rec, rid, coor, v, eff=A) for v in (x.double(), x))
        seen = (f > 1e-12) & ((p - f).abs() < 1e-3 * f)
        rec, rid = rec[seen], rid[seen]
    rec, rid = rec[:n_ev].repeat(repeat, 1).contiguous(), rid[:n_ev].repeat(repeat).contiguous()
    assert rec.size(0) == n_ev * repeat
    return coor, rec, rid, A, x


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("shape", [(2, 4), (8, 8)])
def test_millions_of_events_on_a_small_grid(shape):
    coor, rec, rid, A, x = _events(shape, 100_000 // 43, repeat=43)
    part = rec.size(0) // 43
    one = ops.compton_weight(rec[:part], rid[:part], coor, x, eff=A)
    f1, g1 = ops.compton_loglik(rec[:part], rid[:part], coor, x, eff=A)
    rec, rid = rec.repeat(43, 1), rid.repeat(43)
    assert rec.size(0) > 64 * 65535
    times = rec.size(0) // part
    assert _rel(ops.compton_weight(rec, rid, coor, x, eff=A), one * times) < 1e-5
    f, grad = ops.compton_loglik(rec, rid, coor, x, eff=A)
    assert _rel(grad, g1 * times) < 1e-5
    assert _rel(f.sort().values, f1.repeat(times).sort().values) < 2e-6
