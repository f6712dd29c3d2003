"""Scratch of the Compton passes: only what stores rows holds room for them, a call whose preferred scratch
cannot be had runs in less.

Tolerance: the routes evaluate the same float32 values and differ in the order of their sums: 2e-6 as for the
stored rows."""
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


@pytest.mark.parametrize("call", ["backproject", "project", "window", "legacy", "simple", "legacy_project"])
def test_no_room_for_rows_that_are_not_stored(call):
    model = {"legacy": _lib.CONE_LEGACY, "legacy_project": _lib.CONE_LEGACY, "simple": _lib.CONE_SIMPLE}.get(
        call, _lib.CONE_STRICT)
    coor, rec, rid, A, x = _events((100, 360), 2000, model)
    g = torch.rand(rec.size(0), device="cuda")
    run = {"backproject": lambda: ops.compton_backproject(rec, rid, coor, g, eff=A),
           "project": lambda: ops.compton_project(rec, rid, coor, x, eff=A),
           "legacy_project": lambda: ops.compton_project(rec, rid, coor, x, model=model, eff=A),
           "window": lambda: ops.compton_weight(rec, rid, coor, x, eff=A, use_window=True)}.get(
               call, lambda: ops.compton_weight(rec, rid, coor, x, model=model, eff=A))
    _lib.workspace.clear()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    run()
    # the rows alone are 288 MB; the back pass's partial images and the projection's slices take a few
    assert torch.cuda.max_memory_allocated() - before < 32 << 20


def test_less_scratch_where_memory_is_short():
    coor, rec, rid, A, x = _events((100, 360), 6000)
    ref = ops.compton_weight(rec, rid, coor, x, eff=A)
    g_ref = ops.compton_loglik(rec, rid, coor, x, eff=A)[1]
    _lib.workspace.clear()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (200 << 20)) / total)  # rows: 864 MB
    try:
        got = [ops.compton_weight(rec, rid, coor, x, eff=A) for _ in range(2)]
        assert ops.compton_loglik(rec, rid, coor, x, eff=A) is None  # the projector pair takes over
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        _lib.workspace.clear()
    assert torch.equal(got[0], got[1]) and _rel(got[0], ref) < 2e-6
    assert torch.equal(ops.compton_weight(rec, rid, coor, x, eff=A), ref)
    assert torch.equal(ops.compton_loglik(rec, rid, coor, x, eff=A)[1], g_ref)
