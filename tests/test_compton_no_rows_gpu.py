"""Compton calls without efficiency rows and without row ids (the C entries take NULL for both), against the
same calls with row ids: the ids are not read."""
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _compton, _lib, ops, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [_lib.CONE_STRICT, _lib.CONE_LEGACY, _lib.CONE_SIMPLE])
@pytest.mark.parametrize("window", [0, 1])
@pytest.mark.parametrize("preferred", [0, 1])
def test_null_row_ids(model, window, preferred):
    grid = synthetic.polar_grid(20, 60, 100.0, device="cuda")
    scat = synthetic.cylinder_pixels(120.0, 64, 4, 2.0, device="cuda")
    absb = synthetic.cylinder_pixels(150.0, 64, 4, 2.0, device="cuda")
    n, g = scat.size(0), torch.Generator(device="cuda").manual_seed(5)
    i1, i2 = (torch.randint(n, (500,), generator=g, device="cuda") for _ in range(2))
    e1 = 0.06 + 0.4 * torch.rand(500, generator=g, device="cuda")
    lst = torch.stack((i1 + 1.0, e1, i2 + 1.0 + n, 0.662 - e1), dim=1)
    _, rec, rid = _compton.select_events(lst, torch.cat((scat, absb)).float(), 1.0, 1.0, 0.662, 0.08, 0.47, 0.05, 0.6,
                                         model=model)
    coor, V, E = grid.coor.contiguous(), grid.n_vox, rec.size(0)
    assert E > 100
    x = torch.rand((V, 1), generator=g, device="cuda") + 0.3
    q = torch.rand(E, generator=g, device="cuda")
    lib, st = _lib.load(), _lib.stream_handle(x.device)
    got = []
    for ids in (rid.data_ptr(), None):
        f, w, u = torch.zeros(E, device="cuda"), torch.zeros(V, device="cuda"), torch.zeros(V, device="cuda")
        ws = [torch.empty(lib.jscc_compton_workspace_bytes(E, V, call, model, window, preferred), dtype=torch.uint8,
                          device="cuda") for call in range(3)]
        a = (rec.data_ptr(), ids, E, coor.data_ptr(), V, model, window, None, 0, 0)
        _lib.check(lib.jscc_compton_weight(*a, x.data_ptr(), None, None, 0, 1.0, w.data_ptr(), ws[0].data_ptr(),
                                           ws[0].numel(), st), "weight")
        _lib.check(lib.jscc_compton_project(*a, x.data_ptr(), None, 0, f.data_ptr(), ws[1].data_ptr(), ws[1].numel(),
                                            st), "project")
        _lib.check(lib.jscc_compton_backproject(*a, q.data_ptr(), None, 0, 1.0, u.data_ptr(), ws[2].data_ptr(),
                                                ws[2].numel(), st), "backproject")
        got.append((w, f, u))
    for a, b in zip(*got):
        assert torch.equal(a.nan_to_num(), b.nan_to_num())
    assert float(got[0][1].sum()) > 0
