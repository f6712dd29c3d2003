"""Two rotated views of float32 matrices past the size from which the one-view forward kernel takes both
images, against a float64 product: odd column counts, padded pitches, row ids, the stored projections and
the likelihood, and less workspace than it needs (the kernels of several views then run).

Tolerance: positive terms, float32 chains of at most 1,200 / 32 x 4 columns a lane and 100 rows, then trees: a few
hundred roundings of random sign, 1e-5 as for the other SC routes; the likelihood's gradient relative to the
sum of its positive and its negative part."""
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib, ops

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _rel(got, ref):
    return float((got.double().reshape(ref.shape) - ref).norm() / ref.norm())


@pytest.mark.parametrize("V,rows,pitch,split", [
    (4800, 5200, 4800, True), (25600, 950, 25600, True), (1001, 24000, 1004, True), (70, 350_000, 72, True),
    (25601, 950, 25604, False), (4800, 4900, 4800, False), (4801, 5200, 4801, False)])
def test_two_views(V, rows, pitch, split):
    g = torch.Generator(device="cuda").manual_seed(rows)
    A = (torch.rand((rows, pitch), generator=g, device="cuda") + 0.05)[:, :V]
    y = torch.rand((rows, 2), generator=g, device="cuda") + 0.5
    x = torch.rand((V, 1), generator=g, device="cuda") + 0.2
    rot = torch.stack([torch.randperm(V, generator=g, device="cuda") for _ in range(2)], dim=1)
    inv = torch.argsort(rot, dim=0) + 1
    rot += 1
    f = torch.cat([A.double() @ x.double()[rot[:, r] - 1] for r in range(2)], dim=1)
    back = lambda q: sum((A.double().t() @ q[:, r])[inv[:, r] - 1] for r in range(2))  # noqa: E731
    ref = back(y.double() / f)
    _lib.kernel_timing_collect()
    _lib.kernel_timing_enable(True)
    out = ops.sc_weight(A, y, x, rot, inv, scale=0.5, out=torch.ones((V, 1), device="cuda"))
    _lib.kernel_timing_enable(False)
    assert ("sc_forward_split" in _lib.kernel_timing_collect()) == split
    assert _rel(out, 1 + 0.5 * ref) < TOL
    assert torch.equal(out, ops.sc_weight(A, y, x, rot, inv, scale=0.5, out=torch.ones((V, 1), device="cuda")))
    assert _rel(ops.sc_project(A, x, rot), f) < TOL
    got, grad = ops.sc_loglik(A, y, x, rot, inv, eps=1e-9)
    ones = back(torch.ones_like(f))
    assert _rel(got, f) < TOL
    assert float((grad[:, 0].double() - (ref - ones)).norm() / (ref + ones).norm()) < TOL
    ids = torch.randperm(rows, generator=g, device="cuda")
    assert _rel(ops.sc_weight(A, y, x, rot, inv, row_idx=ids), ref) < TOL
    lib = _lib.load()
    full = lib.jscc_sc_weight_workspace_bytes(rows, V, 2)
    tried = 0
    for nbytes in (full, full * 3 // 4, full // 2, full // 4):
        ws, out = torch.empty(nbytes, dtype=torch.uint8, device="cuda"), torch.zeros((V, 1), device="cuda")
        rc = lib.jscc_sc_weight(A.data_ptr(), 0, A.stride(0), None, rows, V, y.data_ptr(), 2, 2, x.data_ptr(),
                                rot.data_ptr(), inv.data_ptr(), 2, 0, 0.0, 1.0, out.data_ptr(), ws.data_ptr(), nbytes,
                                _lib.stream_handle(A.device))
        if rc == 0:
            tried += 1
            assert _rel(out, ref) < TOL
    assert tried >= 1
