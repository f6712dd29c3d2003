"""One view at exactly the two-pass kernels' workspace, the documented minimum: the weight of many short
rows and the projector's halves of rows off 16-byte boundaries, against a float64 product; and the
allocation-free entry near its 16 MiB.

Tolerance: positive terms, the one-view kernels' longest float32 chain (1,216 chunks of 300 rows, or 1,126
columns a lane): 1e-5 with errors of random sign, as for the other SC routes."""
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _two_pass_bytes(rows, V):
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32
    ldx, tiles = (V + 7) // 8 * 8, max(1, -(-V // 1024))
    chunks = max(1, min(-(-1216 // tiles), -(-rows // 16)))
    chunks = -(-rows // -(-rows // chunks))
    parts = (warps * (-(-rows // warps) + 2), ldx, rows, chunks * ldx)
    return sum((4 * n + 255) // 256 * 256 for n in parts) + 256


def _rel(got, ref):
    return float((got.double().reshape(ref.shape) - ref).norm() / ref.norm())


@pytest.mark.parametrize("rows,V,pitch,first", [
    (10, 36001, 36001, 0), (10, 36000, 36002, 1), (400_000, 100, 100, 0), (300_000, 99, 99, 0), (70_000, 1200, 1200, 0)])
def test_two_pass_workspace(rows, V, pitch, first):
    g = torch.Generator(device="cuda").manual_seed(V)
    A = (torch.rand(rows * pitch + first, generator=g, device="cuda") + 0.05)[first:].view(rows, pitch)[:, :V]
    y = torch.rand((rows, 1), generator=g, device="cuda") + 0.5
    x = torch.rand((V, 1), generator=g, device="cuda") + 0.2
    f = A.double() @ x.double()
    lib, st = _lib.load(), _lib.stream_handle(A.device)
    nbytes = _two_pass_bytes(rows, V)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    w, u, p = (torch.zeros((n, 1), device="cuda") for n in (V, V, rows))
    a = (A.data_ptr(), 0, A.stride(0), None, rows, V)
    rc = lib.jscc_sc_weight(*a, y.data_ptr(), 1, 1, x.data_ptr(), None, None, 0, 0, 0.0, 1.0, w.data_ptr(),
                            ws.data_ptr(), nbytes, st)
    assert rc == 0, lib.jscc_last_error()
    rc = lib.jscc_sc_project(*a, 1, x.data_ptr(), None, 0, p.data_ptr(), 1, ws.data_ptr(), nbytes, st)
    assert rc == 0, lib.jscc_last_error()
    rc = lib.jscc_sc_backproject(*a, 1, y.data_ptr(), 1, None, 0, 1.0, u.data_ptr(), ws.data_ptr(), nbytes, st)
    assert rc == 0, lib.jscc_last_error()
    assert _rel(w, A.double().t() @ (y.double() / f)) < TOL
    assert _rel(p, f) < TOL
    assert _rel(u, A.double().t() @ y.double()) < TOL
    assert lib.jscc_sc_project(*a, 1, x.data_ptr(), None, 0, p.data_ptr(), 1, ws.data_ptr(), nbytes - 256, st) != 0


@pytest.mark.parametrize("rows,V", [(1_900_000, 100), (1_600_000, 1200)])
def test_noalloc_of_many_short_rows(rows, V):
    A = torch.rand((rows, V), device="cuda") + 0.05
    y = torch.rand((rows, 1), device="cuda") + 0.5
    x = torch.rand((V, 1), device="cuda") + 0.2
    w = torch.zeros((V, 1), device="cuda")
    lib = _lib.load()
    rc = lib.jscc_sc_weight_noalloc(A.data_ptr(), 0, V, None, rows, V, y.data_ptr(), 1, 1, x.data_ptr(), None, None, 0,
                                    0, 0.0, 1.0, w.data_ptr(), _lib.stream_handle(A.device))
    assert rc == 0, lib.jscc_last_error()
    ref = torch.zeros((V, 1), dtype=torch.float64, device="cuda")
    for a in range(0, rows, 100_000):
        Ad = A[a:a + 100_000].double()
        ref += Ad.t() @ (y[a:a + 100_000].double() / (Ad @ x.double()))
    assert _rel(w, ref) < TOL
