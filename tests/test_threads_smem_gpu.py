"""Calls of different sizes from several threads at once, each on its own stream: a launch must not find
its kernel's shared-memory limit lowered by another thread's smaller call. The library's entries are
called back to back, so that the threads are inside them at the same time."""
import threading

import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _compton, _lib, compton_sparse_ops as cso, ops, synthetic

pytestmark = pytest.mark.gpu


class _Recorder:
    """The library, with the last call's function and arguments kept."""

    def __init__(self, lib):
        self._real = lib

    def __getattr__(self, name):
        fn = getattr(self._real, name)

        def call(*a):
            self.last = (fn, a)
            return fn(*a)

        return call


def _weight(V, rows, R):
    A = torch.rand((rows, V), device="cuda") + 0.05
    y = torch.rand((rows, R), device="cuda") + 0.5
    x = torch.rand((V, 1), device="cuda") + 0.2
    out = torch.zeros((V, 1), device="cuda")
    rot = torch.stack([torch.roll(torch.arange(V, device="cuda"), r + 1) + 1 for r in range(R)], dim=1)
    inv = torch.stack([torch.roll(torch.arange(V, device="cuda"), -r - 1) + 1 for r in range(R)], dim=1)
    return lambda: ops.sc_weight(A, y, x, rot, inv, out=out)


def _project(V, rows):
    x = torch.rand((V, 1), device="cuda") + 0.2
    A = torch.rand((rows, V), device="cuda") + 0.05
    return lambda: ops.sc_project(A, x)


def _build(n_r, n_theta):
    grid = synthetic.polar_grid(n_r, n_theta, 100.0)
    scat = synthetic.cylinder_pixels(120.0, 64, 4, 2.0, device="cuda")
    absb = synthetic.cylinder_pixels(150.0, 64, 4, 2.0, device="cuda")
    n = scat.size(0)
    i1, i2 = (torch.randint(n, (200,), device="cuda") for _ in range(2))
    e1 = 0.06 + 0.4 * torch.rand(200, device="cuda")
    lst = torch.stack((i1 + 1.0, e1, i2 + 1.0 + n, 0.662 - e1), dim=1)
    _, rec, rid = _compton.select_events(lst, torch.cat((scat, absb)).float(), 1.0, 1.0, 0.662, 0.08, 0.47, 0.05, 0.6)
    A = torch.rand((n, grid.n_vox), device="cuda") + 0.01
    cp = cso.build_compton_sparse_projector(grid.coor, 1, 1, rotate_num=1)
    tb, coor = cso.tables(cp, "cuda"), cp.coor_coarse.to("cuda", torch.float32).contiguous()
    rec, rid = rec[:20].contiguous(), rid[:20].contiguous()
    return lambda: ops.sparse_build_rows(rec, rid, coor, A, tb.red, tb.red_single, cp.coarse_z_num, cp.fine_z_num,
                                         cp.coarse_layer_num, cp.fine_layer_num, 50.0)


@pytest.mark.parametrize("make,sizes", [
    (_weight, [(1000, 19456, 3), (70, 16, 3)]), (_weight, [(1500, 9728, 20), (70, 16, 20)]),
    (_weight, [(36000, 16, 1), (3000, 16, 1)]), (_project, [(36000, 16), (400, 16)]),
    (_build, [(200, 240), (20, 60)])])
def test_two_sizes_at_once(monkeypatch, make, sizes):
    calls = [make(*s) for s in sizes] * 2
    torch.cuda.synchronize()
    start, wrong = threading.Barrier(len(calls)), [None] * len(calls)
    lib = _lib.load()
    stage, kept = [], []
    for call in calls:  # each call's buffers, on a stream of its own
        rec, stream = _Recorder(lib), torch.cuda.Stream()
        monkeypatch.setattr(_lib, "load", lambda rec=rec: rec)
        with torch.cuda.stream(stream):
            kept.append(call())
        stage.append((stream, *rec.last))
    torch.cuda.synchronize()

    def work(k):
        stream, fn, args = stage[k]
        start.wait()
        wrong[k] = sum(fn(*args) != 0 for _ in range(2000))
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0] * len(calls), lib.jscc_last_error()
