"""The bench's cone rooflines describe the kernels that the timed steps launch."""
from types import SimpleNamespace

import pytest
import torch

import bench
from jscc_recon_spect_cylinder_gb300 import _compton, _lib, synthetic


def test_flops_weighted_by_the_pairs_of_each_kernel():
    one = {k: bench.cone_flop_per_pair((k,))[0] for k in ("cone_forward_pair", "cone_back_pair", "cone_rows_pair")}
    pairs = {"cone_forward_pair": 1.0, "cone_back_pair": 1.0, "cone_rows_pair": 6.0}
    want = sum(one[k] * n for k, n in pairs.items()) / 8
    assert bench.cone_flop_per_pair(pairs)[0] == pytest.approx(want)
    assert bench.cone_flop_per_pair({**pairs, "cone_rows_pair": 0.0})[0] == pytest.approx(
        bench.cone_flop_per_pair(("cone_forward_pair", "cone_back_pair"))[0])


@pytest.mark.gpu
def test_map_cone_pass_is_the_steps():
    grid = synthetic.polar_grid(20, 60, 100.0, device="cuda")
    scat = synthetic.cylinder_pixels(120.0, 64, 4, 2.0, device="cuda")
    absb = synthetic.cylinder_pixels(150.0, 64, 4, 2.0, device="cuda")
    n = scat.size(0)
    i1, i2 = (torch.randint(n, (500,), device="cuda") for _ in range(2))
    e1 = 0.06 + 0.4 * torch.rand(500, device="cuda")
    lst = torch.stack((i1 + 1.0, e1, i2 + 1.0 + n, 0.662 - e1), dim=1)
    _, rec, rid = _compton.select_events(lst, torch.cat((scat, absb)).float(), 1.0, 1.0, 0.662, 0.08, 0.47, 0.05, 0.6)

    class Events(SimpleNamespace):
        def __len__(self):
            return self.records.size(0)

    case = SimpleNamespace(V=grid.n_vox, dev=torch.device("cuda", 0), coor=grid.coor.contiguous(),
                           eff=torch.rand((n, grid.n_vox), device="cuda") + 0.1,
                           ev=Events(records=rec, row_id=rid, model=_lib.CONE_STRICT))
    _lib.kernel_timing_collect()
    _lib.kernel_timing_enable(True)
    out = bench.Map5Bench.extra(case, 1.0)
    _lib.kernel_timing_enable(False)
    ran = _lib.kernel_timing_collect()
    assert "cone_rows_pair" in ran and not {"cone_forward", "cone_back"} & set(ran)
    assert out["fp32_roofline"]["flop_per_pair"] == bench.cone_flop_per_pair(("cone_rows_pair",))[0]
    assert out["cone_pass"]["pairs_per_s"] * out["cone_pass"]["ms"] / 1e3 == pytest.approx(len(rec) * grid.n_vox)
