"""The adjoint's launch shape goes by the items of the launch: a plan with room
for more items than the GPU has SMs runs few items as a plan made for them does,
and gives the same bits."""
import numpy as np
import pytest

from discoeb_gb300 import _native
from discoeb_gb300.gradient import SEG_CAP, GradientProblem, perturbed_params
from discoeb_gb300.workloads import fiducial_mnu_param

pytestmark = pytest.mark.gpu

SIZES = [dict(lmaxg=12, lmaxgp=12, lmaxr=17, lmaxnu=17, nqmax=15), dict(lmaxg=32, lmaxgp=32, lmaxr=32, lmaxnu=32, nqmax=30)]


@pytest.mark.parametrize("dims", SIZES, ids=["323", "1098"])
def test_few_items_on_a_large_plan(dims):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    base = fiducial_mnu_param()
    gp = GradientProblem([base], "native", [perturbed_params(base)], np.geomspace(1e-3, 0.01, 3), [1.0], method="adjoint",
                         rtol=1e-3, atol=1e-3, max_steps=4000, **dims)
    out = {}
    for room in (3, sms, 4 * sms):
        gp.adj_plan = _native.Plan(gp.dims, room, adjoint_seg_cap=SEG_CAP)
        out[room] = gp.adj_plan.launch_info(3), gp.run()[1].cpu().numpy().copy()
        gp.check()
    for room in (sms, 4 * sms):
        assert out[room][0] == out[3][0]
        np.testing.assert_array_equal(out[room][1], out[3][1])
    assert out[3][0]["modes_per_sm"] == 1
    assert gp.adj_plan.launch_info(sms)["modes_per_sm"] == 1 and gp.adj_plan.launch_info(sms + 1)["modes_per_sm"] == 2
    with pytest.raises(RuntimeError):
        gp.adj_plan.launch_info(4 * sms + 1)
