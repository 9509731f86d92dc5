"""Every mode of a launch is solved once, whatever the number of modes per SM.

Modes do not depend on one another, so the outputs have the same bits when the
queue hands them out in the opposite order.
"""
import numpy as np
import pytest
import torch

from discoeb_gb300 import perturbations as pt
from discoeb_gb300 import tables as tb
from discoeb_gb300.background import evolve_background
from discoeb_gb300.workloads import lcdm_massless_param

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm, extra", [(0, 1), (1, -1), (1, 0), (1, 1), (5, 3)])
def test_queue_hands_out_every_mode_once(per_sm, extra):
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    p = evolve_background(param=lcdm_massless_param())
    prob = pt.DeviceProblem(tb.pack_cosmology(p, 3)[None], np.geomspace(1e-4, 1e-2, n) if n > 1 else np.array([1e-3]),
                            tb.tau_of_a(p, [0.01])[None], None, lmaxg=8, lmaxgp=8, lmaxr=8, lmaxnu=6, nqmax=3)
    cfg = pt._cfg(1e-2, 1e-3, .25, .8, 0., 20., .3, 2000)
    out = []
    for order in (np.arange(n, dtype=np.int32), np.arange(n, dtype=np.int32)[::-1].copy()):
        prob.order = torch.as_tensor(order).cuda()
        prob.y.fill_(float("nan"))
        prob.steps.zero_()
        prob.launch(cfg)
        torch.cuda.synchronize()
        assert (prob.status == 0).all() and (prob.steps.sum(1) > 0).all()
        out.append(prob.y.clone())
    assert torch.equal(out[0], out[1]) and torch.isfinite(out[0]).all()
