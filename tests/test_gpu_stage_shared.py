"""An explicit "shared" launch shape is taken for every mode whose slot fits the
shared memory a block may have: at 16 vectors of nvar doubles and 31 momentum bins
that is up to nvar 1786, of which the block kernel with its own shared state
reaches 1678.

The result does not depend on the shape: the step sequences are those of the
all-global shape, the fields agree to 1e-12 of their largest value (the output
conversion is compiled separately in the two kernels, as in test_gpu_block.py).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dims(lmaxg):
    return dict(lmaxg=lmaxg, lmaxgp=32, lmaxr=32, lmaxnu=50, nqmax=31)


@pytest.mark.parametrize("lmaxg", [8, 32, 100, 128])      # nvar 1665, 1689, 1757, 1785
def test_shared_shape_up_to_the_shared_memory_of_a_block(lmaxg):
    import torch

    import discoeb_gb300 as deb
    import discoeb_gb300.tables as tb
    from discoeb_gb300 import perturbations as pt
    from discoeb_gb300.workloads import fiducial_mnu_param

    dims = _dims(lmaxg)
    p = deb.evolve_background(param=fiducial_mnu_param(), producer="native")
    prob = pt.DeviceProblem(tb.pack_cosmology(p, dims["nqmax"])[None], np.geomspace(1e-4, 1e-2, 5),
                            tb.tau_of_a(p, [0.01])[None], None, **dims)
    cfg = pt._cfg(1e-3, 1e-3, 0.25, 0.80, 0.0, 20.0, 0.3, 4096)
    out = {}
    for shape in ("all_global", "shared"):
        prob.plan = pt.get_plan(prob.dims, prob.nmode, (shape, 0))
        assert prob.plan.launch_info()["stage_vectors"] == shape
        prob.launch(cfg)
        torch.cuda.synchronize()
        assert (prob.status == 0).all()
        out[shape] = prob.y.cpu().numpy().copy(), prob.steps.cpu().numpy().copy()
    np.testing.assert_array_equal(out["shared"][1], out["all_global"][1])
    ref = out["all_global"][0]
    assert (np.abs(out["shared"][0] - ref) <= 1e-12 * np.abs(ref).max(axis=(0, 1))).all()
