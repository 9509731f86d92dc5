"""The block adjoint at the sizes where its split has edges: the shortest
hierarchies it takes with one momentum bin, 31 bins (a warp of neutrino chains),
33 bins (more than a warp), unequal lengths, and the longest one; one and two
outputs, the first interpolated inside a step.

Reference: the replay's central differences of the same frozen-step map on the
same tables.  Tolerance, from what limits that reference: the quotient's O(eps^2)
term at eps = 1e-4 theta (below 1e-6 of each parameter's largest derivative in
the other adjoint tests) plus the rounding of the replayed ln P, a few 1e-12
after thousands of steps, over 2 eps.  Outputs next to a recorded step end are
left out, as there.
"""
import numpy as np
import pytest

from test_gpu_adjoint import _kinks

from discoeb_gb300.gradient import THETA, GradientProblem, perturbed_params
from discoeb_gb300.workloads import fiducial_mnu_param

pytestmark = pytest.mark.gpu

SIZES = [dict(lmaxg=5, lmaxgp=5, lmaxr=5, lmaxnu=3, nqmax=1), dict(lmaxg=6, lmaxgp=9, lmaxr=5, lmaxnu=5, nqmax=31),
         dict(lmaxg=5, lmaxgp=6, lmaxr=7, lmaxnu=4, nqmax=33), dict(lmaxg=32, lmaxgp=32, lmaxr=32, lmaxnu=32, nqmax=30)]


@pytest.mark.parametrize("dims", SIZES, ids=lambda d: "-".join(str(v) for v in d.values()))
@pytest.mark.parametrize("a_out", [[1.0], [0.4, 1.0]], ids=["1out", "2out"])
def test_adjoint_matches_replayed_quotients(dims, a_out):
    base = fiducial_mnu_param()
    k = np.geomspace(1e-3, 0.03, 5)
    pert = [perturbed_params(base)]
    kw = dict(rtol=1e-5, atol=1e-5, max_steps=8000, **dims)
    D, gp = {}, {}
    for method in ("adjoint", "replay"):
        gp[method] = GradientProblem([base], "native", pert, k, a_out, method=method, **kw)
        D[method] = gp[method].run()[1].cpu().numpy()
        gp[method].check()
    kink = _kinks(gp["replay"], 1e-4)
    eps = {name: e for (name, e, _, _) in pert[0]}
    for j, name in enumerate(THETA):
        err = np.abs(D["adjoint"][..., j] - D["replay"][..., j]) - (4e-12 / (2 * eps[name]) if name in eps else 0.0)
        assert np.where(kink, 0.0, err).max() <= 1e-6 * np.abs(D["replay"][..., j]).max(), name
