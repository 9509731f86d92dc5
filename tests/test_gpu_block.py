"""The block kernel (a block of four warps per mode, deb_block.cuh) against the
warp kernel (deb_forward_static runs it) at the sizes where its split of the
work has edges: shortest hierarchies (no general rows, one-element tails), one
momentum bin, as many bins as a warp has lanes, one more than fills a warp of
chains, and unequal lengths that leave remainders in every pass.

Both kernels evaluate the same expressions with the same roundings, so the step
sequences are equal; a single rounding that differed would, through the
accept / reject decisions, move some mode's steps.  The fields are compared at
1e-12 of each field's largest value: the output conversion alone is compiled
separately in the two (a few operations of 1.1e-16 each, at most ~1e-14).
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [dict(lmaxg=3, lmaxgp=3, lmaxr=3, lmaxnu=3, nqmax=1), dict(lmaxg=5, lmaxgp=4, lmaxr=6, lmaxnu=5, nqmax=31),
         dict(lmaxg=4, lmaxgp=5, lmaxr=3, lmaxnu=4, nqmax=32), dict(lmaxg=13, lmaxgp=9, lmaxr=21, lmaxnu=10, nqmax=5),
         dict(lmaxg=31, lmaxgp=31, lmaxr=31, lmaxnu=31, nqmax=5), dict(lmaxg=32, lmaxgp=32, lmaxr=32, lmaxnu=32, nqmax=30)]


@pytest.mark.parametrize("dims", SIZES, ids=lambda d: "-".join(str(v) for v in d.values()))
def test_block_kernel_takes_the_warp_kernels_steps(dims):
    import torch

    import discoeb_gb300 as deb
    import discoeb_gb300.tables as tb
    from discoeb_gb300 import _native
    from discoeb_gb300 import perturbations as pt
    from discoeb_gb300.workloads import sample_cosmologies

    p = deb.evolve_background(param=sample_cosmologies(1, seed=23)[0][0])
    blob, tau = tb.pack_cosmology(p, dims["nqmax"]), tb.tau_of_a(p, [0.2, 0.7, 1.0])
    k = np.geomspace(1e-4, 2.0, 33)
    y, st = pt.solve(blob[None], k, tau[None], rtol=1e-3, atol=1e-3, max_steps=4096, return_stats=True, **dims)
    dev = torch.device("cuda", torch.cuda.current_device())
    t = {n: torch.as_tensor(a).to(dev) for n, a in (("tab", blob[None]), ("k", k), ("tau", tau[None]))}
    t["y"] = torch.empty((k.size, 3, 20), dtype=torch.float64, device=dev)
    t["st"] = torch.empty(k.size, dtype=torch.int32, device=dev)
    t["steps"] = torch.empty((k.size, 2), dtype=torch.int32, device=dev)
    c = {n: ctypes.c_void_p(a.data_ptr()) for n, a in t.items()}
    d = pt._dims(nout=3, return_full=False, linear_solver="structured", **dims)
    cfg = pt._cfg(1e-3, 1e-3, 0.25, 0.80, 0.0, 20.0, 0.3, 4096)
    _native.check(_native.load().deb_forward_static(
        ctypes.byref(d), c["tab"], 1, blob.shape[0], c["k"], None, k.size, c["tau"], ctypes.byref(cfg), c["y"], c["st"],
        c["steps"], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "deb_forward_static")
    torch.cuda.synchronize()
    assert (st["status"] == 0).all() and (t["st"].cpu().numpy() == 0).all()
    np.testing.assert_array_equal(st["steps"], t["steps"].cpu().numpy())
    ref = t["y"].cpu().numpy()
    assert (np.abs(y - ref) <= 1e-12 * np.abs(ref).max(axis=(0, 1))).all()
