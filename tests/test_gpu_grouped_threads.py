"""Grouped solves from two host threads: on one stream with one plan (launches in
stream order, each with more groups than are in flight), and through the public
call on a stream each."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import discoeb_gb300.background as bg
import discoeb_gb300.tables as tb
from discoeb_gb300 import _native
from discoeb_gb300 import perturbations as pt
from discoeb_gb300.workloads import fiducial_mnu_param

pytestmark = pytest.mark.gpu

DIMS = dict(lmaxg=3, lmaxgp=3, lmaxr=3, lmaxnu=3, nqmax=1)
NK = 2560      # groups of one: more than eight per SM


def _both(work):
    start, errors = threading.Barrier(2), []

    def run(i):
        start.wait()
        try:
            work(i)
        except Exception as e:   # noqa: BLE001 -- reported below
            errors.append(e)

    th = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
    torch.cuda.synchronize()


def _inputs():
    p = bg.evolve_background(param=fiducial_mnu_param(), producer="native")
    return tb.pack_cosmology(p, DIMS["nqmax"])[None], tb.tau_of_a(p, [1e-3])[None], np.geomspace(1e-4, 1e-2, NK)


def test_one_plan_on_one_stream():
    blob, tau, k = _inputs()
    t = [torch.as_tensor(a).cuda() for a in (blob, k, tau)]
    plan = _native.Plan(pt._dims(nout=1, return_full=False, linear_solver="structured", exec_mode="warp", **DIMS), NK,
                        batch_size=1)
    assert plan.launch_info()["modes_in_flight"] < NK
    cfg = pt._cfg(1e-2, 1e-2, 0.25, 0.80, 0.0, 20.0, 0.3, 4096)
    n = 40
    y = torch.full((2, n, NK, 20), float("nan"), dtype=torch.float64, device="cuda")
    st = torch.full((2, n, NK), -1, dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    fn = _native.load().deb_forward_grouped
    c = lambda a: ctypes.c_void_p(a.data_ptr())
    args = [[(plan.ptr, c(t[0]), 1, blob.shape[1], c(t[1]), None, NK, c(t[2]), ctypes.byref(cfg), c(y[i, j]), c(st[i, j]),
              None, ctypes.c_void_p(s.cuda_stream)) for j in range(n)] for i in range(2)]

    def work(i):
        for a in args[i]:
            assert fn(*a) == 0

    _both(work)
    assert (st == 0).all()
    assert torch.equal(y, y[:1, :1].expand_as(y)) and torch.isfinite(y[0, 0]).all()


def test_public_call_on_a_stream_each():
    blob, tau, k = _inputs()
    kw = dict(rtol=1e-2, atol=1e-2, max_steps=4096, **DIMS)
    ref = pt.solve_grouped(blob, k, tau, 1, **kw)
    out = [[], []]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(40):
                out[i].append(pt.solve_grouped(blob, k, tau, 1, **kw))

    _both(work)
    for y in out[0] + out[1]:
        np.testing.assert_array_equal(y, ref)
