"""Two host threads that produce frozen tables of different sizes at once, each
on a stream and buffers of its own: every call is accepted, and the tables are
those of a call alone.
"""
import ctypes
import threading

import numpy as np
import pytest
import torch

from discoeb_gb300 import _native, tables_gpu
from discoeb_gb300.workloads import fiducial_mnu_param

pytestmark = pytest.mark.gpu


class _Call:
    """deb_evolve_background_frozen of a leader and a follower with its arguments laid out once."""

    def __init__(self, num_thermo):
        p = fiducial_mnu_param()
        dev = torch.device("cuda", torch.cuda.current_device())
        cap = 16 * num_thermo
        self.bl = tables_gpu.blob_len(num_thermo, 3)
        t = dict(pm=torch.as_tensor(tables_gpu.param_matrix([p, dict(p, Omegam=1.001 * p["Omegam"])])),
                 leader=torch.tensor([-1, 0], dtype=torch.int32), consts=torch.as_tensor(tables_gpu.constants()),
                 grid=torch.as_tensor(tables_gpu.grid(num_thermo, 3)),
                 steps=torch.zeros((2, 3 * num_thermo + 1 + 2 * cap), dtype=torch.float64),
                 tabs=torch.zeros((2, self.bl), dtype=torch.float64), status=torch.zeros(2, dtype=torch.int32))
        self.t = {n: a.to(dev) for n, a in t.items()}
        self.stream = torch.cuda.Stream()
        c = {n: ctypes.c_void_p(a.data_ptr()) for n, a in self.t.items()}
        self.cfg = tables_gpu.DebBgCfg(num_thermo, tables_gpu.NUM_NU, tables_gpu.NQ_BG, 3, 128, tables_gpu.AMIN, 1e-3, 1e-6)
        self.args = (ctypes.byref(self.cfg), c["pm"], 2, c["leader"], c["consts"], c["grid"], c["steps"], cap, c["tabs"],
                     self.bl, c["status"], ctypes.c_void_p(self.stream.cuda_stream))

    def tables(self):
        torch.cuda.synchronize()
        assert (self.t["status"] == 0).all()
        return self.t["tabs"].cpu().numpy().copy()


def test_two_sizes_from_two_threads():
    fn = _native.load().deb_evolve_background_frozen
    calls = [_Call(32), _Call(256)]
    torch.cuda.synchronize()
    alone = []
    for c in calls:
        assert fn(*c.args) == 0
        alone.append(c.tables())
    rcs, start = [set(), set()], threading.Barrier(2)

    def work(i):
        start.wait()
        for _ in range(100):
            rcs[i].add(fn(*calls[i].args))

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert rcs == [{0}, {0}]
    for c, ref in zip(calls, alone):
        np.testing.assert_array_equal(c.tables(), ref)
