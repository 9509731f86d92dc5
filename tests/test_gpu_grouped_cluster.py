"""The group kernel's cluster: groups of one block and of several, blocks whose
last warps have no mode, slots in shared and in global memory, more groups than
are in flight at once.

Against the host build of the same driver at rtol 1e-8, where two valid step
sequences of a mode agree to ~1e-7 in P(k) (test_gpu_grouped.py; its bar 1e-6).
A group's norm is an RMS over its modes, so one mode may take sqrt(B) times the
error: bar 1e-6 sqrt(B).
"""
import numpy as np
import pytest
import torch

from native import harness as H

import discoeb_gb300.background as bg
import discoeb_gb300.tables as tb
from discoeb_gb300 import _native
from discoeb_gb300 import perturbations as pt
from discoeb_gb300.workloads import sample_cosmologies

pytestmark = pytest.mark.gpu

SMALL = dict(lmaxg=8, lmaxgp=8, lmaxr=10, lmaxnu=8, nqmax=3)
LONG = dict(lmaxg=20, lmaxgp=20, lmaxr=20, lmaxnu=20, nqmax=20)     # nvar 492: four slots exceed an SM


@pytest.fixture(scope="module")
def cosmologies():
    return [bg.evolve_background(param=p, producer="native") for p in sample_cosmologies(2, seed=29)[0]]


def _inputs(cosmologies, dims, a_out):
    return (np.stack([tb.pack_cosmology(p, dims["nqmax"]) for p in cosmologies]),
            np.stack([tb.tau_of_a(p, a_out) for p in cosmologies]))


@pytest.mark.parametrize("B", [1, 2, 3, 5, 9, 17])
def test_an_sm_holds_four_modes_or_more(B):
    """Fewer than four warps leave an SM's FP64 unit idle (19 cycles an instruction, 64 for one warp)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for dims in (SMALL, LONG):
        plan = _native.Plan(pt._dims(nout=1, return_full=False, linear_solver="structured", **dims), 9180, batch_size=B)
        assert plan.launch_info()["modes_in_flight"] >= 4 * sms


@pytest.mark.parametrize("dims, B", [(SMALL, 1), (SMALL, 2), (SMALL, 3), (SMALL, 5), (SMALL, 16), (SMALL, 17), (SMALL, 32),
                                     (LONG, 1), (LONG, 5)])
def test_groups_follow_the_host_driver(cosmologies, dims, B):
    tabs, tau = _inputs(cosmologies, dims, [0.01])
    k = np.tile(np.geomspace(1e-3, 0.3, 2 * B), 2)
    com = np.repeat(np.array([0, 1], dtype=np.int32), 2 * B)
    kw = dict(rtol=1e-8, atol=1e-8, max_steps=20000, **dims)
    y, st = pt.solve_grouped(tabs, k, tau, B, com, return_stats=True, **kw)
    yh, sh = H.solve_grouped(tabs, k, tau, B, cosmo_of_mode=com, **kw)
    assert (st["status"] == 0).all() and (sh[:, 0] == 0).all()
    assert len({tuple(s) for s in st["steps"][:B]}) == 1
    np.testing.assert_allclose(y[:, 0, 4] ** 2, yh[:, 0, 4] ** 2, rtol=1e-6 * np.sqrt(B))


@pytest.mark.parametrize("B", [5, 9, 17, 32])
def test_every_block_of_a_cluster_enters_the_norm(cosmologies, B):
    """One mode that needs several times the steps of the others, in turn in each
    block of the cluster.  Its share of the RMS lets it take B^(1/10) times its own
    step lengths (error of order 5): 0.7 of its own steps at B = 32, where a norm
    without its block would give those of the easy modes."""
    tabs, tau = _inputs(cosmologies[:1], SMALL, [0.01])
    kw = dict(rtol=1e-8, atol=1e-8, max_steps=20000, return_stats=True, **SMALL)
    alone = pt.solve_grouped(tabs, np.array([1e-3, 0.3]), tau, 1, **kw)[1]["steps"].sum(1)
    assert alone[0] < 0.4 * alone[1]
    at = list(range(0, B, 4)) + [B - 1]
    k = np.full((len(at), B), 1e-3)
    k[np.arange(len(at)), at] = 0.3
    steps = pt.solve_grouped(tabs, k.ravel(), tau, B, **kw)[1]["steps"].sum(1).reshape(k.shape)
    assert (steps >= 0.55 * alone[1]).all()


@pytest.mark.parametrize("dims, B, kept", [(SMALL, 1, False), (SMALL, 5, False), (SMALL, 32, False), (LONG, 3, False),
                                           (dict(SMALL, lmaxnu=30, nqmax=8), 2, True)])
def test_repeated_groups_have_the_same_bits(cosmologies, dims, B, kept):
    """More groups than are in flight, every third one the same; and a launch of few groups on the plan
    made for many (kept), which may hold its slots elsewhere."""
    tabs, tau = _inputs(cosmologies[:1], dims, [0.01])
    n = 3 * (1300 // B + 1) if B < 5 else 3 * (320 // B + 30)
    base = np.geomspace(1e-3, 0.3, 3 * B)
    kw = dict(rtol=1e-3, atol=1e-3, max_steps=4000, return_stats=True, **dims)
    y, st = pt.solve_grouped(tabs, np.tile(base, n // 3), tau, B, **kw)
    assert (st["status"] == 0).all()
    y = y.reshape(n // 3, 3 * B, -1)
    np.testing.assert_array_equal(y, np.broadcast_to(y[:1], y.shape))
    if kept:
        few, _ = pt.solve_grouped(tabs, base, tau, B, **kw)
        np.testing.assert_array_equal(few.reshape(3 * B, -1), y[0])
