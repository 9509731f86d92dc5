"""GradientProblem.tune times the launches that take the plan, on a plan of their size (stand-in launches)."""
import pytest

from discoeb_gb300 import autotune
from discoeb_gb300 import perturbations as pt
from discoeb_gb300.gradient import GradientProblem


@pytest.mark.parametrize("method, launches, modes", [("replay", ["deb_forward_record", "deb_replay"], 12 * 128),
                                                     ("adjoint", ["deb_forward_record_ckpt"], 128)])
def test_tune_times_record_and_replay(monkeypatch, method, launches, modes):
    import types

    from discoeb_gb300 import _native

    seen = []

    class _Lib:
        def __getattr__(self, name):
            return lambda *a: seen.append(name) or 0

    class _Tensor:
        def data_ptr(self):
            return 0

    gp = object.__new__(GradientProblem)
    for n in ("d_tab0", "d_tabs", "d_k", "d_com", "d_tau0", "d_taus", "d_rec", "d_nrec", "d_y0", "d_st0", "d_steps",
              "d_ys", "d_sts", "d_ckpt", "d_ckstride"):
        setattr(gp, n, _Tensor())
    gp.d_ckoff = gp.d_ckcap = None
    gp.method, gp.nset, gp.nmode, gp.nc, gp.blob_len, gp.rec_len, gp.ck_cap = method, 12, 128, 1, 100, 10, 32
    gp.order, gp.dims, gp.cfg = None, None, pt._cfg(1e-5, 1e-5, 0.25, 0.8, 0.0, 20.0, 0.3, 9)
    plan, s = types.SimpleNamespace(ptr=None), types.SimpleNamespace(cuda_stream=0)
    tuned = []

    def tune(dims, max_modes, launch_fn, candidates):
        launch_fn(plan, s)
        tuned.append(max_modes)
        return ("shared", 0), {("shared", 0): 1.0}

    monkeypatch.setattr(_native, "load", lambda: _Lib())
    monkeypatch.setattr(autotune, "tune", tune)
    monkeypatch.setattr(pt, "get_plan", lambda dims, n, launch=None: (n, launch))
    gp.tune()
    assert seen == launches
    assert tuned == [modes] and gp.plan == (modes, ("shared", 0))
