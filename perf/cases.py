"""Timed cases of the perturbation path, by what a user's program calls.

A case is a dict of plain values; ``kind`` names the entry point:

* ``power``: one cosmology, ``evolve_perturbations`` and ``get_power`` on its result;
* ``multi``: several cosmologies in one ``evolve_perturbations_multi``;
* ``grouped``: ``evolve_perturbations_batched`` (shared step sequence per group of modes);
* ``jacobian``: ``evolve_perturbations_grad``, d ln P(k, a) / d theta;
* ``loglike``: ``loglike_grad``, a Gaussian likelihood of P(k, a) and its gradient;
* ``tables``: ``evolve_background_tables``, the input tables of many parameter sets on the GPU;
* ``observables``: redshift-space multipoles, smoothed P(k) and the correlation function of a solve's output.

Every case draws its cosmologies from the seed, in the ranges of
``workloads.sample_cosmologies``.  Grids and tolerances are those of the
workloads, the tests and the benchmark, at sizes a single pass of which takes
microseconds to about a second.
"""
import math

import numpy as np
import torch

import discoeb_gb300 as deb
from discoeb_gb300 import observables, tables_gpu, workloads
from discoeb_gb300.gradient import perturbed_params

SMALL = dict(lmaxg=11, lmaxgp=11, lmaxr=11, lmaxnu=8, nqmax=3)        # the entry points' defaults: 72 variables
LCDM = dict(lmaxg=12, lmaxgp=12, lmaxr=17, lmaxnu=8, nqmax=3)         # 80 variables
FIDUCIAL = dict(lmaxg=12, lmaxgp=12, lmaxr=17, lmaxnu=17, nqmax=15)   # 323 variables
CLASSY = dict(lmaxg=31, lmaxgp=31, lmaxr=31, lmaxnu=31, nqmax=5)      # 265 variables
LARGE = dict(lmaxg=32, lmaxgp=32, lmaxr=32, lmaxnu=32, nqmax=30)      # 1098 variables
DIMS = ("lmaxg", "lmaxgp", "lmaxr", "lmaxnu", "nqmax")
MAX_STEPS = 20000


def listed():
    return [
        # the smallest complete solve: massless LCDM transfer functions at a = 1 on a coarse grid
        dict(name="lcdm_64k", kind="power", **LCDM, kmin=1e-4, kmax=1.0, num_k=64, nout=1, amin=1.0, rtol=1e-3,
             atol=1e-6, massless=True),
        # the everyday call: P(k) today at the default hierarchy sizes, 512 modes
        dict(name="default_512k", kind="power", **SMALL, kmin=1e-4, kmax=10.0, num_k=512, nout=1, amin=1.0, rtol=1e-3,
             atol=1e-3, massless=False),
        # an ordinary call at odd sizes: unequal hierarchies, a prime number of modes, three outputs
        dict(name="odd_97k_3a", kind="power", lmaxg=13, lmaxgp=9, lmaxr=21, lmaxnu=10, nqmax=5, kmin=3e-4, kmax=3.0,
             num_k=97, nout=3, amin=0.35, rtol=1e-4, atol=1e-4, massless=False),
        # precision P(k) with massive neutrinos and a dark-energy fluid
        dict(name="fiducial_256k", kind="power", **FIDUCIAL, kmin=1e-4, kmax=10.0, num_k=256, nout=1, amin=1.0,
             rtol=1e-5, atol=1e-5, massless=False),
        # long hierarchies and an early output, as compared with a Boltzmann code after recombination
        dict(name="early_512k_lmax31", kind="power", **CLASSY, kmin=1e-5, kmax=10.0, num_k=512, nout=1, amin=0.01,
             rtol=1e-5, atol=1e-5, massless=False),
        # training data for an emulator: every mode of eight sampled cosmologies in one launch
        dict(name="multi_8c_512k", kind="multi", **FIDUCIAL, kmin=1e-4, kmax=10.0, num_k=512, ncosmo=8, nout=1,
             amin=1.0, rtol=1e-5, atol=1e-5),
        # the batched form of the early-time benchmark: groups of 16 modes (the default) share their steps
        dict(name="grouped_256k_b16", kind="grouped", **SMALL, kmin=1e-4, kmax=10.0, num_k=256, nout=1, amin=0.01,
             rtol=1e-3, atol=1e-3, batch_size=16),
        # Fisher forecast: d ln P(k, a) / d theta at eight outputs for eight parameters
        dict(name="jacobian_128k_8a", kind="jacobian", **FIDUCIAL, kmin=1e-3, kmax=1.0, num_k=128, ncosmo=1, nout=8,
             amin=0.2, rtol=1e-5, atol=1e-5, land=True),
        # one step of a gradient-based sampler: likelihood and gradient of P(k, a)
        dict(name="loglike_128k_8a", kind="loglike", **FIDUCIAL, kmin=1e-3, kmax=0.1, num_k=128, ncosmo=1, nout=8,
             amin=0.2, rtol=1e-4, atol=1e-4, land=True),
        # the same with the largest hierarchy: long state vectors, many outputs
        dict(name="loglike_large_96k_64a", kind="loglike", **LARGE, kmin=1e-5, kmax=0.006, num_k=96, ncosmo=1, nout=64,
             amin=0.2, rtol=1e-6, atol=1e-6, land=True),
        # input tables of a gradient call on the GPU: nominal and theta +- eps sets of two cosmologies
        dict(name="tables_26", kind="tables", ncosmo=2, nqmax=15, nout=8, amin=0.2),
        # the smallest calls: observables of one solve's output
        dict(name="observables_512k", kind="observables", num_k=512, dlogk=0.2, bias=1.7),
    ]


def _odd(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["power", "power", "power", "multi", "grouped", "jacobian", "loglike", "loglike", "tables",
                       "observables"])
    if kind == "observables":
        return dict(kind=kind, num_k=2 * _odd(rng, 32, 512), dlogk=rng.uniform(0.15, 0.4), bias=rng.uniform(1.0, 2.5))
    if kind == "tables":
        return dict(kind=kind, ncosmo=rng.randint(1, 2), nqmax=rng.randint(3, 15), nout=rng.randint(1, 8),
                    amin=rng.uniform(0.1, 0.9))
    rtol = 10.0 ** rng.uniform(-5.0, -3.0)
    c = dict(kind=kind, kmin=10.0 ** rng.uniform(-4.5, -3.0), kmax=10.0 ** rng.uniform(-0.5, 1.0), rtol=rtol, atol=rtol)
    dims = dict(lmaxg=_odd(rng, 8, 32), lmaxgp=_odd(rng, 8, 32), lmaxr=_odd(rng, 8, 32), lmaxnu=_odd(rng, 6, 32),
                nqmax=_odd(rng, 3, 15))
    if kind == "power":
        c.update(dims, num_k=_odd(rng, 24, 512), nout=rng.randint(1, 4), amin=rng.uniform(0.01, 1.0), massless=False)
    elif kind == "multi":
        c.update(dims, num_k=_odd(rng, 24, 256), ncosmo=rng.randint(2, 7), nout=1, amin=1.0)
        c["rtol"] = c["atol"] = 10.0 ** rng.uniform(-4.5, -3.0)
    elif kind == "grouped":
        b = rng.choice([3, 4, 8, 16])
        c.update(SMALL, num_k=b * rng.randint(2, 16), nout=1, amin=rng.uniform(0.01, 0.1), rtol=1e-3, atol=1e-3,
                 batch_size=b)
        c["lmaxg"] = rng.randint(8, 14)
    else:
        c.update(dims, lmaxnu=_odd(rng, 6, 17), kmax=10.0 ** rng.uniform(-2.0, -1.0), num_k=_odd(rng, 24, 128), ncosmo=1,
                 nout=rng.randint(1, 8), amin=rng.uniform(0.15, 0.8), land=rng.random() < 0.7)
        c["rtol"] = c["atol"] = 10.0 ** rng.uniform(-4.0, -3.0)
    return c


def _aexp(case):
    return np.linspace(case["amin"], 1.0, case["nout"]) if case["nout"] > 1 else np.array([case["amin"]])


def _cosmologies(case, seed, n):
    ps, _ = workloads.sample_cosmologies(n, seed=seed)
    if case.get("massless"):
        for p in ps:
            p.update(Neff=3.046, Nmnu=0, mnu=0.0)
    return ps


def _grid(case):
    return dict(kmin=case["kmin"], kmax=case["kmax"], num_k=case["num_k"])


def _solver(case):
    return dict({d: case[d] for d in DIMS}, rtol=case["rtol"], atol=case["atol"], max_steps=MAX_STEPS)


def _delta_m(p, k, a):
    """Matter transfer function delta(k, a) of a smooth fitting form (BBKS with a matter-era growth)."""
    h = p["H0"] / 100.0
    q = k / (p["Omegam"] * h * h)
    t = np.log1p(2.34 * q) / (2.34 * q) * (1 + 3.89 * q + (16.1 * q) ** 2 + (5.46 * q) ** 3 + (6.71 * q) ** 4) ** -0.25
    hub = p["H0"] / 299792.458
    return 0.4 * (k / hub)[:, None] ** 2 / p["Omegam"] * t[:, None] * (0.8 * np.asarray(a))[None, :]


def _primordial(p, k):
    return 2.0 * math.pi ** 2 * p["A_s"] * (k / p["k_p"]) ** (p["n_s"] - 1.0) * k ** -3.0


def _fields(case, seed):
    """k-grid, output fields y and parameters of an observables case."""
    p = workloads.sample_cosmologies(1, seed=seed)[0][0]
    rng = np.random.default_rng(seed)
    k = np.geomspace(1e-4, 10.0, case["num_k"])
    y = rng.normal(size=(case["num_k"], 20))
    wiggle = 1.0 + 0.05 * np.sin(150.0 * k) * np.exp(-(k / 0.2) ** 2) + 0.01 * rng.normal(size=k.size)
    y[:, 4] = _delta_m(p, k, [1.0])[:, 0] * wiggle
    y[:, 5] = -0.5 * y[:, 4] * (1.0 + 0.01 * rng.normal(size=k.size))
    return k, y, p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "observables":
        k, y, p = _fields(case, seed)
        return dict(case=case, param=p, k=torch.as_tensor(k, device="cuda"), y=torch.as_tensor(y, device="cuda"))
    nc = case.get("ncosmo", 1)
    ps = _cosmologies(case, seed, nc)
    if kind == "tables":
        pert = [q for p in ps for (_, _, a, b) in perturbed_params(p) for q in (a, b)]
        return dict(case=case, params=ps + pert, leader=tables_gpu.follow_nominal(nc, len(pert) // nc))
    if kind in ("power", "grouped", "multi"):
        return dict(case=case, params=tables_gpu.evolve_backgrounds_native(ps))
    if kind == "jacobian":
        return dict(case=case, params=ps)
    k, a = np.geomspace(case["kmin"], case["kmax"], case["num_k"]), _aexp(case)
    rng = np.random.default_rng(seed)
    data = np.stack([np.log(_primordial(p, k)[:, None] * _delta_m(p, k, a) ** 2) for p in ps])
    data += 0.05 * rng.normal(size=data.shape)
    weights = 1e9 * k ** 3 * math.log(k[1] / k[0]) / (4.0 * math.pi ** 2)      # N_k / 2 of a (1 Gpc)^3 volume
    return dict(case=case, params=ps, data=data, weights=np.repeat(weights[:, None], case["nout"], axis=1))


def _sections(t, nqmax):
    """A blob's sections by type: the FP64 part (scalars, splines, momentum nodes), then per spline its
    polynomial coefficients and its knots in FP32."""
    sizes = [256, 256, tables_gpu.NUM_NU, tables_gpu.NUM_NU, 256, 256, 256]
    at = 32 + 3 * sum(sizes) + 2 * nqmax
    out = [t[:, :at]]
    for n in sizes:
        out += [t[:, at:at + 4 * (n - 1)], t[:, at + 4 * (n - 1):at + 4 * (n - 1) + n // 2].view(torch.float32)]
        at += 4 * (n - 1) + n // 2
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "observables":
        k, y, p = state["k"], state["y"], state["param"]
        P = deb.get_power(k=k, y=y, idx=4, param=p)
        p0, p2, p4 = observables.power_multipoles(y=y, kmodes=k, b=case["bias"], param=p)
        smooth = observables.get_power_smoothed(k=k, y=y, dlogk=case["dlogk"], idx=4, param=p)
        xi, r = observables.get_xi_from_P(k=k, Pk=P)
        return dict(P=P, p0=p0, p2=p2, p4=p4, smooth=smooth, xi=xi, r=r)
    if kind == "tables":
        t, tau, status = deb.evolve_background_tables(state["params"], case["nqmax"], aexp_out=_aexp(case),
                                                      leader=state["leader"])
        return dict(sections=_sections(t, case["nqmax"]), tau=tau, status=status)
    if kind == "power":
        y, k, p = deb.evolve_perturbations(param=state["params"][0], aexp_out=_aexp(case), **_grid(case), **_solver(case))
        return dict(y=y, k=k, P=deb.get_power(k=k, y=y, idx=4, param=p))
    if kind == "multi":
        y, k = deb.evolve_perturbations_multi(params=state["params"], aexp_out=_aexp(case), **_grid(case), **_solver(case))
        return dict(y=y, k=k)
    if kind == "grouped":
        y, k = deb.evolve_perturbations_batched(param=state["params"][0], aexp_out=_aexp(case),
                                                batch_size=case["batch_size"], **_grid(case), **_solver(case))
        return dict(y=y, k=k)
    if kind == "jacobian":
        P, D, k = deb.evolve_perturbations_grad(params=state["params"], aexp_out=_aexp(case),
                                                step_to_outputs=case["land"], **_grid(case), **_solver(case))
        return dict(P=P, dlogP=D, k=k)
    P, lnL, g, k = deb.loglike_grad(params=state["params"], lnP_data=state["data"], weights=state["weights"],
                                    aexp_out=_aexp(case), step_to_outputs=case["land"], **_grid(case), **_solver(case))
    return dict(P=P, lnL=lnL, grad=g, k=k)


def _nvar(case):
    return deb.nvar(*(case[d] for d in DIMS))


def _attempts(case):
    """Attempted steps of one mode, averaged over its k-grid (fit of counted steps)."""
    return 120.0 * (1e-3 / case["rtol"]) ** 0.3


def work(case):
    """Bytes: each input and output once.  Operations: of the structured Rodas5 steps (about 190 per state
    element: nine right-hand sides, one factorisation, eight solves and the stage sums), a replayed parameter
    set at the same cost, an adjoint step at five."""
    kind = case["kind"]
    if kind == "observables":
        n = case["num_k"]
        return dict(bytes=8.0 * n * (21 + 7), flops=n * (400.0 + 10.0 * math.log2(n)))
    nc, nout = case.get("ncosmo", 1), case["nout"]
    if kind == "tables":
        sets = nc * 13
        blob = tables_gpu.blob_len(256, case["nqmax"])
        return dict(bytes=8.0 * sets * (blob + nout + 15), flops=sets * 640 * 3000.0)
    modes, n = nc * case["num_k"], _nvar(case)
    blob = 8.0 * tables_gpu.blob_len(256, case["nqmax"])
    step = modes * _attempts(case) * 190.0 * n
    if kind in ("power", "grouped", "multi"):
        return dict(bytes=nc * blob + 8.0 * modes * (1 + nout * 21), flops=step)
    if kind == "jacobian":
        return dict(bytes=13 * nc * blob + 8.0 * modes * (1 + nout * 9), flops=13 * step)
    return dict(bytes=13 * nc * blob + 8.0 * modes * (1 + nout * 3), flops=6 * step)


def _lgamma(z):
    """ln Gamma of complex z by Stirling's series after shifting Re z beyond 20."""
    s = np.zeros_like(z)
    while z.real.min() < 20.0:
        s = s + np.log(z)
        z = z + 1.0
    i = 1.0 / z
    i2 = i * i
    return ((z - 0.5) * np.log(z) - z + 0.5 * math.log(2.0 * math.pi)
            + i * (1 / 12 + i2 * (-1 / 360 + i2 * (1 / 1260 + i2 * (-1 / 1680 + i2 * (1 / 1188)))))) - s


def exact(case, seed):
    """Observables in plain numpy; the adaptive solves and the tables have no closed form to compare with."""
    if case["kind"] != "observables":
        return None
    k, y, p = _fields(case, seed)
    fac = _primordial(p, k)
    P = fac * y[:, 4] ** 2
    d, th, b = np.sqrt(fac) * y[:, 4], np.sqrt(fac) * y[:, 5], case["bias"]
    w = int(round(case["dlogk"] / (math.log(k[1]) - math.log(k[0]))))
    w += (w + 1) % 2
    h = w // 2
    x = np.arange(-h, h + 1, dtype=np.float64)
    c = np.linalg.pinv(x[:, None] ** np.arange(4))[0]
    smooth = np.exp(np.convolve(np.log(P), c[::-1], mode="same"))
    smooth[:h] = P[:h]
    smooth[len(P) - h - 1:] = P[len(P) - h - 1:]
    n = k.size
    t = np.pi * np.arange(n // 2 + 1) / math.log(k[-1] / k[0])
    phase = np.exp(2j * (_lgamma(0.75 + 1j * t).imag - math.log(math.pi) * t))
    r = 2.0 * np.pi / k
    xi = np.fft.irfft(np.fft.rfft(P * k ** 1.5) * phase, n=n) / (2.0 * np.pi * r) ** 1.5
    return dict(P=P, p0=b * b * d * d - 2.0 * b / 3.0 * d * th + th * th / 5.0,
                p2=-4.0 * b / 3.0 * d * th + 4.0 / 7.0 * th * th, p4=8.0 / 35.0 * th * th, smooth=smooth,
                xi=xi[::-1].copy(), r=r[::-1].copy())
