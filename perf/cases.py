"""What a program that uses this framework has it do, as cases that can be timed.

A case is a dict of plain values; `kind` names the call it stands for:

  step      a stretch of a run: `steps` fused time steps, then the result
            fields as the GiD writer takes them (FP32 snapshot; FP64 download
            in the plain form, whose solves end at 1e-12)
  routines  the drop-in swapped in call by call: host arrays in, the seven
            module procedures, every host array back (plain FP64, solved to
            1e-13 as in the parity runs)
  solve     steady flow through a new rock: upload, calcPermeability,
            solvePressure from a flat pressure, calcVelocity, download
            (FP32-refined, to a 1e-12 residual)
  ensemble  `steps` steps of a few uneven domains advanced together
  diag      the showProgress reductions, on a handle's fields or (`noalloc`)
            on device arrays the caller holds
  conv3d    one 3x3x3 convolution of the warm-start net, or (`op` wgrad) its
            weight gradient
  forward   the warm-start net's forward pass
  train     one Adam step of the warm-start net

The rocks are seeded Gaussian random fields (log-variance, correlation
length), as in the tests and the benchmark.  A step, ensemble or routines case
starts from rock with a flat inlet (`stage` early) or from a dissolution
front part of the way through the domain, with the smooth phase profile and the
acid distribution of a run that has been going for long (`stage` late).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from mizuho_edit_gb300 import capi
from mizuho_edit_gb300.cases import make_case
from mizuho_edit_gb300.learned import DEFAULT_WEIGHTS, WarmStartNet
from mizuho_edit_gb300.sim import Simulation

CHANNELS = ((16, 16), (16, 32), (32, 64), (64, 64), (64, 32), (32, 16))


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # the smallest run: a core-plug test domain, every kernel a few microseconds
        dict(name="step-40x36x28", kind="step", nx=40, ny=36, nz=28, solver="mixed", stage="early", steps=10,
             spin=12, log_var=1.0, corr=4.0, kwh=20.0, wlevel=0),
        # an ordinary run early on: most of the rock untouched, a few PCG iterations a step
        dict(name="step-128", kind="step", nx=128, ny=128, nz=128, solver="mixed", stage="early", steps=10,
             spin=40, log_var=2.0, corr=8.0, kwh=20.0, wlevel=0),
        # a ragged domain late in its run
        dict(name="step-150x83x61", kind="step", nx=150, ny=83, nz=61, solver="mixed", stage="late", steps=10,
             spin=14, log_var=3.0, corr=6.0, kwh=1000.0, wlevel=0),
        # the headline size late in its run: fronts and acid through most of the domain
        dict(name="step-256", kind="step", nx=256, ny=256, nz=256, solver="mixed", stage="late", steps=10,
             spin=20, log_var=2.0, corr=8.0, kwh=1000.0, wlevel=3),
        # the plain FP64 form of the step, at the parity runs' tolerance
        dict(name="step-fp64-96x80x72", kind="step", nx=96, ny=80, nz=72, solver="fp64", stage="early", steps=4,
             spin=6, log_var=1.0, corr=4.0, kwh=20.0, wlevel=0),
        # the call-by-call drop-in at the plain method's size
        dict(name="routines-64", kind="routines", nx=64, ny=64, nz=64, log_var=1.0, corr=4.0, kwh=20.0),
        # one rock realisation after the other
        dict(name="solve-100x90x110", kind="solve", nx=100, ny=90, nz=110, log_var=2.0, corr=8.0, kwh=20.0),
        # the ensemble of uneven domains, a quarter of the shapes' number
        dict(name="ensemble-4", kind="ensemble", shapes="64x64x64,96x96x96,64x64x64,48x40x56", steps=6, spin=12,
             log_var=1.5, corr=6.0, kwh=20.0),
        # progress lines of a run
        dict(name="diag-160", kind="diag", nx=160, ny=160, nz=160, noalloc=False, log_var=1.0, corr=4.0, kwh=20.0),
        # a deep layer of the net on a grid that is no multiple of anything
        dict(name="conv-64-64-36x28x21", kind="conv3d", op="forward", cin=64, cout=64, nx=36, ny=28, nz=21,
             fp32_out=False),
        # the net beside a 128^3 run
        dict(name="forward-64", kind="forward", nx=64, ny=64, nz=64),
        # training it
        dict(name="train-48x40x32", kind="train", nx=48, ny=40, nz=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi, cells):
    while True:
        d = [_log(rng, lo, hi) for _ in range(3)]
        if d[0] * d[1] * d[2] <= cells:
            return dict(nx=d[0], ny=d[1], nz=d[2])


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step-fp64", "routines", "solve", "ensemble", "diag", "conv3d",
                       "conv3d", "forward", "train"])
    rock = dict(log_var=round(rng.uniform(0.5, 3.0), 2), corr=round(rng.uniform(3.0, 12.0), 1),
                kwh=rng.choice([20.0, 1000.0]))
    stage = rng.choice(["early", "late"])
    if kind == "step":
        return dict(kind="step", **_dims(rng, 24, 240, 1 << 22), solver="mixed", stage=stage,
                    steps=rng.choice([4, 10]), spin=14, wlevel=rng.choice([0, 3]), **rock)
    if kind == "step-fp64":
        return dict(kind="step", **_dims(rng, 24, 128, 1 << 20), solver="fp64", stage=stage, steps=rng.choice([2, 4]),
                    spin=6, wlevel=0, **rock)
    if kind == "routines":
        return dict(kind="routines", **_dims(rng, 20, 112, 1 << 19), **rock)
    if kind == "solve":
        return dict(kind="solve", **_dims(rng, 20, 160, 1 << 21), **rock)
    if kind == "ensemble":
        shapes = [_dims(rng, 24, 112, 1 << 20) for _ in range(rng.randint(2, 5))]
        return dict(kind="ensemble", shapes=",".join("%dx%dx%d" % (s["nx"], s["ny"], s["nz"]) for s in shapes),
                    steps=rng.choice([3, 6]), spin=12, **rock)
    if kind == "diag":
        return dict(kind="diag", **_dims(rng, 16, 256, 1 << 23), noalloc=rng.random() < 0.4, **rock)
    if kind == "conv3d":
        cin, cout = rng.choice(CHANNELS)
        most = (1 << 21) * 16 // max(cin, cout)
        return dict(kind="conv3d", op=rng.choice(["forward", "wgrad"]), cin=cin, cout=cout,
                    **_dims(rng, 8, 128, most), fp32_out=rng.random() < 0.3)
    while True:
        d = dict(nx=8 * _log(rng, 1, 16), ny=8 * _log(rng, 1, 16), nz=8 * _log(rng, 1, 16))
        if d["nx"] * d["ny"] * d["nz"] <= (1 << 20):
            return dict(kind=kind, **d)


# ---- inputs -------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _grf(shape, corr, gen):
    """Zero-mean, unit-variance Gaussian random field on the GPU (squared-exponential covariance)."""
    w = torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)
    k2 = 0
    for a, n in enumerate(shape):
        f = torch.fft.rfftfreq(n, device="cuda", dtype=torch.float64) if a == len(shape) - 1 else \
            torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)
        k2 = k2 + ((2 * math.pi * f) ** 2).reshape([-1 if b == a else 1 for b in range(len(shape))])
    g = torch.fft.irfftn(torch.fft.rfftn(w) * torch.exp(-0.25 * k2 * corr * corr), s=shape)
    g = g - g.mean()
    return g / g.std().clamp_min(1e-300)


def _fields(shape, case, stage, seed):
    """(K_rock, phase, concentration) of one domain, (nz, ny, nx) on the GPU."""
    nx, ny, nz = shape
    gen = _gen(seed)
    kr = torch.exp(math.sqrt(case["log_var"]) * _grf((nz, ny, nx), case["corr"], gen))
    if stage == "early":
        ph = torch.full((nz, ny, nx), -1.0, dtype=torch.float64, device="cuda")
        cc = torch.zeros_like(ph)
    else:
        # a front at 30 % of the length with fingers, the tanh profile of the phase equation
        # cut off where a run has not carried it yet, acid behind it and a tail ahead of it
        front = 0.3 * nx + 0.05 * nx * _grf((nz, ny), max(4.0, 0.06 * (ny + nz)), gen).clamp(-2.5, 2.5)
        d = torch.arange(1, nx + 1, dtype=torch.float64, device="cuda") - front[..., None]
        ph = -torch.tanh(d / 4.0)
        ph = torch.where(d.abs() > 0.05 * nx + 3, -torch.sign(d), ph)
        cc = torch.where(d < 0, torch.ones_like(d), torch.exp(-d.clamp_min(0.0) / (0.05 * nx + 2)))
        cc = torch.where(d > 0.3 * nx, torch.zeros_like(cc), cc)
    ph[..., 0], ph[..., -1] = 1.0, -1.0
    cc[..., 0], cc[..., -1] = 1.0, 0.0
    return kr, ph, cc


def _host(t):
    """The (nx, ny, nz) Fortran-order host array of an (nz, ny, nx) tensor."""
    return t.cpu().numpy().transpose(2, 1, 0)


def _halo(t):
    """One-cell halo that copies the nearest interior cell (updateHalo)."""
    for a in range(3):
        n = t.shape[a]
        t = torch.cat([t.narrow(a, 0, 1), t, t.narrow(a, n - 1, 1)], a)
    return t


def _params(shape, kwh):
    return make_case(shape, log_var=0.0, kwh=kwh)


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


class Pinned:
    """A page-locked host array from the library (wpf_host_alloc); given back with the last view of it."""

    def __init__(self, shape, dtype=np.float64):
        n = int(np.prod(shape))
        self.L, p = capi.load(), C.c_void_p()
        capi.check(self.L.wpf_host_alloc(n * np.dtype(dtype).itemsize, C.byref(p)), "wpf_host_alloc")
        self.ptr = p
        self.__array_interface__ = dict(shape=(n,), typestr=np.dtype(dtype).str, data=(p.value, False), version=3)

    def __del__(self):
        self.L.wpf_host_free(self.ptr)


def _pinned(shape, dtype=np.float64):
    a = np.asarray(Pinned(shape, dtype)).reshape(shape, order="F")
    a[...] = 0
    return a


def _snapshot_array(shape):
    """Pressure, phase, concentration and cell permeability of the interior, one after the other."""
    return _pinned(tuple(shape) + (4,), np.float32)


def _dp(a):
    return a.ctypes.data_as(capi.DP)


def _step_sim(shape, case, stage, seed, solver, wlevel):
    kr, ph, cc = (_host(t) for t in _fields(shape, case, stage, seed))
    p = _params(shape, case["kwh"]).params
    if solver == "fp64":
        return Simulation(p, kr, ph, cc, solver="fp64", rtol=1e-12, w_from_level=wlevel)
    return Simulation(p, kr, ph, cc, solver="mixed", rtol=1e-8, extrapolate=True, step_graph=True,
                      w_from_level=wlevel)


def _solution_guess(shape, kr, ph, kwh):
    """A smooth pressure between the two ends: what a run holds from its last step is near the solution."""
    f = 0.5 * (1 + ph)
    r = (1 / (kwh * f + kr * (1 - f))).mean(dim=(0, 1))
    c = torch.cumsum(r, 0) - r[0]
    p = 1 - c / c[-1]
    return p.expand(shape[2], shape[1], shape[0]).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        sim = _step_sim(_shape(case), case, case["stage"], seed, case["solver"], case["wlevel"])
        sim.run(case["spin"])
        s = dict(kind=kind, sim=sim, steps=case["steps"], snapshot=case["solver"] == "mixed")
        if s["snapshot"]:
            s["out"] = _snapshot_array(_shape(case))
        return s
    if kind == "ensemble":
        shapes = [tuple(int(v) for v in t.split("x")) for t in case["shapes"].split(",")]
        sims = [_step_sim(t, case, "early", seed * 16 + m, "mixed", 0) for m, t in enumerate(shapes)]
        n = len(sims)
        s = dict(kind=kind, sims=sims, n=n, steps=case["steps"], done=0, L=sims[0].L,
                 hs=(C.c_void_p * n)(*[x.h.value for x in sims]), dt=(C.c_double * n)(*[x.dtime for x in sims]),
                 out=[_snapshot_array(t) for t in shapes])
        _ensemble(s, case["spin"])
        return s
    if kind in ("routines", "solve", "diag"):
        shape = _shape(case)
        stage = "early" if kind == "solve" else "late"
        kr, ph, cc = _fields(shape, case, stage, seed)
        p = _params(shape, case["kwh"]).params
        if kind == "diag" and case["noalloc"]:
            cp = capi.Params(p.nx, p.ny, p.nz, p.ix_ref, p.iy_ref, p.iz_ref, p.dx, p.epsilon, p.lambda_, p.porosity,
                             p.viscosity, p.diffusion, p.ral, p.rat, p.permeab_hole, p.alpha, p.tfac)
            return dict(kind=kind, noalloc=True, L=capi.load(), prm=cp, ph=_halo(ph).contiguous(),
                        cc=_halo(cc).contiguous())
        pr = _solution_guess(shape, kr, ph, case["kwh"]) if kind != "solve" else torch.zeros_like(ph)
        s = dict(kind=kind, noalloc=False)
        for name, t in (("kr", kr), ("ph", ph), ("cc", cc), ("pr", pr)):
            s[name] = _pinned(tuple(n + 2 for n in shape))
            s[name][...] = _host(_halo(t))
        if kind == "diag":
            sim = Simulation(p, _host(kr), _host(ph), _host(cc), solver="mixed")
            sim.upload(pressure=s["pr"])
            sim.calcPermeability()
            s.update(sim=sim)
            return s
        sim = Simulation(p, solver="fp64" if kind == "routines" else "mixed",
                         rtol=1e-13 if kind == "routines" else 1e-12)
        sh = tuple(n + 2 for n in shape)
        names = ("phase", "concent", "dphasedt", "dconcentdt") if kind == "routines" else ()
        s["out"] = {n: _pinned(sh) for n in names + ("pressure",)}
        s["out"]["velocity"] = _pinned((3,) + sh)
        if kind == "routines":
            s["out"]["permeab"] = _pinned((4,) + sh)
        s.update(sim=sim, dt=0.05)
        return s
    if kind == "conv3d":
        return _conv_state(case, seed)
    net = WarmStartNet(*_shape(case))
    net.set_params(WarmStartNet.load_params(DEFAULT_WEIGHTS))
    x, target = _net_inputs(case, seed)
    s = dict(kind=kind, net=net, x=x.view(torch.int16), target=target)
    if kind == "forward":
        s["out"] = torch.empty(x.numel() // 16, dtype=torch.float32, device="cuda")
    else:
        s["grads"] = np.zeros(net.nparam, np.float32)
    return s


def _conv_state(case, seed):
    gen = _gen(seed)
    nvox, cin, cout = case["nx"] * case["ny"] * case["nz"], case["cin"], case["cout"]

    def normal(*shape):
        return torch.randn(shape, device="cuda", generator=gen)
    x = normal(nvox, cin).bfloat16()
    s = dict(kind="conv3d", op=case["op"], L=capi.load(), dims=(cin, cout) + _shape(case), x=x)
    if case["op"] == "forward":
        s["w"] = (normal(cout, 27, cin) * (2.0 / (27 * cin)) ** 0.5).bfloat16()
        s["b"] = 0.1 * normal(cout)
        s["out"] = torch.empty(nvox, cout, dtype=torch.float32 if case["fp32_out"] else torch.bfloat16, device="cuda")
    else:
        s["gy"] = normal(nvox, cout).bfloat16()
        s["gw"] = torch.empty(cout, 27, cin, device="cuda")
        s["gb"] = torch.empty(cout, device="cuda")
    return s


def _net_inputs(case, seed):
    """Features like those of a run (normalised log K, phase, pressure, increments), and a target."""
    nx, ny, nz = _shape(case)
    gen = _gen(seed)
    x = torch.zeros(nz * ny * nx, 16, device="cuda")
    x[:, 0] = _grf((nz, ny, nx), 4.0, gen).reshape(-1)
    x[:, 1] = torch.tanh(4 * _grf((nz, ny, nx), 6.0, gen)).reshape(-1)
    x[:, 2] = torch.linspace(1, 0, nx, device="cuda").repeat(nz * ny)
    for c in (3, 4, 5):
        x[:, c] = _grf((nz, ny, nx), 5.0, gen).reshape(-1)
    target = 0.5 * x[:, 4] + 0.1 * _grf((nz, ny, nx), 3.0, gen).reshape(-1).float()
    return x.bfloat16().contiguous(), target.contiguous()


# ---- one pass -------------------------------------------------------------------
def _ensemble(s, steps):
    capi.check(s["L"].wpf_ensemble_run(s["hs"], s["n"], 1 + s["done"], steps, 4, s["dt"], None, None),
               "wpf_ensemble_run")
    s["done"] += steps


def _snapshot(sim, out):
    capi.check(sim.L.wpf_snapshot(sim.h, C.c_void_p(out.ctypes.data)), "wpf_snapshot")


def run(s):
    kind = s["kind"]
    if kind == "step":
        sim = s["sim"]
        sim.run(s["steps"])
        if not s["snapshot"]:
            return sim.download("phase", "concent", "pressure")
        _snapshot(sim, s["out"])
        capi.check(sim.L.wpf_snapshot_wait(sim.h), "wpf_snapshot_wait")
        return s["out"]
    if kind == "ensemble":
        _ensemble(s, s["steps"])
        for sim, out in zip(s["sims"], s["out"]):
            _snapshot(sim, out)
        for sim in s["sims"]:
            capi.check(sim.L.wpf_snapshot_wait(sim.h), "wpf_snapshot_wait")
        return s["out"]
    if kind == "diag":
        if not s["noalloc"]:
            return s["sim"].diagnostics()
        d = capi.Diag()
        capi.check(s["L"].wpf_reduce_noalloc(C.byref(s["prm"]), C.c_void_p(s["ph"].data_ptr()),
                                             C.c_void_p(s["cc"].data_ptr()), C.byref(d), None), "wpf_reduce_noalloc")
        return d.as_dict()
    if kind in ("routines", "solve"):
        sim, out = s["sim"], s["out"]
        L, h = sim.L, sim.h
        capi.check(L.wpf_upload(h, _dp(s["kr"]), _dp(s["ph"]), _dp(s["cc"]), _dp(s["pr"])), "wpf_upload")
        sim.calcPermeability()
        sim.solvePressure()
        sim.calcVelocity()
        if kind == "solve":
            capi.check(L.wpf_download(h, None, None, _dp(out["pressure"]), None, _dp(out["velocity"]), None, None),
                       "wpf_download")
            return out
        sim.calcPhaseDeriv()
        sim.calcConcentDeriv()
        sim.evolvePhase(s["dt"])
        sim.evolveConcent(s["dt"])
        capi.check(L.wpf_download(h, *[_dp(out[n]) for n in ("phase", "concent", "pressure", "permeab", "velocity",
                                                             "dphasedt", "dconcentdt")]), "wpf_download")
        return out
    if kind == "conv3d":
        cin, cout, nx, ny, nz = s["dims"]
        at = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        if s["op"] == "forward":
            f32 = s["out"].dtype == torch.float32
            capi.check(s["L"].wpf_conv3d(cin, cout, nx, ny, nz, at(s["x"]), at(s["w"]), at(s["b"]), 1,
                                         None if f32 else at(s["out"]), at(s["out"]) if f32 else None, None),
                       "wpf_conv3d")
            return s["out"]
        s["gw"].zero_()
        s["gb"].zero_()
        capi.check(s["L"].wpf_conv3d_wgrad(cin, cout, nx, ny, nz, at(s["x"]), at(s["gy"]), at(s["gw"]), at(s["gb"]),
                                           None), "wpf_conv3d_wgrad")
        return [s["gw"], s["gb"]]
    net = s["net"]
    if kind == "forward":
        net.forward(s["x"], s["out"])
        return s["out"]
    loss = net.train_step(s["x"], s["target"], 1e-4)
    capi.check(net.L.wpf_net_get_grads(net.h, s["grads"].ctypes.data_as(C.c_void_p)), "wpf_net_get_grads")
    return dict(loss=np.float32(loss), grads=s["grads"], params=net.params())


# ---- what a pass cannot do without ------------------------------------------------
def _net_flops(vox):
    cin, cout = (16, 16, 32, 64, 64, 32, 16), (16, 32, 64, 64, 32, 16, 16)
    return sum(2.0 * 27 * a * b * vox / 8 ** lv for a, b, lv in zip(cin, cout, (0, 1, 2, 3, 2, 1, 0)))


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(math.prod(int(v) for v in t.split("x")) for t in case["shapes"].split(","))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    if kind in ("step", "ensemble"):
        # a step reads K_rock, phase, concentration and pressure and writes the last three (FP64)
        out = 16 if kind == "ensemble" or case["solver"] == "mixed" else 24
        return dict(bytes=case["steps"] * cells * 56.0 + cells * out, flops=case["steps"] * cells * 150.0)
    if kind == "routines":   # four arrays in, twelve values a cell back
        return dict(bytes=cells * 128.0, flops=cells * 200.0)
    if kind == "solve":      # four arrays in, four values a cell back
        return dict(bytes=cells * 64.0, flops=cells * 60.0)
    if kind == "diag":
        return dict(bytes=cells * 16.0, flops=cells * 8.0)
    if kind == "conv3d":
        cin, cout = case["cin"], case["cout"]
        flops = 2.0 * 27 * cin * cout * cells
        if case["op"] == "wgrad":
            return dict(bytes=cells * 2.0 * (cin + cout) + 27 * cin * cout * 4.0, flops=flops)
        return dict(bytes=cells * (2.0 * cin + (4.0 if case["fp32_out"] else 2.0) * cout) + 27 * cin * cout * 2.0,
                    flops=flops)
    if kind == "forward":
        return dict(bytes=cells * 36.0, flops=_net_flops(cells))
    return dict(bytes=cells * 36.0, flops=3 * _net_flops(cells))


# ---- the same in 64 bits ------------------------------------------------------------
def _exact_flow(kr, ph, kwh, mu, outlet):
    """K0, face K, pressure and velocity of calcPermeability, solvePressure and calcVelocity; halo arrays."""
    f = 0.5 * (1 + _halo(ph))
    k0 = kwh * f + _halo(kr) * (1 - f)
    nz, ny, nx = ph.shape
    kf = []
    for a in (2, 1, 0):      # x, y, z faces, at the cell below them
        lo, hi = k0.narrow(a, 0, k0.shape[a] - 1), k0.narrow(a, 1, k0.shape[a] - 1)
        t = torch.zeros_like(k0)
        t[:nz + 1, :ny + 1, :nx + 1] = (2 * lo * hi / (lo + hi))[:nz + 1, :ny + 1, :nx + 1]
        kf.append(t)
    inner = (slice(1, -1),) * 3
    tx = kf[0][inner][..., :-1] / mu
    ty = kf[1][inner][:, :-1] / mu
    tz = kf[2][inner][:-1] / mu

    def apply(p):            # sum over the faces of T (p_c - p_nb)
        r = torch.zeros_like(p)
        for a, t in ((2, tx), (1, ty), (0, tz)):
            n = p.shape[a]
            q = t * (p.narrow(a, 1, n - 1) - p.narrow(a, 0, n - 1))
            r.narrow(a, 0, n - 1).sub_(q)
            r.narrow(a, 1, n - 1).add_(q)
        return r
    diag = torch.zeros_like(ph)
    for a, t in ((2, tx), (1, ty), (0, tz)):
        n = ph.shape[a]
        diag.narrow(a, 0, n - 1).add_(t)
        diag.narrow(a, 1, n - 1).add_(t)
    free = torch.ones_like(ph)
    free[..., 0] = free[..., -1] = 0
    p = torch.linspace(1, 0, nx, dtype=torch.float64, device=ph.device).expand(nz, ny, nx).clone()
    p[..., 0], p[..., -1] = 1.0, outlet
    minv = free / diag.clamp_min(1e-300)
    for _ in range(3):       # restarted: the residual is taken anew
        r = -apply(p) * free
        z = minv * r
        d, rz = z.clone(), (r * z).sum()
        stop = None
        for it in range(6000):
            q = apply(d) * free
            al = rz / (d * q).sum()
            p += al * d
            r -= al * q
            z = minv * r
            new = (r * z).sum()
            d = z + (new / rz) * d
            rz = new
            if it % 50 == 49:
                v = float(new)
                stop = v if stop is None else stop
                if not v > 1e-26 * stop:
                    break
    ph_ = _halo(p)
    vel = []
    for a, k in zip((2, 1, 0), kf):
        n = ph_.shape[a]
        v = torch.zeros_like(ph_)
        v.narrow(a, 0, n - 1).copy_(-k.narrow(a, 0, n - 1) / mu * (ph_.narrow(a, 1, n - 1) - ph_.narrow(a, 0, n - 1)))
        vel.append(torch.where(k != 0, v, torch.zeros_like(v)))
    return k0, kf, ph_, vel


def _sh(t, z, y, x):
    """The interior of a halo array, shifted."""
    nz, ny, nx = (n - 2 for n in t.shape)
    return t[1 + z:1 + z + nz, 1 + y:1 + y + ny, 1 + x:1 + x + nx]


def _exact_rates(p, ph, cc, vel):
    """dphase/dt and dconcent/dt of calcPhaseDeriv and calcConcentDeriv (dx = 1, no overshoot, rat = 0)."""
    F, Cc = _halo(ph), _halo(cc)
    lap = lambda t: (_sh(t, 0, 0, 1) + _sh(t, 0, 0, -1) + _sh(t, 0, 1, 0) + _sh(t, 0, -1, 0) +  # noqa: E731
                     _sh(t, 1, 0, 0) + _sh(t, -1, 0, 0) - 6 * _sh(t, 0, 0, 0)) / p.dx ** 2
    gx, gy, gz = (0.5 / p.dx * (_sh(F, *a) - _sh(F, *(-v for v in a))) for a in ((0, 0, 1), (0, 1, 0), (1, 0, 0)))
    g = torch.sqrt(gx * gx + gy * gy + gz * gz)
    th = torch.atan(gy / (gx + 1e-20))
    fi = torch.acos((gz / (g + 1e-20)).clamp(-1, 1))
    c, s = torch.cos(th), torch.sin(th)
    w = 2 * p.dx * (1 + p.epsilon * (7 * c ** 4 - 6 * c ** 2 + s ** 4 * torch.cos(4 * fi)))
    u = [[_sh(vel[0], 0, 0, 0), _sh(vel[0], 0, 0, -1)], [_sh(vel[1], 0, 0, 0), _sh(vel[1], 0, -1, 0)],
         [_sh(vel[2], 0, 0, 0), _sh(vel[2], -1, 0, 0)]]
    tau = 5.0 / 3.0 * p.alpha * p.lambda_ * p.epsilon ** 2 / p.diffusion
    rate = ((1 - ph * ph) * (ph - p.lambda_ * cc) + w * w * lap(F)) / tau
    rate[..., 0] = rate[..., -1] = 0
    div = 0
    for (up, um), a in zip(u, ((0, 0, 1), (0, 1, 0), (1, 0, 0))):
        b = tuple(-v for v in a)
        div = div + up * torch.where(up > 0, cc, _sh(Cc, *a)) - um * torch.where(um > 0, _sh(Cc, *b), cc)
    conc = p.diffusion * lap(Cc) + p.alpha * rate - div / p.dx
    conc[..., 0] = conc[..., -1] = 0
    return rate, conc


def _pad0(t):
    return torch.nn.functional.pad(t, (1, 1, 1, 1, 1, 1))


def _np(t):
    return t.cpu().numpy().transpose(2, 1, 0)


def _conv64(x, w):
    """(C, z, y, x) input, [cout][27][cin] weights."""
    cout, _, cin = w.shape
    k = w.reshape(cout, 3, 3, 3, cin).permute(0, 4, 1, 2, 3)
    return torch.nn.functional.conv3d(x[None], k, padding=1)[0]


def _net64(par, x):
    """The U-Net with its BF16-stored weights and no rounding in between."""
    cin, cout = (16, 16, 32, 64, 64, 32, 16), (16, 32, 64, 64, 32, 16, 16)
    at, ws = 0, []
    for a, b in zip(cin, cout):
        w, bias = par[at:at + 27 * a * b].reshape(b, 27, a), par[at + 27 * a * b:at + 27 * a * b + b]
        at += 27 * a * b + b
        ws.append((w, bias[:, None, None, None]))
    layer = lambda n, t: _conv64(t, ws[n][0]) + ws[n][1]  # noqa: E731
    pool = lambda t: torch.nn.functional.avg_pool3d(t[None], 2)[0]  # noqa: E731
    up = lambda t: t.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)  # noqa: E731
    y0 = torch.relu(layer(0, x))
    y1 = torch.relu(layer(1, pool(y0)))
    y2 = torch.relu(layer(2, pool(y1)))
    y3 = torch.relu(layer(3, pool(y2)))
    y4 = torch.relu(layer(4, up(y3) + y2))
    y5 = torch.relu(layer(5, up(y4) + y1))
    return layer(6, up(y5) + y0)[0]


def _stored(par):
    """The parameters as the kernels use them: BF16 weights, FP32 biases."""
    cin, cout = (16, 16, 32, 64, 64, 32, 16), (16, 32, 64, 64, 32, 16, 16)
    q, at = par.clone(), 0
    for a, b in zip(cin, cout):
        q[at:at + 27 * a * b] = par[at:at + 27 * a * b].bfloat16().float()
        at += 27 * a * b + b
    return q.double()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "ensemble"):
        return None      # many steps, each with a solve of its own
    if kind == "diag":
        shape = _shape(case)
        kr, ph, cc = _fields(shape, case, "late", seed)
        p = _params(shape, case["kwh"]).params
        nx, ny, nz = shape
        z, y, x = torch.meshgrid(*[torch.arange(n, dtype=torch.float64, device="cuda") for n in (nz, ny, nx)],
                                 indexing="ij")
        r2 = p.dx ** 2 * ((x - (p.ix_ref - 1)) ** 2 + (y - (p.iy_ref - 1)) ** 2 + (z - (p.iz_ref - 1)) ** 2)
        d = dict(pv=p.dx ** 3 * p.porosity * 0.5 * float((1 - ph).sum()),
                 vcal=p.dx ** 3 * (1 - p.porosity) * 0.5 * float((1 + ph).sum()),
                 rwhmax=math.sqrt(float(torch.where(ph > 0, r2, torch.zeros_like(r2)).max())),
                 phase_max=float(ph.max()), phase_min=float(ph.min()), concent_max=float(cc.max()),
                 concent_min=float(cc.min()), pressure_ref=0.0, inlet_flux=0.0, phase_max_outlet=math.nan)
        if not case["noalloc"]:
            pr = _solution_guess(shape, kr, ph, case["kwh"])
            k = [case["kwh"] * 0.5 * (1 + ph[..., i]) + kr[..., i] * (1 - 0.5 * (1 + ph[..., i])) for i in (0, 1)]
            t = 2 * k[0] * k[1] / (k[0] + k[1]) / p.viscosity
            # the well planes hold the wells' pressures
            first = pr[..., 1] if nx > 2 else torch.full_like(pr[..., 0], 1e-300)
            d.update(pressure_ref=1.0 if p.ix_ref == 1 else float(pr[p.iz_ref - 1, p.iy_ref - 1, p.ix_ref - 1]),
                     inlet_flux=float((-t * (first - 1.0)).sum()) * p.dx,
                     phase_max_outlet=float(ph[..., max(1, nx - math.ceil(2 * p.epsilon / p.dx)) - 1].max()))
        return d
    if kind in ("routines", "solve"):
        shape = _shape(case)
        kr, ph, cc = _fields(shape, case, "early" if kind == "solve" else "late", seed)
        p = _params(shape, case["kwh"]).params
        k0, kf, pr, vel = _exact_flow(kr, ph, case["kwh"], p.viscosity, p.wells[-1].pressure)
        velocity = np.stack([_np(v) for v in vel])
        if kind == "solve":
            return dict(pressure=_np(pr), velocity=velocity)
        rate, conc = _exact_rates(p, ph, cc, vel)
        return dict(phase=_np(_halo(ph + 0.05 * rate)), concent=_np(_halo(cc + 0.05 * conc)),
                    dphasedt=_np(_pad0(rate)), dconcentdt=_np(_pad0(conc)), pressure=_np(pr), velocity=velocity,
                    permeab=np.stack([_np(t) for t in [k0] + kf]))
    nx, ny, nz = _shape(case)
    if kind == "conv3d":
        s = _conv_state(case, seed)
        x = s["x"].double().reshape(nz, ny, nx, -1).permute(3, 0, 1, 2)
        if case["op"] == "forward":
            y = torch.relu(_conv64(x, s["w"].double()) + s["b"].double()[:, None, None, None])
            return y.permute(1, 2, 3, 0).reshape(-1, case["cout"])
        gy = s["gy"].double()
        xp = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
        gw = torch.stack([gy.t() @ xp[:, k:k + nz, j:j + ny, i:i + nx].reshape(case["cin"], -1).t()
                          for k in range(3) for j in range(3) for i in range(3)], 1)
        return [gw, gy.sum(0)]
    x, target = _net_inputs(case, seed)
    x = x.double().reshape(nz, ny, nx, 16).permute(3, 0, 1, 2)
    par = _stored(torch.from_numpy(WarmStartNet.load_params(DEFAULT_WEIGHTS)).cuda())
    if kind == "forward":
        return _net64(par, x).reshape(-1)
    par.requires_grad_(True)
    loss = ((_net64(par, x).reshape(-1) - target.double()) ** 2).mean()
    loss.backward()
    return dict(loss=float(loss), grads=par.grad, params=None)
