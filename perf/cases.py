"""What this framework's speed is judged by: the work that its users have it do.

``listed()`` names the workloads, ``draw(rng)`` gives more of the same ranges,
``prepare`` / ``run`` hold one program's state and one pass through the public
entry points, ``work`` the bytes and operations a pass cannot do without, and
``exact`` the result in 64 bits from plain torch, where one fits.

The kinds of work:

* ``forecast``: an ensemble member's forecast segment.  The analysis (the
  prognostic fields of the synthetic moist state of
  :mod:`pywrf_b200.synthetic`, with seeded precipitating cloud bands) is
  copied from device memory into the member's state, then the segment's
  steps are replayed (``Integrator.run``).
* ``wsm6``: the reference-signature ``microphysics_driver`` on a column block
  with the same cloud bands, for a caller that keeps its own time loop.
* ``advect``: the differentiable scalar advection, forward and reverse.
* ``wsolve``: the implicit w solve with its coefficients, forward and reverse.
* ``train``: one optimiser step of the per-column network on a full batch.
* ``grad_step``: the gradient of a linear functional of the state after one
  whole step (WSM6 included) in the prognostic state before it, the unit of
  work of variational assimilation; eager, or captured once in a CUDA graph
  and replayed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pywrf_b200 import adjoint, synthetic
from pywrf_b200.config import Grid
from pywrf_b200.solver import Integrator
from pywrf_b200.state import DeviceState
from pywrf_b200.surrogate import MlpNet, Trainer
from pywrf_b200.wrf_physics import microphysics_driver

DEVICE = "cuda"
#: every field that one step reads from the step before it
CARRIED = ("u", "v", "w", "t", "ph", "mu", "p", "al", "moist", "h_diabatic", "status", "dscal")
#: what a forecast returns
FORECAST = ("u", "v", "w", "t", "ph", "mu", "p", "al", "moist", "h_diabatic", "rainnc")
#: the control variables of an assimilation, and the fields its functional weighs
CONTROL = ("u", "v", "w", "t", "ph", "mu", "p", "al", "moist")


def listed():
    return [
        # a teaching / regression-test domain: latency and launches are all there is
        dict(name="forecast_28x16", kind="forecast", n=28, nz=16, dt=45.0, soundsteps=4, nsteps=10),
        # a small nest, the 10-step configuration of the test suite
        dict(name="forecast_64x41", kind="forecast", n=64, nz=41, dt=45.0, soundsteps=4, nsteps=10),
        # a regional domain whose rows are no multiple of 16 bytes
        dict(name="forecast_131x35", kind="forecast", n=131, nz=35, dt=45.0, soundsteps=4, nsteps=4),
        # the 1-h regional integration of the benchmark (two of its steps)
        dict(name="forecast_240x41", kind="forecast", n=240, nz=41, dt=45.0, soundsteps=4, nsteps=2),
        # the large domain of the benchmark
        dict(name="forecast_512x61", kind="forecast", n=512, nz=61, dt=30.0, soundsteps=4, nsteps=1),
        # the microphysics alone, called by a solver that keeps its own loop
        dict(name="wsm6_240x41", kind="wsm6", n=240, nz=41, dt=45.0),
        # tracer transport in a gradient computation, odd rows
        dict(name="advect_151x37", kind="advect", n=151, nz=37),
        # the implicit vertical solve in a gradient computation
        dict(name="wsolve_240x41", kind="wsolve", n=240, nz=41),
        # one training step of the network at the batch the training uses
        dict(name="train_8192", kind="train", batch=8192, km=40, hidden=512),
        # assimilation on a regional domain with odd rows, captured once
        dict(name="grad_step_101x35", kind="grad_step", n=101, nz=35, dt=45.0, soundsteps=4, captured=True),
        # assimilation on the benchmark's domain, as a checkpointed rollout runs it
        dict(name="grad_step_240x41", kind="grad_step", n=240, nz=41, dt=45.0, soundsteps=4, captured=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("forecast", "forecast", "wsm6", "advect", "wsolve", "train", "grad_step"))
    if kind == "forecast":
        n, nz = _log_int(rng, 26, 440), rng.randint(16, 61)
        return dict(kind=kind, n=n, nz=nz, dt=rng.choice((30.0, 45.0)), soundsteps=rng.choice((4, 6)),
                    nsteps=10 if n < 100 else 3 if n < 200 else 1)
    if kind == "train":
        return dict(kind=kind, batch=128 * _log_int(rng, 8, 128), km=rng.randint(30, 60),
                    hidden=rng.choice((256, 512)))
    n, nz = _log_int(rng, 32, 240), rng.randint(16, 50)
    if kind == "wsm6":
        return dict(kind=kind, n=n, nz=nz, dt=rng.choice((30.0, 45.0, 150.0, 250.0)))
    if kind == "grad_step":
        small = n <= 128
        return dict(kind=kind, n=n, nz=nz, dt=rng.choice((30.0, 45.0)), soundsteps=4,
                    captured=small and rng.random() < 0.5)
    return dict(kind=kind, n=n, nz=nz)


# ---------------------------------------------------------------- inputs

def _spec(case, seed):
    return synthetic.CaseSpec(n=case["n"], nz=case["nz"], dt=case.get("dt", 45.0), soundsteps=case.get("soundsteps", 4),
                              bdy_tend_amp=1.0e-4, seed=int(seed))


def _weather(spec):
    """The synthetic moist state with precipitating cloud bands: about a
    fifth of the columns hold all five condensates at the temperatures where
    they occur, and are close to saturation there."""
    inputs, bdy = synthetic.build(spec)
    rng = np.random.default_rng([spec.seed, 77])
    _, km, m, _ = inputs["T"].shape
    x = np.arange(m) / m
    wave = np.zeros((m, m))
    for _ in range(6):
        kx, ky, ph = rng.integers(1, 5), rng.integers(0, 5), rng.uniform(0.0, 2.0 * np.pi, 2)
        wave += np.sin(2.0 * np.pi * kx * x + ph[0])[None, :] * np.cos(2.0 * np.pi * ky * x + ph[1])[:, None]
    rise = np.clip(wave - np.quantile(wave, 0.8), 0.0, None)
    cloud = (rise / max(rise.max(), 1e-9)).astype(np.float32)[None]
    p = inputs["PB"][0] + inputs["P"][0]
    temp = (inputs["T"][0] + np.float32(300.0)) * (p / np.float32(1.0e5)) ** np.float32(287.0 / 1004.5)
    warm = np.clip((temp - 263.0) / 20.0, 0.0, 1.0)
    cold = np.clip((275.0 - temp) / 20.0, 0.0, 1.0) * (temp > 220.0)
    noise = rng.uniform(0.5, 1.5, (5, m, m)).astype(np.float32)
    for i, (name, amount) in enumerate((("QCLOUD", 8e-4 * warm), ("QRAIN", 1e-3 * warm), ("QICE", 8e-5 * cold),
                                        ("QSNOW", 8e-4 * cold), ("QGRAUP", 4e-4 * cold))):
        inputs[name] = (inputs[name] + (cloud * noise[i] * amount)[None]).astype(np.float32)
    inputs["QVAPOR"] = (inputs["QVAPOR"] * (1.0 + 0.25 * cloud * (warm + cold > 0.0))[None]).astype(np.float32)
    return inputs, bdy


def _frame(a, nz, n):
    """A mass-point array in the solver's 5-cell frame on the device."""
    out = torch.zeros(nz, n, n, device=DEVICE)
    out[:a.shape[0], 5:n - 6, 5:n - 6] = torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEVICE)
    return out


def _levels(case):
    lev = synthetic._eta_levels(case["nz"])
    out = {}
    for k in ("fnm", "fnp", "rdnw", "rdn"):
        v = np.zeros(case["nz"], np.float32)
        v[:-1] = lev[k]
        out[k] = v
    return out


def _generator(seed, salt):
    return torch.Generator(device=DEVICE).manual_seed(1000003 * int(seed) + salt)


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEVICE)


def _advect_inputs(case, seed):
    """A smooth positive tracer with noise, mass fluxes of about 10 m/s, the
    eta-coordinate flux, and the reverse's cotangent."""
    gen, n, nz = _generator(seed, 1), case["n"], case["nz"]
    x = torch.arange(n, device=DEVICE) / n
    ph = 6.283 * torch.rand(4, generator=gen, device=DEVICE)
    wave = torch.sin(18.8 * x + ph[0])[None, None, :] * torch.cos(12.6 * x + ph[1])[None, :, None]
    f = dict(field=(1.0 + 0.5 * wave + 0.1 * _randn(gen, nz, n, n)).contiguous(),
             tendency=_randn(gen, nz, n, n),
             ru=9.0e5 * (1.0 + wave) + 5.0e4 * _randn(gen, nz, n, n), rv=3.0e5 * _randn(gen, nz, n, n),
             rom=50.0 * _randn(gen, nz, n, n))
    f["rom"][0] = 0.0
    f["rom"][nz - 1] = 0.0
    f["msftx"] = 1.0 + 0.05 * torch.rand(n, n, generator=gen, device=DEVICE)
    for k, v in _levels(case).items():
        f[k] = torch.from_numpy(v).to(DEVICE)
    f["cot"] = _randn(gen, nz, n, n)
    return f


def _wsolve_inputs(case, seed):
    """Column mass, water loading, c2a = (cp/cv) p / alpha of a standard
    column, the right-hand side of w and the reverse's cotangent."""
    gen, n, nz = _generator(seed, 2), case["n"], case["nz"]
    znu = torch.linspace(0.995, 0.005, nz, device=DEVICE)[:, None, None]
    mut = 9.4e4 + 1.0e3 * _randn(gen, n, n)
    p = 5.0e3 + znu * mut
    alt = 287.0 * (210.0 + 80.0 * znu + 2.0 * _randn(gen, nz, n, n)) / p
    f = dict(mut=mut, cqw=1.0 / (1.0 + 0.012 * znu * torch.rand(nz, n, n, generator=gen, device=DEVICE)),
             c2a=1.4 * p / alt, rhs=mut * _randn(gen, nz, n, n), cot=_randn(gen, nz, n, n))
    f = {k: v.contiguous() for k, v in f.items()}
    lev = _levels(case)
    return f | {k: torch.from_numpy(lev[k]).to(DEVICE) for k in ("rdn", "rdnw")}


def _train_inputs(case, seed):
    """A network of the case's column layout and one standardised batch."""
    km = case["km"]
    nfeat, nout = 9 * km, 7 * km + 3
    lay = dict(km=km, ncx=0, ncy=0, ncols=case["batch"], nfeat=nfeat, d0=(nfeat + 63) // 64 * 64, nout=nout,
               d4=(nout + 63) // 64 * 64)
    gen = _generator(seed, 3)
    net = MlpNet(lay, hidden=case["hidden"], device=DEVICE, seed=int(seed))
    x = _randn(gen, case["batch"], lay["d0"])
    x[:, nfeat:] = 0.0
    t = _randn(gen, case["batch"], lay["d4"])
    t[:, nout:] = 0.0
    return net, x.to(torch.bfloat16), t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "forecast":
        spec = _spec(case, seed)
        inputs, bdy = _weather(spec)
        member = DeviceState.from_inputs(synthetic.grid_for(spec), inputs, bdy, device=DEVICE)
        s = dict(integrator=Integrator(member), state=member,
                 analysis=[member[k].clone() for k in CARRIED], fields=[member[k] for k in CARRIED])
        s["integrator"].capture()
    elif kind == "wsm6":
        spec = _spec(case, seed)
        i, _ = _weather(spec)
        n, nz = case["n"], case["nz"]
        p = i["PB"][0] + i["P"][0]
        pii = (p / np.float32(1.0e5)) ** np.float32(0.2857143)
        z = (i["PH"][0] + i["PHB"][0]) / np.float32(9.81)
        th = i["T"][0] + np.float32(300.0)
        given = dict(th=th, qv=i["QVAPOR"][0], qc=i["QCLOUD"][0], qr=i["QRAIN"][0], qi=i["QICE"][0], qs=i["QSNOW"][0],
                     qg=i["QGRAUP"][0], rho=p / (np.float32(287.0) * th * pii), pii=pii, p=p, dz=z[1:] - z[:-1])
        s = dict(given={k: _frame(v, nz, n) for k, v in given.items()},
                 rain={k: torch.zeros(n, n, device=DEVICE)
                       for k in ("rainnc", "rainncv", "snownc", "snowncv", "sr", "graupelnc", "graupelncv")})
        s["work"] = {k: s["given"][k].clone() for k in ("th", "qv", "qc", "qr", "qi", "qs", "qg")}
        s["refl"] = torch.zeros(nz, n, n, device=DEVICE)
    elif kind == "advect":
        s = _advect_inputs(case, seed)
        for k in ("field", "tendency", "ru", "rv", "rom"):
            s[k].requires_grad_(True)
    elif kind == "wsolve":
        s = _wsolve_inputs(case, seed)
        for k in ("mut", "cqw", "c2a", "rhs"):
            s[k].requires_grad_(True)
    elif kind == "train":
        net, x, t = _train_inputs(case, seed)
        s = dict(net=net, trainer=Trainer(net, batch=case["batch"]), x=x, t=t)
    else:
        s = _prepare_grad(case, seed)
    s["case"] = case
    return s


def _prepare_grad(case, seed):
    spec = _spec(case, seed)
    inputs, bdy = _weather(spec)
    g = synthetic.grid_for(spec)
    st = DeviceState.from_inputs(g, inputs, bdy, device=DEVICE)
    names = tuple(dict.fromkeys(adjoint.RK_STATE + ("u_1", "w_1", "ph_1", "mu_1", "t_1", "v_1")))
    state = {k: st[k] for k in names}
    for k in CONTROL:
        state[k] = st[k].clone().requires_grad_(True)
    data = {k: st[k] for k in dict.fromkeys(adjoint.STEP_DATA + ("alb", "pb", "phb", "rdnw"))}
    keys = (("bxs", "xs"), ("bxe", "xe"), ("bys", "ys"), ("bye", "ye"), ("btxs", "txs"), ("btxe", "txe"),
            ("btys", "tys"), ("btye", "tye"))
    bd = {f: {key: st[f"{f}_{n}"] for n, key in keys} for f in ("u", "v", "ph", "t", "mu", "qv")}
    scal = dict(epssm=g.epssm, emdiv=g.emdiv, smdiv=g.smdiv, rdx=g.rdx, rdy=g.rdy, **st.scal)
    gen = _generator(seed, 4)
    # the functional weighs the points that hold the model's state
    inside = torch.zeros(g.ny, g.nx, device=DEVICE)
    inside[5:g.ny - 6, 5:g.nx - 6] = 1.0
    cot = [_randn(gen, *st[k].shape) * inside for k in CONTROL]
    s = dict(grid=g, state=state, data=data, bdy=bd, scal=scal, cot=cot, result=None)
    if case["captured"]:
        s["graph"] = adjoint.capture(lambda: _gradient(s))
    return s


def _gradient(s):
    g = s["grid"]
    out = adjoint.step(s["state"], s["data"], s["bdy"], g.dt, dt=g.dt, soundsteps=g.soundsteps,
                       microphysics=lambda q: adjoint.microphysics(q, s["data"], g.dt, g.rdx, g.rdy), **s["scal"])
    after = [out[k] for k in CONTROL]
    grads = torch.autograd.grad(after, [s["state"][k] for k in CONTROL], grad_outputs=s["cot"])
    s["result"] = {k: a.detach() for k, a in zip(CONTROL, after)} | {"grad_" + k: b for k, b in zip(CONTROL, grads)}
    return s["result"]


# ---------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "forecast":
        torch._foreach_copy_(s["fields"], s["analysis"])
        s["integrator"].run(case["nsteps"])
        return {k: s["state"][k] for k in FORECAST}
    if kind == "wsm6":
        q, w, r = s["given"], s["work"], s["rain"]
        torch._foreach_copy_(list(w.values()), [q[k] for k in w])
        torch._foreach_zero_(list(r.values()))
        n, nz = case["n"], case["nz"]
        tile = (6, n - 6, 6, n - 6, 0, nz)
        microphysics_driver(w["th"], q["rho"], q["pii"], q["p"], None, q["dz"], None, case["dt"], 9000.0, 9000.0,
                            w["qv"], w["qc"], w["qr"], w["qi"], w["qs"], w["qg"], r["rainnc"], r["rainncv"],
                            r["snownc"], r["snowncv"], r["sr"], s["refl"], 0, 0, r["graupelnc"], r["graupelncv"],
                            0, 0, 0, None, None, None, *tile, 0, n, 0, n, 0, nz, *tile)
        return w | r
    if kind == "advect":
        out = adjoint.advect_scalar(s["field"], s["tendency"], s["ru"], s["rv"], s["rom"], s["msftx"], s["fnm"],
                                    s["fnp"], s["rdnw"], 1.0 / 9000.0, 1.0 / 9000.0)
        names = ("field", "tendency", "ru", "rv", "rom")
        grads = torch.autograd.grad(out, [s[k] for k in names], grad_outputs=s["cot"])
        return {"out": out.detach()} | dict(zip(names, grads))
    if kind == "wsolve":
        a, alpha, gamma = adjoint.coef_w(s["mut"], s["cqw"], s["c2a"], s["rdn"], s["rdnw"], 11.25)
        w = adjoint.vsolve_w(s["rhs"], a, alpha, gamma)
        names = ("mut", "cqw", "c2a", "rhs")
        grads = torch.autograd.grad(w, [s[k] for k in names], grad_outputs=s["cot"])
        return {"w": w.detach(), "alpha": alpha.detach()} | dict(zip(names, grads))
    if kind == "train":
        net, tr = s["net"], s["trainer"]
        tr.loss.zero_()
        tr.step(s["x"], s["t"])
        return {"y": tr.y, "loss": tr.loss, "mw": net.mw, "mb": net.mb}
    if case["captured"]:
        s["graph"].replay()
        return s["result"]
    return _gradient(s)


# ---------------------------------------------------------------- what a pass needs

def work(case):
    """Inputs read once and outputs written once, and the operations of the
    formulas (a power, logarithm or exponential counted as ten)."""
    kind = case["kind"]
    if kind == "train":
        km, b, h = case["km"], case["batch"], case["hidden"]
        d = [(9 * km + 63) // 64 * 64, h, h, h, (7 * km + 3 + 63) // 64 * 64]
        params = sum(d[i] * d[i + 1] + d[i + 1] for i in range(4))
        # batch in, prediction out; weights and both moments read and written
        return dict(bytes=b * (2 * d[0] + 8 * d[4]) + params * 24,
                    flops=2 * b * (3 * sum(d[i] * d[i + 1] for i in range(4)) - d[0] * d[1]))
    points = case["n"] ** 2 * case["nz"]
    if kind == "forecast":
        # per step: 15 fields of state in, 16 out (u v w t ph p al, six
        # species, h_diabatic, pb phb alb t_init in); three stages of
        # advection and tendencies, the substeps, the microphysics
        sub = 1 + case["soundsteps"] // 2 + case["soundsteps"]
        return dict(bytes=4 * points * (18 + 14) * case["nsteps"],
                    flops=points * (3 * 1300 + 220 * sub + 1500) * case["nsteps"])
    if kind == "wsm6":
        return dict(bytes=4 * points * (11 + 7), flops=points * 1500)
    if kind == "advect":
        return dict(bytes=4 * points * (6 + 5), flops=points * 300)
    if kind == "wsolve":
        return dict(bytes=4 * points * (4 + 5), flops=points * 90)
    # one step and its reverse: the state and the cotangents in, the state
    # and the gradients out
    sub = 1 + case["soundsteps"] // 2 + case["soundsteps"]
    return dict(bytes=4 * points * (18 + 14 + 14 + 14), flops=4 * points * (3 * 1300 + 220 * sub + 1500))


# ---------------------------------------------------------------- 64-bit results

def _flux5(q, lo, hi, dim, v, up):
    """5th-order upwind-biased face values times v at the faces [lo, hi) of
    ``dim`` (between cell f - 1 and f), with the sign of ``up``."""
    c = [q.narrow(dim, lo + o, hi - lo) for o in (-3, -2, -1, 0, 1, 2)]
    even = (37.0 * (c[3] + c[2]) - 8.0 * (c[4] + c[1]) + (c[5] + c[0])) / 60.0
    odd = ((c[5] - c[0]) - 5.0 * (c[4] - c[1]) + 10.0 * (c[3] - c[2])) / 60.0
    return v * (even - torch.where(up >= 0, 1.0, -1.0) * odd)


def _flux3(q, f, dim, v, up):
    """The 3rd-order face value times v at face f."""
    c = [q.narrow(dim, f + o, 1) for o in (-2, -1, 0, 1)]
    even = (7.0 * (c[2] + c[1]) - (c[3] + c[0])) / 12.0
    odd = ((c[3] - c[0]) - 3.0 * (c[2] - c[1])) / 12.0
    return v * (even + torch.where(up >= 0, 1.0, -1.0) * odd)


def _side_faces(q, vel, dim, sides_from):
    """The interior faces 6 .. end-2 of one horizontal direction: 2nd order
    at the outermost, 3rd at the next, 5th inside.  ``sides_from``: the face
    whose velocity gives the 3rd-order face at the far side its sign."""
    end = q.shape[dim] - 5
    at = lambda a, f: a.narrow(dim, f, 1)  # noqa: E731
    second = lambda f: 0.5 * at(vel, f) * (at(q, f) + at(q, f - 1))  # noqa: E731
    inner = vel.narrow(dim, 8, end - 11)
    return torch.cat([second(6), _flux3(q, 7, dim, at(vel, 7), at(vel, 7)), _flux5(q, 8, end - 3, dim, inner, inner),
                      _flux3(q, end - 3, dim, at(vel, end - 3), at(vel, sides_from)), second(end - 2)], dim)


def _exact_advect(case, seed):
    f = {k: v.double().cpu() for k, v in _advect_inputs(case, seed).items()}
    n, nz = case["n"], case["nz"]
    names = ("field", "tendency", "ru", "rv", "rom")
    for k in names:
        f[k].requires_grad_(True)
    kt, e, q = nz - 1, n - 5, f["field"][:nz - 1]
    fy = _side_faces(q[:, :, 5:e - 1], f["rv"][:kt, :, 5:e - 1], 1, e - 3)
    fx = _side_faces(q[:, 5:e - 1, :], f["ru"][:kt, 5:e - 1, :], 2, e - 2)
    m = f["msftx"]
    adv = torch.zeros(nz, n, n, dtype=torch.float64)
    y = torch.zeros_like(adv)
    y[:kt, 6:e - 2, 5:e - 1] = (m[6:e - 2, 5:e - 1] / 9000.0) * (fy[:, 1:] - fy[:, :-1])
    x = torch.zeros_like(adv)
    x[:kt, 5:e - 1, 6:e - 2] = (m[5:e - 1, 6:e - 2] / 9000.0) * (fx[:, :, 1:] - fx[:, :, :-1])
    qc, r = q[:, 5:e - 1, 5:e - 1], f["rom"][:, 5:e - 1, 5:e - 1]
    lin = lambda k: r[k:k + 1] * (f["fnm"][k] * qc[k:k + 1] + f["fnp"][k] * qc[k - 1:k])  # noqa: E731
    zero = torch.zeros_like(qc[:1])
    fz = torch.cat([zero, lin(1), _flux3(qc, 2, 0, r[2:3], -r[2:3]),
                    _flux5(qc, 3, kt - 2, 0, r[3:kt - 2], -r[3:kt - 2]),
                    _flux3(qc, kt - 2, 0, r[kt - 2:kt - 1], -r[kt - 2:kt - 1]), lin(kt - 1), zero])
    z = torch.zeros_like(adv)
    z[:kt, 5:e - 1, 5:e - 1] = f["rdnw"][:kt, None, None] * (fz[1:] - fz[:-1])
    out = f["tendency"] - y - x - z
    grads = torch.autograd.grad(out, [f[k] for k in names], grad_outputs=f["cot"])
    return {"out": out.detach()} | dict(zip(names, grads))


def _exact_wsolve(case, seed):
    f = {k: v.double().cpu() for k, v in _wsolve_inputs(case, seed).items()}
    n, nz = case["n"], case["nz"]
    names = ("mut", "cqw", "c2a", "rhs")
    for k in names:
        f[k].requires_grad_(True)
    R = (slice(5, n - 6), slice(5, n - 6))
    cof = (0.5 * 11.25 * 9.81 * 1.1) ** 2
    mm = f["mut"][R] ** 2
    cw, c2, rdn, rdnw = f["cqw"][(slice(None),) + R], f["c2a"][(slice(None),) + R], f["rdn"], f["rdnw"]
    zero = torch.zeros_like(mm)
    a, al, ga = [zero], [zero], [zero]
    top = nz - 1
    for k in range(1, nz):
        if k < top:
            lower = zero if k == 1 else -cw[k] * cof * rdn[k] * rdnw[k - 1] * c2[k - 1] / mm
            b = 1.0 + cw[k] * cof * rdn[k] * (rdnw[k] * c2[k] / mm + rdnw[k - 1] * c2[k - 1] / mm)
            c = -cw[k] * cof * rdn[k] * rdnw[k] * c2[k] / mm
        else:
            lower = -2.0 * cof * rdnw[top - 1] ** 2 * c2[top - 1] / mm
            b, c = 1.0 + 2.0 * cof * rdnw[top - 1] ** 2 * c2[top - 1] / mm, zero
        a.append(lower)
        al.append(1.0 / (b - lower * ga[k - 1]))
        ga.append(c * al[k])
    full = lambda v: torch.nn.functional.pad(torch.stack(v), (5, 6, 5, 6))  # noqa: E731
    alpha = full(al)
    A, G, x = full(a), full(ga), f["rhs"]
    y = [x[0]]
    for k in range(1, nz):
        y.append((x[k] - A[k] * y[k - 1]) * alpha[k])
    w = y[:1] + [None] * (nz - 2) + y[nz - 1:]
    for k in range(nz - 2, 0, -1):
        w[k] = y[k] - G[k] * w[k + 1]
    w = torch.stack(w)
    grads = torch.autograd.grad(w, [f[k] for k in names], grad_outputs=f["cot"])
    return {"w": w.detach(), "alpha": alpha.detach()} | dict(zip(names, grads))


def _exact_train(case, seed):
    net, x, t = _train_inputs(case, seed)
    w = [v.to(torch.bfloat16).double().requires_grad_(True) for v in net.w32]
    b = [v.double().requires_grad_(True) for v in net.b32]
    nout = net.layout["nout"]
    h = x.double()
    for i in range(3):
        h = torch.nn.functional.gelu(h @ w[i].t() + b[i], approximate="tanh")
    y = h @ w[3].t() + b[3]
    err = (y - t.double())[:, :nout].square()
    grads = torch.autograd.grad(err.mean(), w + b)
    # the running mean of the gradients after the first step is a tenth of them
    return {"y": y.detach(), "loss": err.sum().detach().reshape(1), "mw": [0.1 * g for g in grads[:4]],
            "mb": [0.1 * g for g in grads[4:]]}


def exact(case, seed):
    """The kinds that fit in plain torch; a whole step, its gradient and the
    microphysics scheme have no 64-bit form outside this repository."""
    if case["kind"] == "advect":
        return _exact_advect(case, seed)
    if case["kind"] == "wsolve":
        return _exact_wsolve(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None
