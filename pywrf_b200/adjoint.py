"""Hand-written adjoints of step operators behind ``torch.autograd.Function``.

The reference differentiates its step with PyTorch's taped autograd; here
each operator's reverse product is its own CUDA kernel
(include/pywrf_b200.h, ``wrf_*_adj``), so backpropagation through these
operators keeps no tape of the forward's intermediates.

* :class:`AdvectScalar` -- ``tendency + advect(field; ru, rv, rom)``
  (pywrf/wrf_dynamics.py:1841-2028); gradients with respect to the field, the
  incoming tendency and the three mass fluxes.
* :class:`AdvectMomentum` -- ``tendency + advect_u / advect_v / advect_w``
  (pywrf/wrf_dynamics.py:1112-1823); gradients with respect to the advected
  component, the incoming tendency and ru, rv, rom.
* :class:`AdvanceUV` -- advance_uv followed by spec_bdyupdate of u and v
  (pywrf/wrf_dynamics.py:3391-3525, pywrf/wrf_boundary.py:244-290), the
  horizontal-momentum part of the acoustic substep; gradients with respect to
  u, v, ru_tend, rv_tend, p, pb, ph, php, alt, al, mu, muu, muv, cqu, cqv and
  mudf (map factors and vertical profiles are data).
* :class:`CalcPRho` -- calc_p_rho (pywrf/wrf_dynamics.py:3269-3313): al, p,
  pm1 from ph, alt, t_2, t_1, c2a, pm1, mu, mut at a given acoustic step;
  gradients with respect to all ten.
* :class:`AdvanceMuT` -- advance_mu_t (pywrf/wrf_dynamics.py:3528-3638): the
  column mass, eta-velocity and theta update of the acoustic substep;
  gradients with respect to its 18 array inputs, either of the operator
  (default) or as the reference's autograd gives them (``ref_no_grad``: its
  mu / muts / mudf / muave update runs under ``torch.no_grad()``).
* :class:`AdvanceW` -- advance_w (pywrf/wrf_dynamics.py:3641-3796): the
  vertically implicit w / phi update with its terrain lower boundary and
  Rayleigh damping; gradients with respect to its 23 array inputs.
* :class:`Forces` -- the large-step tendency terms rhs_ph,
  horizontal_pressure_gradient, pg_buoy_w, coriolis and curvature
  (pywrf/wrf_dynamics.py:2031-2620), any subset by a mask; gradients with
  respect to the incoming tendencies, cqw (which pg_buoy_w overwrites) and the
  21 state arrays they read.
* :class:`Sumflux`, :class:`SpecUpdate`, :class:`SpecUpdatePh` -- sumflux
  (pywrf/wrf_dynamics.py:3799-3839), spec_bdyupdate and spec_bdyupdate_ph
  (pywrf/wrf_boundary.py:244-355), the rest of the acoustic substep.
* :class:`Prep` -- rk_step_prep's functions calculate_full, calc_mu_uv,
  couple_momentum, calc_ww_cp, calc_cq, calc_alt, calc_php
  (pywrf/wrf_dynamics.py:30-159), any subset by a mask.
* :class:`RelaxBdytend` -- ``tendency + relax(field)`` toward the lateral
  boundary values (pywrf/wrf_boundary.py:52-147); gradients with respect to
  the field and the incoming tendency (the boundary arrays are data).
* :class:`CoefW` -- calc_coef_w (pywrf/wrf_dynamics.py:3316-3388): the
  implicit solve's coefficients a, alpha, gamma from mut, cqw, c2a;
  gradients with respect to those three.
* :class:`VSolveW` -- the vertically implicit w solve of advance_w
  (pywrf/wrf_dynamics.py:3761-3767); gradients with respect to the
  right-hand side and the coefficients a, alpha, gamma (the transposed solve).
* :class:`HorizontalDiffusion`, :func:`eddy_viscosity`, :class:`MassWeight`
  -- the first RK stage's diffusion (pywrf/wrf_dynamics.py:2623-2915), the
  eddy viscosities (compute_diff_metrics, cal_deform_and_div,
  calculate_km_kh: :491-995) and mass_weight (pywrf/wrf_boundary.py:408).
* :func:`addtend`, :class:`SpecBdytend`, the moisture update
  (rk_update_scalar, flow_dep_bdy, calc_p_rho_phi), :func:`microphysics`
  (moist_physics_prep_em, WSM6, moist_physics_finish_em, calc_p_rho_phi;
  WSM6's sedimentation in reverse mode over tapes of a restatement, the rest
  of it per level by forward-mode tangents) and
  :func:`step_end` (halo copies, spec_bdy_final, set_w_surface).
* Composed in the reference's order: :func:`acoustic_substep`,
  :func:`acoustic_stage`, :func:`dynamics_stage`, :func:`moist_stage`,
  :func:`rk_stage` and :func:`step` (one whole time step,
  pywrf/solver.py:709-1910, with an optional theta-tendency bias).
* :func:`rollout` -- truncated backpropagation through ``n_steps`` of a
  step made of these operators with per-step (or per-segment) checkpointing:
  only each segment's input state is kept, and the backward pass recomputes
  the segment's forward once before back-propagating through it.
"""
from __future__ import annotations

import ctypes
import functools
from typing import Callable, Sequence

import torch
from torch.utils.checkpoint import checkpoint

from . import _native as N
from .config import Grid
from .state import make_cgrid


def _ptr(t: torch.Tensor) -> int:
    """The address of a contiguous float32 CUDA tensor."""
    if not (t.is_cuda and t.dtype is torch.float32 and t.is_contiguous()):
        raise TypeError("a contiguous float32 CUDA tensor is required (no CPU path)")
    return t.data_ptr()


# The device is named by its index: from a torch.device (or none at all)
# current_stream and device each take several microseconds to find it, which
# is most of what a small operator's call spends outside its kernels.
def _stream(t: torch.Tensor) -> int:
    """The handle of the stream that is current on the tensor's device."""
    return torch.cuda.current_stream(t.get_device()).cuda_stream


def _on(t: torch.Tensor):
    """The tensor's device as the current one."""
    return torch.cuda.device(t.get_device())


def _cuda_only(*ts) -> None:
    """Refuse anything but contiguous float32 CUDA tensors before any
    library or stream call (None entries are optional operands)."""
    for t in ts:
        if t is not None:
            _ptr(t)


def scalar_grid(shape, rdx: float, rdy: float):
    """The C grid record of the solver's 5-cell frame for a field of ``shape``
    (the caller's own copy)."""
    return N.WrfGridC.from_buffer_copy(_frame(tuple(shape), float(rdx), float(rdy)))


@functools.lru_cache(maxsize=64)
def _frame(shape, rdx: float, rdy: float):
    nz, ny, nx = shape
    g = Grid.make(nx, ny, nz, 1.0 / float(rdx), 1.0 / float(rdy), 1.0)
    cg = make_cgrid(g, {"cf1": 0.0, "cf2": 0.0, "cf3": 0.0, "cfn": 0.0, "cfn1": 0.0})
    cg.dx = 1.0 / float(rdx)
    cg.dy = 1.0 / float(rdy)
    return cg


@functools.lru_cache(maxsize=64)
def _advect_work_floats(shape) -> int:
    n = ctypes.c_size_t(0)
    N.check(N.lib().wrf_advect_scalar_adj_work(ctypes.byref(_frame(shape, 1.0, 1.0)), ctypes.byref(n)), "work")
    return n.value


class AdvectScalar(torch.autograd.Function):
    """out = tendency + flux-form advection of ``field`` by (ru, rv, rom)."""

    @staticmethod
    def forward(ctx, field, tendency, ru, rv, rom, msftx, fnm, fnp, rdnw, rdx: float, rdy: float):
        q, _, *rest = [_ptr(t) for t in (field, tendency, ru, rv, rom, msftx, fnm, fnp, rdnw)]
        cg = scalar_grid(field.shape, rdx, rdy)
        out = tendency.detach().clone()
        stream = _stream(field)
        with _on(field):
            rc = N.lib().wrf_advect_scalar(ctypes.byref(cg), q, out.data_ptr(), *rest, stream)
        N.check(rc, "wrf_advect_scalar")
        ctx.save_for_backward(field, ru, rv, rom, msftx, fnm, fnp, rdnw)
        ctx.cg = cg
        return out

    @staticmethod
    def backward(ctx, gout):
        field, ru, rv, rom, msftx, fnm, fnp, rdnw = ctx.saved_tensors
        gout = gout.contiguous()
        qb, rub, rvb, romb = _zeros(field, field, field, field)
        n = _advect_work_floats(tuple(field.shape))
        work = torch.empty(n, dtype=torch.float32, device=field.device)
        stream = _stream(field)
        with _on(field):
            rc = N.lib().wrf_advect_scalar_adj(ctypes.byref(ctx.cg), _ptr(field), _ptr(ru), _ptr(rv), _ptr(rom),
                                               _ptr(msftx), _ptr(fnm), _ptr(fnp), _ptr(rdnw), _ptr(gout), _ptr(qb),
                                               _ptr(rub), _ptr(rvb), _ptr(romb), _ptr(work), n, stream)
        N.check(rc, "wrf_advect_scalar_adj")
        return qb, gout, rub, rvb, romb, None, None, None, None, None, None


def advect_scalar(field, tendency, ru, rv, rom, msftx, fnm, fnp, rdnw, rdx, rdy):
    """Differentiable ``tendency + advect(field)`` on the GPU."""
    return AdvectScalar.apply(field, tendency, ru, rv, rom, msftx, fnm, fnp, rdnw, rdx, rdy)


class AdvectMomentum(torch.autograd.Function):
    """out = tendency + flux-form advection of one momentum component
    (0 u with msf = msfux, 1 v with msf = msfvy and msf2 = msfvx, 2 w with
    msf = msftx; rdz = rdnw for u and v, rdn for w)."""

    @staticmethod
    def forward(ctx, component: int, field, tendency, ru, rv, rom, msf, msf2, fzm, fzp, rdz, rdx: float, rdy: float):
        _cuda_only(field, tendency, ru, rv, rom, msf, msf2, fzm, fzp, rdz)
        if component not in (0, 1, 2):
            raise ValueError("component must be 0 (u), 1 (v) or 2 (w)")
        if component == 1 and msf2 is None:
            raise ValueError("advect_v needs msf2 (msfvx)")
        cg = scalar_grid(field.shape, rdx, rdy)
        out = tendency.detach().clone()
        m2 = _ptr(msf2) if msf2 is not None else None
        stream = _stream(field)
        with _on(field):
            rc = N.lib().wrf_advect_momentum(ctypes.byref(cg), int(component), _ptr(field), _ptr(out), _ptr(ru),
                                             _ptr(rv), _ptr(rom), _ptr(msf), m2, _ptr(fzm), _ptr(fzp), _ptr(rdz),
                                             0, stream)
        N.check(rc, "wrf_advect_momentum")
        ctx.save_for_backward(field, ru, rv, rom, msf, msf if msf2 is None else msf2, fzm, fzp, rdz)
        ctx.cg, ctx.component, ctx.has_msf2 = cg, int(component), msf2 is not None
        return out

    @staticmethod
    def backward(ctx, gout):
        field, ru, rv, rom, msf, msf2, fzm, fzp, rdz = ctx.saved_tensors
        gout = gout.contiguous()
        qb, rub, rvb, romb = _zeros(field, field, field, field)
        m2 = _ptr(msf2) if ctx.has_msf2 else None
        n = ctypes.c_size_t(0)
        N.check(N.lib().wrf_advect_momentum_adj_work(ctypes.byref(ctx.cg), ctypes.byref(n)), "work")
        work = torch.empty(int(n.value), dtype=torch.float32, device=field.device)
        stream = _stream(field)
        with _on(field):
            rc = N.lib().wrf_advect_momentum_adj(ctypes.byref(ctx.cg), ctx.component, _ptr(field), _ptr(ru), _ptr(rv),
                                                 _ptr(rom), _ptr(msf), m2, _ptr(fzm), _ptr(fzp), _ptr(rdz), _ptr(gout),
                                                 _ptr(qb), _ptr(rub), _ptr(rvb), _ptr(romb), _ptr(work), n, stream)
        N.check(rc, "wrf_advect_momentum_adj")
        return None, qb, gout, rub, rvb, romb, None, None, None, None, None, None, None


def advect_momentum(component, field, tendency, ru, rv, rom, msf, msf2, fzm, fzp, rdz, rdx, rdy):
    """Differentiable ``tendency + advect_{u,v,w}(field)`` on the GPU
    (component 0, 1, 2)."""
    return AdvectMomentum.apply(component, field, tendency, ru, rv, rom, msf, msf2, fzm, fzp, rdz, rdx, rdy)


UV_INPUTS = ("u", "v", "ru_tend", "rv_tend", "p", "pb", "ph", "php", "alt", "al", "mu", "muu", "muv", "cqu", "cqv",
             "mudf")
UV_DATA = ("msfux", "msfuy", "msfvx", "msfvx_inv", "msfvy", "fnm", "fnp", "rdnw")


def _table(named: dict):
    """A state table (WrfState) holding the given fields by name."""
    index = _field_index()
    arr = (ctypes.c_void_p * len(index))()
    for k, t in named.items():
        if not (t.is_cuda and t.dtype is torch.float32 and t.is_contiguous()):
            raise TypeError("a contiguous float32 CUDA tensor is required (no CPU path)")
        arr[index[k]] = t.data_ptr()
    return arr


@functools.lru_cache(maxsize=1)
def _field_index() -> dict:
    return {k: q for q, k in enumerate(N.field_names())}


def _zeros(*likes):
    """Zero float32 tensors shaped like ``likes``, carved (at 256-byte
    aligned offsets) from one buffer that a single fill clears: one launch
    instead of one per cotangent buffer."""
    if not likes:
        return []
    sizes = [(t.numel() + 63) // 64 * 64 for t in likes]
    buf = torch.zeros(sum(sizes), dtype=torch.float32, device=likes[0].device)
    out, o = [], 0
    for t, n in zip(likes, sizes):
        out.append(torch.as_strided(buf, t.shape, _packed(t), o))
        o += n
    return out


def _packed_like(t: torch.Tensor) -> torch.Tensor:
    """An uninitialised tensor like ``t``, its points without gaps."""
    return torch.empty_like(t, memory_format=torch.contiguous_format)


def _packed(t: torch.Tensor) -> tuple:
    """The strides of ``t``'s shape without gaps."""
    if t.is_contiguous():
        return t.stride()
    s = [1]
    for n in reversed(t.shape[1:]):
        s.append(s[-1] * n)
    return tuple(reversed(s))


def _bars(named: dict, fields, grads: dict) -> dict:
    """Cotangent buffers for ``fields``: a clone of the incoming gradient
    where ``grads`` holds one (the adjoint rewrites it in place), zeros from
    one shared buffer for the rest."""
    rest = [k for k in fields if grads.get(k) is None]
    bars = dict(zip(rest, _zeros(*[named[k] for k in rest])))
    for k in fields:
        if k not in bars:
            bars[k] = grads[k].contiguous().clone()
    return bars


class AdvanceUV(torch.autograd.Function):
    """(u', v') = advance_uv + spec_bdyupdate(u), (v); the tensors follow
    UV_INPUTS then UV_DATA, ``scal`` = (dts, emdiv, cf1, cf2, cf3, rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, *tensors):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        _cuda_only(*tensors)
        dts, emdiv, cf1, cf2, cf3, rdx, rdy = (float(x) for x in scal)
        named = dict(zip(UV_INPUTS + UV_DATA, tensors))
        cg = scalar_grid(named["u"].shape, rdx, rdy)
        cg.emdiv, cg.cf1, cg.cf2, cg.cf3 = emdiv, cf1, cf2, cf3
        u_new, v_new = named["u"].detach().clone(), named["v"].detach().clone()
        tab = _table({**named, "u": u_new, "v": v_new})
        stream = _stream(u_new)
        with _on(u_new):
            rc = N.lib().wrf_advance_uv(ctypes.byref(cg), tab, dts, stream)
        N.check(rc, "wrf_advance_uv")
        ctx.save_for_backward(*tensors)
        ctx.cg, ctx.dts = cg, dts
        return u_new, v_new

    @staticmethod
    def backward(ctx, gu, gv):
        tensors = ctx.saved_tensors
        named = dict(zip(UV_INPUTS + UV_DATA, tensors))
        bars = _bars(named, UV_INPUTS[2:] + tuple(k for k, gk in (("u", gu), ("v", gv)) if gk is None), {})
        gu = bars["u"] if gu is None else gu.contiguous()
        gv = bars["v"] if gv is None else gv.contiguous()
        tab = _table(named)
        btab = _table({"u": gu, "v": gv, **bars})
        stream = _stream(gu)
        with _on(gu):
            rc = N.lib().wrf_advance_uv_adj(ctypes.byref(ctx.cg), tab, btab, ctx.dts, stream)
        N.check(rc, "wrf_advance_uv_adj")
        return (None, gu, gv) + tuple(bars[k] for k in UV_INPUTS[2:]) + (None,) * len(UV_DATA)


def advance_uv(inputs: dict, data: dict, dts, emdiv, cf1, cf2, cf3, rdx, rdy):
    """Differentiable advance_uv + spec_bdyupdate(u), (v) on the GPU:
    ``inputs`` maps UV_INPUTS, ``data`` UV_DATA to tensors; returns (u', v')."""
    return AdvanceUV.apply((dts, emdiv, cf1, cf2, cf3, rdx, rdy), *[inputs[k] for k in UV_INPUTS],
                           *[data[k] for k in UV_DATA])


FORCES_OUTPUTS = ("ph_tend", "ru_tend", "rv_tend", "rw_tend", "cqw")
FORCES_INPUTS = FORCES_OUTPUTS + ("u", "v", "w", "ww", "ph", "phb", "mut", "muu", "muv", "alt", "p", "pb", "al",
                                  "php", "cqu", "cqv", "mu", "mub", "ru", "rv", "rw")
FORCES_DATA = ("msfux", "msfuy", "msfvx", "msfvy", "msftx", "msfty", "f", "e", "sina", "cosa", "fnm", "fnp", "rdnw",
               "rdn")
FORCES_TERMS = {"rhs_ph": 1, "hpg": 2, "pg_buoy_w": 4, "coriolis": 8, "curvature": 16}


class Forces(torch.autograd.Function):
    """(ph_tend', ru_tend', rv_tend', rw_tend', cqw') = the tendency terms of
    the mask ``terms`` (rhs_ph 1, horizontal_pressure_gradient 2, pg_buoy_w 4,
    coriolis 8, curvature 16) added to the incoming tendencies; the tensors
    follow FORCES_INPUTS then FORCES_DATA, ``scal`` = (terms, rdx, rdy, cf1,
    cf2, cf3, cfn, cfn1)."""

    @staticmethod
    def forward(ctx, scal, *tensors):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        _cuda_only(*tensors)
        terms = int(scal[0])
        rdx, rdy, cf1, cf2, cf3, cfn, cfn1 = (float(x) for x in scal[1:])
        named = dict(zip(FORCES_INPUTS + FORCES_DATA, tensors))
        cg = scalar_grid(named["u"].shape, rdx, rdy)
        cg.cf1, cg.cf2, cg.cf3, cg.cfn, cg.cfn1 = cf1, cf2, cf3, cfn, cfn1
        outs = {k: named[k].detach().clone() for k in FORCES_OUTPUTS}
        tab = _table({**named, **outs})
        stream = _stream(outs["ph_tend"])
        with _on(outs["ph_tend"]):
            rc = N.lib().wrf_forces(ctypes.byref(cg), tab, terms, stream)
        N.check(rc, "wrf_forces")
        ctx.save_for_backward(*tensors)
        ctx.cg, ctx.terms = cg, terms
        return tuple(outs[k] for k in FORCES_OUTPUTS)

    @staticmethod
    def backward(ctx, *gouts):
        tensors = ctx.saved_tensors
        named = dict(zip(FORCES_INPUTS + FORCES_DATA, tensors))
        bars = _bars(named, FORCES_INPUTS, dict(zip(FORCES_OUTPUTS, gouts)))
        stream = _stream(bars["u"])
        with _on(bars["u"]):
            rc = N.lib().wrf_forces_adj(ctypes.byref(ctx.cg), _table(named), _table(bars), ctx.terms, stream)
        N.check(rc, "wrf_forces_adj")
        return (None,) + tuple(bars[k] for k in FORCES_INPUTS) + (None,) * len(FORCES_DATA)


def forces(inputs: dict, data: dict, terms, rdx, rdy, cf1, cf2, cf3, cfn, cfn1):
    """Differentiable tendency terms on the GPU: ``inputs`` maps
    FORCES_INPUTS, ``data`` FORCES_DATA to tensors; ``terms`` is a mask or a
    sequence of FORCES_TERMS names; returns (ph_tend', ru_tend', rv_tend',
    rw_tend', cqw')."""
    if not isinstance(terms, int):
        terms = sum(FORCES_TERMS[t] for t in terms)
    return Forces.apply((terms, rdx, rdy, cf1, cf2, cf3, cfn, cfn1), *[inputs[k] for k in FORCES_INPUTS],
                        *[data[k] for k in FORCES_DATA])


SF_INPUTS = ("ru_m", "rv_m", "ww_m", "u", "v", "ww", "u_save", "v_save", "ww1", "muu", "muv")
SF_DATA = ("msfuy", "msfvx_inv")


class Sumflux(torch.autograd.Function):
    """(ru_m', rv_m', ww_m') = sumflux at ``iteration`` of ``nsub``; the
    tensors follow SF_INPUTS then SF_DATA, ``scal`` = (iteration, nsub, rdx,
    rdy)."""

    @staticmethod
    def forward(ctx, scal, *tensors):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        _cuda_only(*tensors)
        iteration, nsub = int(scal[0]), int(scal[1])
        named = dict(zip(SF_INPUTS + SF_DATA, tensors))
        cg = scalar_grid(named["u"].shape, float(scal[2]), float(scal[3]))
        outs = {k: named[k].detach().clone() for k in SF_INPUTS[:3]}
        stream = _stream(named["u"])
        with _on(named["u"]):
            rc = N.lib().wrf_sumflux(ctypes.byref(cg), _table({**named, **outs}), iteration, nsub, stream)
        N.check(rc, "wrf_sumflux")
        ctx.save_for_backward(*tensors)
        ctx.cg, ctx.it = cg, (iteration, nsub)
        return tuple(outs[k] for k in SF_INPUTS[:3])

    @staticmethod
    def backward(ctx, *gouts):
        named = dict(zip(SF_INPUTS + SF_DATA, ctx.saved_tensors))
        bars = _bars(named, SF_INPUTS, dict(zip(SF_INPUTS[:3], gouts)))
        stream = _stream(bars["u"])
        with _on(bars["u"]):
            rc = N.lib().wrf_sumflux_adj(ctypes.byref(ctx.cg), _table(named), _table(bars), ctx.it[0], ctx.it[1],
                                         stream)
        N.check(rc, "wrf_sumflux_adj")
        return (None,) + tuple(bars[k] for k in SF_INPUTS) + (None,) * len(SF_DATA)


def sumflux(inputs: dict, data: dict, iteration: int, nsub: int, rdx, rdy):
    """Differentiable sumflux on the GPU; returns (ru_m', rv_m', ww_m')."""
    return Sumflux.apply((iteration, nsub, rdx, rdy), *[inputs[k] for k in SF_INPUTS], *[data[k] for k in SF_DATA])


class SpecUpdate(torch.autograd.Function):
    """field' = spec_bdyupdate(field, tend, dt, var) (var 't', 'u', 'v' or
    'm'); ``scal`` = (dt, var, rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, field, tend):
        _cuda_only(field, tend)
        dt, var = float(scal[0]), str(scal[1])
        shape = field.shape if field.dim() == 3 else (12,) + tuple(field.shape)
        cg = scalar_grid(shape, float(scal[2]), float(scal[3]))
        out = field.detach().clone()
        stream = _stream(field)
        with _on(field):
            rc = N.lib().wrf_spec_bdyupdate(ctypes.byref(cg), _ptr(out), _ptr(tend), dt, var.encode(), stream)
        N.check(rc, "wrf_spec_bdyupdate")
        ctx.cg, ctx.dt, ctx.var = cg, dt, var
        return out

    @staticmethod
    def backward(ctx, gout):
        gout = gout.contiguous()
        tb = torch.zeros_like(gout)
        stream = _stream(gout)
        with _on(gout):
            rc = N.lib().wrf_spec_bdyupdate_adj(ctypes.byref(ctx.cg), _ptr(gout), _ptr(tb), ctx.dt, ctx.var.encode(),
                                                stream)
        N.check(rc, "wrf_spec_bdyupdate_adj")
        return None, gout, tb


def spec_bdyupdate(field, tend, dt, var: str, rdx, rdy):
    """Differentiable spec_bdyupdate on the GPU."""
    return SpecUpdate.apply((dt, var, rdx, rdy), field, tend)


SPH_INPUTS = ("ph", "ph_save", "ph_tend", "mu_tend", "muts")


class SpecUpdatePh(torch.autograd.Function):
    """ph' = spec_bdyupdate_ph(ph_save, ph, ph_tend, mu_tend, muts, dt); the
    tensors follow SPH_INPUTS, ``scal`` = (dt, rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, *tensors):
        _cuda_only(*tensors)
        named = dict(zip(SPH_INPUTS, tensors))
        cg = scalar_grid(named["ph"].shape, float(scal[1]), float(scal[2]))
        out = named["ph"].detach().clone()
        stream = _stream(out)
        with _on(out):
            rc = N.lib().wrf_spec_bdyupdate_ph(ctypes.byref(cg), _table({**named, "ph": out}), float(scal[0]), stream)
        N.check(rc, "wrf_spec_bdyupdate_ph")
        ctx.save_for_backward(*tensors)
        ctx.cg, ctx.dt = cg, float(scal[0])
        return out

    @staticmethod
    def backward(ctx, gout):
        named = dict(zip(SPH_INPUTS, ctx.saved_tensors))
        bars = _bars(named, SPH_INPUTS, {"ph": gout})
        stream = _stream(gout)
        with _on(gout):
            rc = N.lib().wrf_spec_bdyupdate_ph_adj(ctypes.byref(ctx.cg), _table(named), _table(bars), ctx.dt, stream)
        N.check(rc, "wrf_spec_bdyupdate_ph_adj")
        return (None,) + tuple(bars[k] for k in SPH_INPUTS)


def spec_bdyupdate_ph(inputs: dict, dt, rdx, rdy):
    """Differentiable spec_bdyupdate_ph on the GPU; ``inputs`` maps SPH_INPUTS."""
    return SpecUpdatePh.apply((dt, rdx, rdy), *[inputs[k] for k in SPH_INPUTS])


PREP_FIELDS = ("mu", "mub", "mut", "muu", "muv", "u", "v", "w", "ru", "rv", "rw", "ww", "moist", "cqu", "cqv",
               "cqw", "al", "alb", "alt", "ph", "phb", "php")
PREP_OUTPUTS = ("mut", "muu", "muv", "ru", "rv", "rw", "ww", "cqu", "cqv", "cqw", "alt", "php")
PREP_DATA = ("msfu", "msfvx_inv", "msft", "msftx", "msfuy", "dnw", "c1h")
PREP_OPS = {"calculate_full": 1, "calc_mu_uv": 2, "couple_momentum": 4, "calc_ww_cp": 8, "calc_cq": 16,
            "calc_alt": 32, "calc_php": 64}


class Prep(torch.autograd.Function):
    """PREP_OUTPUTS' = rk_step_prep's functions of the mask ``ops`` (the
    others pass through); the tensors follow PREP_FIELDS then PREP_DATA,
    ``scal`` = (ops, rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, *tensors):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        _cuda_only(*tensors)
        ops = int(scal[0])
        named = dict(zip(PREP_FIELDS + PREP_DATA, tensors))
        cg = scalar_grid(named["u"].shape, float(scal[1]), float(scal[2]))
        outs = {k: named[k].detach().clone() for k in PREP_OUTPUTS}
        stream = _stream(named["u"])
        with _on(named["u"]):
            rc = N.lib().wrf_prep(ctypes.byref(cg), _table({**named, **outs}), ops, stream)
        N.check(rc, "wrf_prep")
        ctx.save_for_backward(*tensors)
        ctx.cg, ctx.ops = cg, ops
        return tuple(outs[k] for k in PREP_OUTPUTS)

    @staticmethod
    def backward(ctx, *gouts):
        named = dict(zip(PREP_FIELDS + PREP_DATA, ctx.saved_tensors))
        bars = _bars(named, PREP_FIELDS, dict(zip(PREP_OUTPUTS, gouts)))
        stream = _stream(bars["u"])
        with _on(bars["u"]):
            rc = N.lib().wrf_prep_adj(ctypes.byref(ctx.cg), _table(named), _table(bars), ctx.ops, stream)
        N.check(rc, "wrf_prep_adj")
        return (None,) + tuple(bars[k] for k in PREP_FIELDS) + (None,) * len(PREP_DATA)


def prep(fields: dict, data: dict, ops, rdx, rdy):
    """Differentiable rk_step_prep functions on the GPU: ``fields`` maps
    PREP_FIELDS, ``data`` PREP_DATA; ``ops`` a mask or PREP_OPS names; returns
    a dict of PREP_OUTPUTS."""
    if not isinstance(ops, int):
        ops = sum(PREP_OPS[o] for o in ops)
    outs = Prep.apply((ops, rdx, rdy), *[fields[k] for k in PREP_FIELDS], *[data[k] for k in PREP_DATA])
    return dict(zip(PREP_OUTPUTS, outs))


class Halo(torch.autograd.Function):
    """field' = set_physical_bc3d / set_physical_bc2d(field, var) (the open
    halo copies); ``scal`` = (var, rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, field):
        _cuda_only(field)
        var = str(scal[0])
        two_d = field.dim() == 2
        shape = (12,) + tuple(field.shape) if two_d else field.shape
        cg = scalar_grid(shape, float(scal[1]), float(scal[2]))
        out = field.detach().clone()
        stream = _stream(field)
        with _on(field):
            rc = N.lib().wrf_halo(ctypes.byref(cg), _ptr(out), var.encode(), int(two_d), stream)
        N.check(rc, "wrf_halo")
        ctx.cg, ctx.var, ctx.two_d = cg, var, two_d
        return out

    @staticmethod
    def backward(ctx, gout):
        gout = gout.contiguous()
        gin = torch.zeros_like(gout)
        stream = _stream(gout)
        with _on(gout):
            rc = N.lib().wrf_halo_adj(ctypes.byref(ctx.cg), _ptr(gout), _ptr(gin), ctx.var.encode(), int(ctx.two_d),
                                      stream)
        N.check(rc, "wrf_halo_adj")
        return None, gin


def halo(field, var: str, rdx=1.0 / 9000.0, rdy=1.0 / 9000.0):
    """Differentiable open-boundary halo copy of a [nz, ny, nx] or [ny, nx] field."""
    return Halo.apply((var, rdx, rdy), field)


class ZeroGradW(torch.autograd.Function):
    """w' = zero_grad_bdy(w, 'w'); ``scal`` = (rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, w):
        _cuda_only(w)
        cg = scalar_grid(w.shape, float(scal[0]), float(scal[1]))
        out = w.detach().clone()
        stream = _stream(w)
        with _on(w):
            rc = N.lib().wrf_zero_grad_w(ctypes.byref(cg), _ptr(out), stream)
        N.check(rc, "wrf_zero_grad_w")
        ctx.cg = cg
        return out

    @staticmethod
    def backward(ctx, gout):
        gout = gout.contiguous()
        gin = torch.zeros_like(gout)
        stream = _stream(gout)
        with _on(gout):
            rc = N.lib().wrf_zero_grad_w_adj(ctypes.byref(ctx.cg), _ptr(gout), _ptr(gin), stream)
        N.check(rc, "wrf_zero_grad_w_adj")
        return None, gin


def zero_grad_w(w, rdx=1.0 / 9000.0, rdy=1.0 / 9000.0):
    """Differentiable zero_grad_bdy of w."""
    return ZeroGradW.apply((rdx, rdy), w)


class Halos(torch.autograd.Function):
    """The halo copies of several fields in one launch each way: ``scal`` =
    (vars, rdx, rdy), one letter of ``vars`` per tensor: a stagger letter of
    :func:`halo`, 'Z' for zero_grad_bdy of w, or for a [7, nz, ny, nx]
    moisture array 'M' (slots 1..6 as 'p', slot 0 copied; each slot's points
    lie together, the slots need not)."""

    @staticmethod
    def _call(name, cg, letters, ins, outs):
        pi, po, vs, td = [], [], [], []
        for var, a, b in zip(letters, ins, outs):
            if var == "M":
                for m in range(1, 7):
                    pi.append(a.data_ptr() + 4 * m * a.stride(0))
                    po.append(b.data_ptr() + 4 * m * b.stride(0))
                    vs.append("p")
                    td.append(0)
                b[0].copy_(a[0])
            else:
                pi.append(a.data_ptr())
                po.append(b.data_ptr())
                vs.append(var)
                td.append(int(a.dim() == 2))
        n = len(pi)
        stream = _stream(ins[0])
        with _on(ins[0]):
            rc = getattr(N.lib(), name)(ctypes.byref(cg), n, (ctypes.c_void_p * n)(*pi), (ctypes.c_void_p * n)(*po),
                                        "".join(vs).encode(), (ctypes.c_int * n)(*td), stream)
        N.check(rc, name)

    @staticmethod
    def forward(ctx, scal, *fields):
        ctx.set_materialize_grads(False)
        letters = str(scal[0])
        if len(letters) != len(fields):
            raise ValueError("one letter per field")
        for var, f in zip(letters, fields):
            _cuda_only(*(f.unbind() if var == "M" else (f,)))
        shape = next((f.shape[-3:] for f in fields if f.dim() > 2), (12,) + tuple(fields[0].shape[-2:]))
        for var, f in zip(letters, fields):
            want = shape[1:] if f.dim() == 2 else ((7,) + tuple(shape) if var == "M" else shape)
            if tuple(f.shape) != tuple(want):
                raise ValueError(f"halos: a field of shape {tuple(f.shape)} where {tuple(want)} is expected")
        cg = scalar_grid(shape, float(scal[1]), float(scal[2]))
        outs = tuple(_packed_like(f) for f in fields)
        Halos._call("wrf_halo_copy", cg, letters, [f.detach() for f in fields], outs)
        ctx.cg, ctx.letters = cg, letters
        return outs

    @staticmethod
    def backward(ctx, *gouts):
        some = [q for q, gq in enumerate(gouts) if gq is not None]
        gins = [None] * len(gouts)
        if some:
            gs = [gouts[q].contiguous() for q in some]
            bs = [torch.empty_like(gq) for gq in gs]
            Halos._call("wrf_halo_copy_adj", ctx.cg, "".join(ctx.letters[q] for q in some), gs, bs)
            for q, b in zip(some, bs):
                gins[q] = b
        return (None,) + tuple(gins)


def halos(fields: Sequence[torch.Tensor], letters: str, rdx=1.0 / 9000.0, rdy=1.0 / 9000.0):
    """Differentiable halo copies of ``fields`` by ``letters`` (:class:`Halos`);
    returns the new fields."""
    return Halos.apply((letters, rdx, rdy), *fields)


AW_INPUTS = ("w", "rw_tend", "ww", "w_save", "u", "v", "muave", "muts", "mut", "t_2ave", "t_2", "t_1", "ph", "ph_1",
             "phb", "ph_tend", "ht", "c2a", "cqw", "alt", "a", "alpha", "gamma")
AW_DATA = ("msftx", "msfty", "fnm", "fnp", "rdnw", "rdn")
AW_OUTPUTS = ("t_2ave", "w", "ph")
_AW_FIELD = {"t_2ave": "t_2save", "t_2": "t", "t_1": "t_save", "ph_1": "ph_save"}


class AdvanceW(torch.autograd.Function):
    """(t_2ave', w', ph') = advance_w(...); the tensors follow AW_INPUTS then
    AW_DATA, ``scal`` = (dts, epssm, cf1, cf2, cf3, rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, *tensors):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        _cuda_only(*tensors)
        dts, epssm, cf1, cf2, cf3, rdx, rdy = (float(x) for x in scal)
        named = dict(zip(AW_INPUTS + AW_DATA, tensors))
        cg = scalar_grid(named["w"].shape, rdx, rdy)
        cg.epssm, cg.cf1, cg.cf2, cg.cf3 = epssm, cf1, cf2, cf3
        outs = {k: named[k].detach().clone() for k in AW_OUTPUTS}
        tab = _table({_AW_FIELD.get(k, k): v for k, v in {**named, **outs}.items()})
        stream = _stream(outs["w"])
        with _on(outs["w"]):
            rc = N.lib().wrf_advance_w(ctypes.byref(cg), tab, dts, stream)
        N.check(rc, "wrf_advance_w")
        ctx.save_for_backward(*tensors)
        ctx.cg, ctx.dts = cg, dts
        return tuple(outs[k] for k in AW_OUTPUTS)

    @staticmethod
    def backward(ctx, *gouts):
        tensors = ctx.saved_tensors
        named = dict(zip(AW_INPUTS + AW_DATA, tensors))
        bars = _bars(named, tuple(dict.fromkeys(AW_OUTPUTS + AW_INPUTS)), dict(zip(AW_OUTPUTS, gouts)))
        work = torch.empty_like(named["ht"])
        tab = _table({_AW_FIELD.get(k, k): v for k, v in named.items()})
        btab = _table({_AW_FIELD.get(k, k): v for k, v in bars.items()})
        stream = _stream(work)
        with _on(work):
            rc = N.lib().wrf_advance_w_adj(ctypes.byref(ctx.cg), tab, btab, ctx.dts, _ptr(work), stream)
        N.check(rc, "wrf_advance_w_adj")
        return (None,) + tuple(bars[k] for k in AW_INPUTS) + (None,) * len(AW_DATA)


def advance_w(inputs: dict, data: dict, dts, epssm, cf1, cf2, cf3, rdx=1.0 / 9000.0, rdy=1.0 / 9000.0):
    """Differentiable advance_w on the GPU: ``inputs`` maps AW_INPUTS, ``data``
    AW_DATA to tensors; returns a dict of AW_OUTPUTS."""
    outs = AdvanceW.apply((dts, epssm, cf1, cf2, cf3, rdx, rdy), *[inputs[k] for k in AW_INPUTS],
                          *[data[k] for k in AW_DATA])
    return dict(zip(AW_OUTPUTS, outs))


MUT_INPUTS = ("ww", "ww_1", "u", "u_1", "v", "v_1", "t", "t_1", "t_ave", "ft", "mu", "mut", "muave", "muts", "muu",
              "muv", "mudf", "mu_tend")
MUT_DATA = ("dnw", "fnm", "fnp", "rdnw", "msfuy", "msfvx_inv", "msftx", "msfty")
MUT_OUTPUTS = ("ww", "t", "t_ave", "muave", "muts", "mudf", "mu")
# the state-table names of advance_mu_t's arguments in the acoustic substep
_MUT_FIELD = {"ww_1": "ww1", "u_1": "u_save", "v_1": "v_save", "t_1": "t_save", "t_ave": "t_2save", "ft": "t_tend"}


class AdvanceMuT(torch.autograd.Function):
    """The seven outputs MUT_OUTPUTS of advance_mu_t; the tensors follow
    MUT_INPUTS then MUT_DATA, ``scal`` = (dts, epssm, rdx, rdy, ref_no_grad)."""

    @staticmethod
    def forward(ctx, scal, *tensors):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        _cuda_only(*tensors)
        dts, epssm, rdx, rdy = (float(x) for x in scal[:4])
        named = dict(zip(MUT_INPUTS + MUT_DATA, tensors))
        cg = scalar_grid(named["ww"].shape, rdx, rdy)
        cg.epssm = epssm
        outs = {k: named[k].detach().clone() for k in MUT_OUTPUTS}
        tab = _table({_MUT_FIELD.get(k, k): v for k, v in {**named, **outs}.items()})
        stream = _stream(outs["ww"])
        with _on(outs["ww"]):
            rc = N.lib().wrf_advance_mu_t(ctypes.byref(cg), tab, dts, stream)
        N.check(rc, "wrf_advance_mu_t")
        ctx.save_for_backward(*tensors)
        ctx.cg, ctx.dts, ctx.ref_no_grad = cg, dts, int(bool(scal[4]))
        return tuple(outs[k] for k in MUT_OUTPUTS)

    @staticmethod
    def backward(ctx, *gouts):
        tensors = ctx.saved_tensors
        named = dict(zip(MUT_INPUTS + MUT_DATA, tensors))
        bars = _bars(named, tuple(dict.fromkeys(MUT_OUTPUTS + MUT_INPUTS)), dict(zip(MUT_OUTPUTS, gouts)))
        work = torch.empty_like(named["ww"])
        tab = _table({_MUT_FIELD.get(k, k): v for k, v in named.items()})
        btab = _table({_MUT_FIELD.get(k, k): v for k, v in bars.items()})
        stream = _stream(work)
        with _on(work):
            rc = N.lib().wrf_advance_mu_t_adj(ctypes.byref(ctx.cg), tab, btab, ctx.dts, ctx.ref_no_grad, _ptr(work),
                                              stream)
        N.check(rc, "wrf_advance_mu_t_adj")
        return (None,) + tuple(bars[k] for k in MUT_INPUTS) + (None,) * len(MUT_DATA)


def advance_mu_t(inputs: dict, data: dict, dts, epssm, rdx=1.0 / 9000.0, rdy=1.0 / 9000.0, ref_no_grad=False):
    """Differentiable advance_mu_t on the GPU: ``inputs`` maps MUT_INPUTS,
    ``data`` MUT_DATA to tensors; returns a dict of MUT_OUTPUTS."""
    outs = AdvanceMuT.apply((dts, epssm, rdx, rdy, ref_no_grad), *[inputs[k] for k in MUT_INPUTS],
                            *[data[k] for k in MUT_DATA])
    return dict(zip(MUT_OUTPUTS, outs))


PRHO_INPUTS = ("al", "p", "ph", "alt", "t_2", "t_1", "c2a", "pm1", "mu", "mut")
# the state-table names of calc_p_rho's arguments in the acoustic substep
_PRHO_FIELD = {"t_2": "t", "t_1": "t_save", "mut": "muts"}


class CalcPRho(torch.autograd.Function):
    """(al', p', pm1') = calc_p_rho(...) at acoustic step ``step``; the
    tensors follow PRHO_INPUTS then rdnw, ``scal`` = (smdiv, step, rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, *tensors):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        _cuda_only(*tensors)
        smdiv, step, rdx, rdy = float(scal[0]), int(scal[1]), float(scal[2]), float(scal[3])
        named = dict(zip(PRHO_INPUTS + ("rdnw",), tensors))
        cg = scalar_grid(named["p"].shape, rdx, rdy)
        cg.smdiv = smdiv
        outs = {k: named[k].detach().clone() for k in ("al", "p", "pm1")}
        tab = _table({_PRHO_FIELD.get(k, k): v for k, v in {**named, **outs}.items()})
        stream = _stream(outs["p"])
        with _on(outs["p"]):
            rc = N.lib().wrf_calc_p_rho(ctypes.byref(cg), tab, step, stream)
        N.check(rc, "wrf_calc_p_rho")
        ctx.save_for_backward(*tensors)
        ctx.cg, ctx.step = cg, step
        return outs["al"], outs["p"], outs["pm1"]

    @staticmethod
    def backward(ctx, gal, gp, gpm1):
        tensors = ctx.saved_tensors
        named = dict(zip(PRHO_INPUTS + ("rdnw",), tensors))
        allb = _bars(named, tuple(dict.fromkeys(("al", "p", "pm1") + PRHO_INPUTS)), {"al": gal, "p": gp, "pm1": gpm1})
        out_b = {k: allb[k] for k in ("al", "p", "pm1")}
        bars = {k: v for k, v in allb.items() if k not in out_b}
        tab = _table({_PRHO_FIELD.get(k, k): v for k, v in named.items()})
        btab = _table({_PRHO_FIELD.get(k, k): v for k, v in {**out_b, **bars}.items()})
        stream = _stream(named["p"])
        with _on(named["p"]):
            rc = N.lib().wrf_calc_p_rho_adj(ctypes.byref(ctx.cg), tab, btab, ctx.step, stream)
        N.check(rc, "wrf_calc_p_rho_adj")
        allb = {**out_b, **bars}
        return (None,) + tuple(allb[k] for k in PRHO_INPUTS) + (None,)


def calc_p_rho(inputs: dict, rdnw, smdiv, step, rdx=1.0 / 9000.0, rdy=1.0 / 9000.0):
    """Differentiable calc_p_rho on the GPU: ``inputs`` maps PRHO_INPUTS to
    tensors; returns (al', p', pm1')."""
    return CalcPRho.apply((smdiv, step, rdx, rdy), *[inputs[k] for k in PRHO_INPUTS], rdnw)


BDY_NAMES = ("xs", "xe", "ys", "ye", "txs", "txe", "tys", "tye")


class RelaxBdytend(torch.autograd.Function):
    """out = tendency + relax_bdytend(field) for one stagger letter."""

    @staticmethod
    def forward(ctx, field, tendency, variable: str, dtbc: float, *bdy8):
        _cuda_only(field, tendency, *bdy8)
        nz, ny, nx = field.shape
        # 'm' (mu) is 2-D: its [1, ny, nx] field rides on a grid record of
        # the frame's minimum depth, and the library relaxes one level
        cg = scalar_grid((12, ny, nx) if variable == "m" else field.shape, 1.0 / 9000.0, 1.0 / 9000.0)
        out = tendency.detach().clone()
        arr = (ctypes.c_void_p * 8)(*[_ptr(b) for b in bdy8])
        stream = _stream(field)
        with _on(field):
            rc = N.lib().wrf_relax_bdytend(ctypes.byref(cg), _ptr(field), _ptr(out), arr, variable.encode(),
                                           float(dtbc), stream)
        N.check(rc, "wrf_relax_bdytend")
        ctx.cg, ctx.variable = cg, variable
        ctx.shape = (nz, ny, nx)
        ctx.device = field.device
        return out

    @staticmethod
    def backward(ctx, gout):
        gout = gout.contiguous()
        fb = torch.zeros(ctx.shape, dtype=torch.float32, device=ctx.device)
        stream = _stream(fb)
        with _on(fb):
            rc = N.lib().wrf_relax_bdytend_adj(ctypes.byref(ctx.cg), _ptr(gout), _ptr(fb), ctx.variable.encode(),
                                               stream)
        N.check(rc, "wrf_relax_bdytend_adj")
        return (fb, gout, None, None) + (None,) * 8


def relax_bdytend(field, tendency, variable: str, dtbc: float, bdy: dict):
    """Differentiable ``tendency + relax_bdytend(field)``; ``bdy`` maps
    xs xe ys ye txs txe tys tye to the boundary arrays (solver layout)."""
    return RelaxBdytend.apply(field, tendency, variable, dtbc, *[bdy[k] for k in BDY_NAMES])


class VSolveW(torch.autograd.Function):
    """w = implicit solve of (x; a, alpha, gamma) per column; arrays [nz, ...]."""

    @staticmethod
    def forward(ctx, x, a, alpha, gamma):
        ptrs = [_ptr(t) for t in (x, a, alpha, gamma)]
        nz = x.shape[0]
        ncol = x.numel() // nz
        w = torch.empty_like(x)
        stream = _stream(x)
        with _on(x):
            rc = N.lib().wrf_vsolve_w(ncol, nz, *ptrs, w.data_ptr(), stream)
        N.check(rc, "wrf_vsolve_w")
        ctx.save_for_backward(x, a, alpha, gamma)
        return w

    @staticmethod
    def backward(ctx, gw):
        x, a, alpha, gamma = ctx.saved_tensors
        nz = x.shape[0]
        ncol = x.numel() // nz
        gw = gw.contiguous()
        gx, ga, gal, gg = _zeros(x, x, x, x)
        stream = _stream(x)
        with _on(x):
            rc = N.lib().wrf_vsolve_w_adj(ncol, nz, _ptr(x), _ptr(a), _ptr(alpha), _ptr(gamma), _ptr(gw), _ptr(gx),
                                          _ptr(ga), _ptr(gal), _ptr(gg), stream)
        N.check(rc, "wrf_vsolve_w_adj")
        return gx, ga, gal, gg


def vsolve_w(x, a, alpha, gamma):
    """Differentiable implicit w solve (all columns of [nz, ...] arrays)."""
    return VSolveW.apply(x, a, alpha, gamma)


class CoefW(torch.autograd.Function):
    """(a, alpha, gamma) = calc_coef_w(mut, cqw, c2a) on the mass columns."""

    @staticmethod
    def forward(ctx, mut, cqw, c2a, rdn, rdnw, dts: float, epssm: float, top_lid: bool, rdx: float, rdy: float):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        ptrs = [_ptr(t) for t in (mut, cqw, c2a, rdn, rdnw)]
        cg = scalar_grid(cqw.shape, rdx, rdy)
        cg.epssm = float(epssm)
        cg.top_lid = int(bool(top_lid))
        a, alpha, gamma = (torch.empty_like(cqw) for _ in range(3))
        torch._foreach_zero_([a, alpha, gamma])  # one launch
        stream = _stream(cqw)
        with _on(cqw):
            rc = N.lib().wrf_coef_w(ctypes.byref(cg), *ptrs, float(dts), a.data_ptr(), alpha.data_ptr(),
                                    gamma.data_ptr(), stream)
        N.check(rc, "wrf_coef_w")
        ctx.save_for_backward(mut, cqw, c2a, rdn, rdnw)
        ctx.cg, ctx.dts = cg, float(dts)
        return a, alpha, gamma

    @staticmethod
    def backward(ctx, ga, galpha, ggamma):
        mut, cqw, c2a, rdn, rdnw = ctx.saved_tensors
        z, mb, cb, c2b = _zeros(cqw, mut, cqw, c2a)
        ga = z if ga is None else ga.contiguous()
        galpha = z if galpha is None else galpha.contiguous()
        ggamma = z if ggamma is None else ggamma.contiguous()
        stream = _stream(cqw)
        with _on(cqw):
            rc = N.lib().wrf_coef_w_adj(ctypes.byref(ctx.cg), _ptr(mut), _ptr(cqw), _ptr(c2a), _ptr(rdn), _ptr(rdnw),
                                        ctx.dts, _ptr(ga), _ptr(galpha), _ptr(ggamma), _ptr(mb), _ptr(cb), _ptr(c2b),
                                        stream)
        N.check(rc, "wrf_coef_w_adj")
        return mb, cb, c2b, None, None, None, None, None, None, None


def coef_w(mut, cqw, c2a, rdn, rdnw, dts, epssm=0.1, top_lid=False, rdx=1.0 / 9000.0, rdy=1.0 / 9000.0):
    """Differentiable calc_coef_w: returns (a, alpha, gamma)."""
    return CoefW.apply(mut, cqw, c2a, rdn, rdnw, dts, epssm, top_lid, rdx, rdy)


def capture(run: Callable[[], object], warmup: int = 2) -> torch.cuda.CUDAGraph:
    """Capture ``run`` -- a forward and its backward through these
    Functions, with fixed input tensors and cotangent seeds -- in a CUDA
    graph, after ``warmup`` eager runs on a side stream; ``graph.replay()``
    then re-runs every kernel of the pass with no host work between them.
    Every Function launches on the current stream, reads its scalars from
    the host arguments (no device-to-host read inside a step) and takes its
    scratch from torch's allocator (the graph's private pool during
    capture), so a whole step forward + reverse is capturable.  The
    gradients that ``run`` leaves (``.grad`` of the leaves) live in the
    graph's pool and are rewritten by each replay."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(warmup):
            run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    return graph


def rollout(step: Callable[..., Sequence[torch.Tensor]], state: Sequence[torch.Tensor], n_steps: int,
            every: int = 1) -> tuple[torch.Tensor, ...]:
    """Apply ``state = step(*state)`` ``n_steps`` times, differentiably, with
    checkpoints every ``every`` steps: the forward keeps only the state at
    the start of each segment (plus whatever ``step`` closes over, e.g.
    learnable parameters, which receive their gradients as usual); the
    backward recomputes each segment's forward once, with its operators'
    hand-written adjoints recording what they need, and back-propagates
    through it.  Peak memory is then one segment's intermediates plus
    n_steps / every states, instead of every intermediate of every step.
    ``every=0`` keeps the whole forward (no recomputation)."""
    if n_steps < 0 or every < 0:
        raise ValueError("n_steps and every must be >= 0")
    state = tuple(state)

    def segment(k, *xs):
        for _ in range(k):
            xs = tuple(step(*xs))
        return xs

    done = 0
    while done < n_steps:
        k = n_steps - done if every == 0 else min(every, n_steps - done)
        if every == 0 or not torch.is_grad_enabled():
            state = segment(k, *state)
        else:
            state = tuple(checkpoint(segment, k, *state, use_reentrant=False))
        done += k
    return state


# the fields one acoustic substep reads (state) and the constant arrays it
# takes as data
SUBSTEP_STATE = ("u", "v", "ru_tend", "rv_tend", "p", "pb", "ph", "php", "alt", "al", "mu", "muu", "muv", "cqu", "cqv",
                 "mudf", "ww", "ww1", "u_save", "v_save", "t", "t_save", "t_2save", "t_tend", "mut", "muave", "muts",
                 "mu_tend", "w", "rw_tend", "w_save", "ph_save", "phb", "ph_tend", "ht", "c2a", "cqw", "a", "alpha",
                 "gamma", "ru_m", "rv_m", "ww_m", "pm1")
SUBSTEP_DATA = ("msfux", "msfuy", "msfvx", "msfvx_inv", "msfvy", "msftx", "msfty", "fnm", "fnp", "rdnw", "rdn", "dnw")


def acoustic_substep(st: dict, data: dict, iteration: int, nsub: int, dts: float, *, epssm: float, emdiv: float,
                     smdiv: float, cf1: float, cf2: float, cf3: float, rdx: float, rdy: float) -> dict:
    """One acoustic substep composed from the operators above, in the
    reference's order (pywrf/solver.py:1394-1445): advance_uv with the
    specified-row update of u and v, advance_mu_t, spec_bdyupdate of t, mu
    and muts, advance_w, sumflux, spec_bdyupdate_ph, zero_grad_bdy of w,
    calc_p_rho and the halo copies of ph, al, p, muts, mu and mudf.  ``st``
    maps SUBSTEP_STATE, ``data`` SUBSTEP_DATA to tensors; returns the state
    after the substep (a new dict).  Differentiable end to end: every piece
    is a hand-written reverse kernel, and the chain keeps only the operators'
    inputs."""
    cg = _chain_grid(st["u"].shape, rdx, rdy, epssm=epssm, emdiv=emdiv, smdiv=smdiv, cf1=cf1, cf2=cf2, cf3=cf3)
    return _run_chain(_substep_ops(iteration, nsub, dts), cg, st, data)


def _scratch_like(cg, per_point: int = 0, per_column: int = 0) -> torch.Tensor:
    """Uninitialised float32 scratch of the grid's size on the current device
    and stream.  An operator takes its scratch when it runs: one that belongs to
    an operator object stays with the graph's node, where a checkpoint cannot
    drop it."""
    return torch.empty((per_point * cg.nz + per_column) * cg.ny * cg.nx, dtype=torch.float32,
                       device=torch.cuda.current_device())


class _TableOp(torch.autograd.Function):
    """A state-table operator with a hand-written adjoint: ``op`` names the
    fields it reads (``op.fields``, the updated ones ``op.outputs`` among
    them), its constant arrays (``op.data``), and runs the forward
    (``op.fwd(cg, table, stream)``) and the reverse product
    (``op.adj(cg, table, bar_table, stream)``, which rewrites the outputs'
    cotangents to the inputs' and accumulates the rest; or ``op.reverse`` on
    the named tensors themselves).  ``op`` holds no tensor."""

    @staticmethod
    def forward(ctx, op, cg, *tensors):
        # outputs without a cotangent reach backward as None (its _bars / None
        # checks hand out zeros from one shared buffer) instead of one
        # zero-filled tensor each, which backward would then clone
        ctx.set_materialize_grads(False)
        _cuda_only(*tensors)
        named = dict(zip(op.fields + op.data, tensors))
        outs = {k: named[k].detach().clone() for k in op.outputs}
        stream = _stream(tensors[0])
        with _on(tensors[0]):
            N.check(op.fwd(cg, _table({**named, **outs}), stream), op.name)
        ctx.save_for_backward(*tensors)
        ctx.op, ctx.cg = op, cg
        return tuple(outs[k] for k in op.outputs)

    @staticmethod
    def backward(ctx, *gouts):
        op = ctx.op
        saved = ctx.saved_tensors  # read once (checkpoint unpacks each saved tensor once)
        named = dict(zip(op.fields + op.data, saved))
        bars = _bars(named, op.fields, dict(zip(op.outputs, gouts)))
        stream = _stream(saved[0])
        with _on(saved[0]):
            if hasattr(op, "reverse"):
                rc = op.reverse(ctx.cg, named, bars, stream)
            else:
                rc = op.adj(ctx.cg, _table(named), _table(bars), stream)
            N.check(rc, op.name + "_adj")
        return (None, None) + tuple(bars[k] for k in op.fields) + (None,) * len(op.data)


# ---- chains: a sequence of operators on one state, reversed on one table of
# cotangents ----
#
# Composed from one autograd Function per operator, a step hands every field
# that several operators read to the autograd engine, which adds their
# cotangents up field by field, and every Function clears buffers for the
# cotangents it adds into and copies those it rewrites: at 240x240x41 about a
# third of the launches of a step's reverse, and most of its time on the host.
# The reverse kernels accumulate into their operands' cotangents and rewrite
# their results' cotangents to those of the values they replaced, so a whole
# sequence of them runs on one table; the engine sees the sequence's ends only.

class _Bars(dict):
    """The cotangents of a chain's state by name; those not yet reached are
    zero and are allocated when an operator asks for them."""

    def need(self, likes: dict) -> dict:
        missing = [k for k in likes if self.get(k) is None]
        self.update(zip(missing, _zeros(*[likes[k] for k in missing])))
        return {k: self[k] for k in likes}


class _ChainOp:
    """One operator of a chain: ``reads`` are the state names its reverse
    needs (their values on entry are kept), ``writes`` those it replaces and
    ``const`` the names of the constant arrays that both directions use.
    ``forward(cg, st, out, const, stream)`` fills ``out`` (copies of the written
    fields, updated in place; with ``fresh``, uninitialised, shaped like
    ``fill``) and ``backward(cg, saved, bars, const, stream)`` turns the written
    names' cotangents into those of the values on entry and adds the rest.  The
    chain saves what the reverse uses with its other tensors (an array changed
    in between raises, saved-tensor hooks see it, a checkpoint drops it), so
    ``backward`` holds no tensor itself; ``const`` maps the constants of the
    whole chain."""

    def __init__(self, reads, writes, forward, backward, const=(), fresh=False, fill=None):
        self.reads, self.writes, self.forward, self.backward = tuple(reads), tuple(writes), forward, backward
        self.const, self.fresh, self.fill = tuple(const), fresh, fill


def _rc(rc, name):
    N.check(rc, name)


def _table_chain_op(op, held=()):
    """A chain operator from a state-table operator (see :class:`_TableOp`);
    ``held`` names those of its constants that are fields of the chain's state
    (which receive no cotangent)."""
    reads, data = op.fields + tuple(held), tuple(k for k in op.data if k not in held)

    def fwd(cg, st, out, const, stream):
        _rc(op.fwd(cg, _table({**{k: const[k] for k in data}, **{k: st[k] for k in reads}, **out}), stream), op.name)

    def bwd(cg, saved, bars, const, stream):
        likes = {k: saved[k] for k in op.fields} if held else saved
        _rc(op.adj(cg, _table({**{k: const[k] for k in data}, **saved}), _table(bars.need(likes)), stream),
            op.name + "_adj")

    return _ChainOp(reads, op.outputs, fwd, bwd, data)


class _CallOp:
    """A state-table operator from two library calls (for the operators
    whose stand-alone Functions call the library directly)."""

    def __init__(self, name, fields, outputs, data, fwd, adj):
        self.name, self.fields, self.outputs, self.data, self.fwd, self.adj = name, fields, outputs, data, fwd, adj


class _Chain(torch.autograd.Function):
    """The operators ``ops`` in order on the state fields ``names`` (each
    with what is used of it, see :func:`_run_chain`) and the constants ``const``;
    returns the final values of ``outs``."""

    @staticmethod
    def forward(ctx, ops, cg, names, outs, const, *tensors):
        ctx.set_materialize_grads(False)
        st = {}
        own = set()   # ids of this chain's tensors that nothing has kept
        for (k, use), v in zip(names.items(), tensors):
            if use == _COPY and v.dim() == 4:  # taken slot by slot
                _cuda_only(*v.unbind())
            elif use != _LIKE:
                _ptr(v)
            st[k] = v.detach()
            if not v.is_contiguous():
                st[k] = st[k].contiguous() if use == _COPY else _packed_like(v)
                own.add(id(st[k]))
        saved = [v.detach() if v.requires_grad else v for v in const.values()]
        kept, steps = {}, []  # id of a kept state tensor -> its place among the saved ones
        with _on(tensors[0]):
            stream = _stream(tensors[0])
            for op in ops:
                at = []
                for k in op.reads:
                    v = st[k]
                    q = kept.get(id(v))
                    if q is None:
                        q = kept[id(v)] = len(saved)
                        saved.append(v)
                        own.discard(id(v))
                    at.append(q)
                steps.append((op.backward, op.reads, at))
                out = {}
                for k in op.writes:
                    if op.fresh:
                        out[k] = torch.empty_like(st[op.fill or k])
                    elif id(st[k]) in own:
                        out[k] = st[k]
                    else:
                        out[k] = st[k].clone()
                op.forward(cg, st, out, const, stream)
                for k, v in out.items():
                    st[k] = v
                    own.add(id(v))
        ctx.save_for_backward(*saved)
        ctx.steps, ctx.cg, ctx.names, ctx.outs, ctx.const = steps, cg, tuple(names), outs, tuple(const)
        ctx.device = tensors[0].get_device()
        return tuple(st[k] for k in outs)

    @staticmethod
    def backward(ctx, *gouts):
        saved = ctx.saved_tensors  # read once (checkpoint unpacks each saved tensor once)
        const = dict(zip(ctx.const, saved))
        bars = _Bars()
        for k, gk in zip(ctx.outs, gouts):
            if gk is not None:
                bars[k] = gk.contiguous().clone()
        with torch.cuda.device(ctx.device):
            stream = torch.cuda.current_stream(ctx.device).cuda_stream
            for backward, reads, at in reversed(ctx.steps):
                backward(ctx.cg, {k: saved[q] for k, q in zip(reads, at)}, bars, const, stream)
        need = ctx.needs_input_grad[5:]
        return (None,) * 5 + tuple(bars.get(k) if w else None for k, w in zip(ctx.names, need))


# what a chain uses of a field it is given: its shape, an updated copy of it, or
# its values
_LIKE, _COPY, _READ = range(3)


def _run_chain(ops, cg, st: dict, data: dict) -> dict:
    """``st`` after the chain, whose constants are in ``data``: the fields the
    operators write replaced."""
    names, made = {}, set()
    for op in ops:
        for k in op.reads:
            if k not in made:
                names[k] = _READ
        use = _LIKE if op.fill else _READ if op.fresh else _COPY
        for k in (op.fill,) if op.fill else op.writes:
            if k not in made:
                names[k] = max(names.get(k, use), use)
        made.update(op.writes)
    outs = tuple(k for k in dict.fromkeys(k for op in ops for k in op.writes) if not k.startswith("_"))
    const = {k: data[k] for k in dict.fromkeys(k for op in ops for k in op.const)}
    new = _Chain.apply(tuple(ops), cg, names, outs, const, *[st[k] for k in names])
    return {**st, **dict(zip(outs, new))}


def _zero_op(name, like):
    """``name`` starts from zero (shaped like the state field ``like``)."""
    def fwd(cg, st, out, const, stream):
        out[name].zero_()

    def bwd(cg, saved, bars, const, stream):
        bars.pop(name, None)

    return _ChainOp((), (name,), fwd, bwd, fresh=True, fill=like)


def _halo_op(names, letters):
    """The halo copies of ``names`` (:class:`Halos`), out of place."""
    def fwd(cg, st, out, const, stream):
        Halos._call("wrf_halo_copy", cg, letters, [st[k] for k in names], [out[k] for k in names])

    def bwd(cg, saved, bars, const, stream):
        some = [q for q, k in enumerate(names) if bars.get(k) is not None]
        if some:
            gs = [bars[names[q]] for q in some]
            new = [torch.empty_like(v) for v in gs]
            Halos._call("wrf_halo_copy_adj", cg, "".join(letters[q] for q in some), gs, new)
            bars.update((names[q], v) for q, v in zip(some, new))

    return _ChainOp((), names, fwd, bwd, fresh=True)


def _spec_update_op(field, tend, dt, var):
    def fwd(cg, st, out, const, stream):
        _rc(N.lib().wrf_spec_bdyupdate(ctypes.byref(cg), _ptr(out[field]), _ptr(st[tend]), dt, var.encode(), stream),
            "wrf_spec_bdyupdate")

    def bwd(cg, saved, bars, const, stream):
        if bars.get(field) is not None:
            b = bars.need({tend: saved[tend]})
            _rc(N.lib().wrf_spec_bdyupdate_adj(ctypes.byref(cg), _ptr(bars[field]), _ptr(b[tend]), dt, var.encode(),
                                               stream), "wrf_spec_bdyupdate_adj")

    return _ChainOp((tend,), (field,), fwd, bwd)


def _spec_tend_op(tend, bt: dict, var):
    def fwd(cg, st, out, const, stream):
        _rc(N.lib().wrf_spec_bdytend(ctypes.byref(cg), _ptr(out[tend]), _ptr(bt["txs"]), _ptr(bt["txe"]),
                                     _ptr(bt["tys"]), _ptr(bt["tye"]), var.encode(), stream), "wrf_spec_bdytend")

    def bwd(cg, saved, bars, const, stream):
        if bars.get(tend) is not None:
            _rc(N.lib().wrf_spec_bdytend_adj(ctypes.byref(cg), _ptr(bars[tend]), var.encode(), stream),
                "wrf_spec_bdytend_adj")

    return _ChainOp((), (tend,), fwd, bwd)


def _relax_op(field, tend, bdy: dict, var, dtbc):
    """tend += relax_bdytend(field); 'm' (mu) is 2-D: the library relaxes one
    level of it."""
    arrays = [bdy[k] for k in BDY_NAMES]

    def fwd(cg, st, out, const, stream):
        arr = (ctypes.c_void_p * 8)(*[_ptr(v) for v in arrays])
        _rc(N.lib().wrf_relax_bdytend(ctypes.byref(cg), _ptr(st[field]), _ptr(out[tend]), arr, var.encode(),
                                      float(dtbc), stream), "wrf_relax_bdytend")

    def bwd(cg, saved, bars, const, stream):
        if bars.get(tend) is not None:
            b = bars.need({field: saved[field]})
            _rc(N.lib().wrf_relax_bdytend_adj(ctypes.byref(cg), _ptr(bars[tend]), _ptr(b[field]), var.encode(),
                                              stream), "wrf_relax_bdytend_adj")

    return _ChainOp((field,), (tend,), fwd, bwd)


def _mass_weight_op(field, mass, out_name, nk):
    def fwd(cg, st, out, const, stream):
        out[out_name].zero_()
        _rc(N.lib().wrf_mass_weight(ctypes.byref(cg), _ptr(st[field]), _ptr(st[mass]), _ptr(out[out_name]), nk,
                                    stream), "wrf_mass_weight")

    def bwd(cg, saved, bars, const, stream):
        gk = bars.pop(out_name, None)
        if gk is not None:
            b = bars.need(saved)
            _rc(N.lib().wrf_mass_weight_adj(ctypes.byref(cg), _ptr(saved[field]), _ptr(saved[mass]), _ptr(gk),
                                            _ptr(b[field]), _ptr(b[mass]), nk, stream), "wrf_mass_weight_adj")

    return _ChainOp((field, mass), (out_name,), fwd, bwd, fresh=True, fill=field)


def _advect_work(cg, name, like):
    n = ctypes.c_size_t(0)
    _rc(getattr(N.lib(), name)(ctypes.byref(cg), ctypes.byref(n)), "work")
    return torch.empty(int(n.value), dtype=torch.float32, device=like.device), n


def _advect_momentum_op(component, field, tend):
    msf = ("msfux", "msfvy", "msftx")[component]
    msf2 = "msfvx" if component == 1 else None
    names = (msf, msf2, "fnm", "fnp", "rdn" if component == 2 else "rdnw")

    def pointers(const):
        return [None if k is None else _ptr(const[k]) for k in names]

    def fwd(cg, st, out, const, stream):
        _rc(N.lib().wrf_advect_momentum(ctypes.byref(cg), component, _ptr(st[field]), _ptr(out[tend]), _ptr(st["ru"]),
                                        _ptr(st["rv"]), _ptr(st["ww"]), *pointers(const), 0, stream),
            "wrf_advect_momentum")

    def bwd(cg, saved, bars, const, stream):
        if bars.get(tend) is None:
            return
        b = bars.need(saved)
        work, n = _advect_work(cg, "wrf_advect_momentum_adj_work", saved[field])
        _rc(N.lib().wrf_advect_momentum_adj(ctypes.byref(cg), component, _ptr(saved[field]), _ptr(saved["ru"]),
                                            _ptr(saved["rv"]), _ptr(saved["ww"]), *pointers(const), _ptr(bars[tend]),
                                            _ptr(b[field]), _ptr(b["ru"]), _ptr(b["rv"]), _ptr(b["ww"]), _ptr(work),
                                            n, stream),
            "wrf_advect_momentum_adj")

    return _ChainOp((field, "ru", "rv", "ww"), (tend,), fwd, bwd, [k for k in names if k])


ADVECT_DATA = ("msftx", "fnm", "fnp", "rdnw")


def _advect_scalar_op(field, tend):
    def fwd(cg, st, out, const, stream):
        _rc(N.lib().wrf_advect_scalar(ctypes.byref(cg), _ptr(st[field]), _ptr(out[tend]), _ptr(st["ru"]),
                                      _ptr(st["rv"]), _ptr(st["ww"]), *[_ptr(const[k]) for k in ADVECT_DATA], stream),
            "wrf_advect_scalar")

    def bwd(cg, saved, bars, const, stream):
        if bars.get(tend) is None:
            return
        b = bars.need(saved)
        work, n = _advect_work(cg, "wrf_advect_scalar_adj_work", saved[field])
        _rc(N.lib().wrf_advect_scalar_adj(ctypes.byref(cg), _ptr(saved[field]), _ptr(saved["ru"]), _ptr(saved["rv"]),
                                          _ptr(saved["ww"]), *[_ptr(const[k]) for k in ADVECT_DATA], _ptr(bars[tend]),
                                          _ptr(b[field]), _ptr(b["ru"]), _ptr(b["rv"]), _ptr(b["ww"]), _ptr(work), n,
                                          stream), "wrf_advect_scalar_adj")

    return _ChainOp((field, "ru", "rv", "ww"), (tend,), fwd, bwd, ADVECT_DATA)


def _advect_moist_op():
    """advect_tend = the advection of qv .. qg (slots 1..6) by the averaged
    fluxes, zero outside the advected points (pywrf/wrf_dynamics.py:
    3982-4051)."""
    fluxes = ("ru_m", "rv_m", "ww_m")

    def fwd(cg, st, out, const, stream):
        out["advect_tend"].zero_()
        _rc(N.lib().wrf_advect_moist(ctypes.byref(cg), _ptr(st["moist"]), _ptr(out["advect_tend"]),
                                     *[_ptr(st[k]) for k in fluxes], *[_ptr(const[k]) for k in ADVECT_DATA], stream),
            "wrf_advect_moist")

    def bwd(cg, saved, bars, const, stream):
        gk = bars.pop("advect_tend", None)
        if gk is None:
            return
        b = bars.need(saved)
        work, n = _advect_work(cg, "wrf_advect_scalar_adj_work", saved["ru_m"])
        maps = [_ptr(const[k]) for k in ADVECT_DATA]
        for m in range(1, 7):
            _rc(N.lib().wrf_advect_scalar_adj(ctypes.byref(cg), _ptr(saved["moist"][m]),
                                              *[_ptr(saved[k]) for k in fluxes], *maps, _ptr(gk[m]),
                                              _ptr(b["moist"][m]), *[_ptr(b[k]) for k in fluxes], _ptr(work), n,
                                              stream), "wrf_advect_scalar_adj")

    return _ChainOp(("moist",) + fluxes, ("advect_tend",), fwd, bwd, ADVECT_DATA, fresh=True, fill="moist")


def _diffusion_op(var, field, tend, mass, visc, base=None):
    """tend += horizontal_diffusion(field - ``base``, a constant); ``field``
    "moist": its six species into the slots of ``tend``."""
    def each(v):
        return [v[m] for m in range(1, 7)] if v.dim() == 4 else [v]

    def fwd(cg, st, out, const, stream):
        tab, bp = _table({k: const[k] for k in HDIFF_DATA}), None if base is None else _ptr(const[base])
        for f, o in zip(each(st[field]), each(out[tend])):
            _rc(N.lib().wrf_horizontal_diffusion(ctypes.byref(cg), tab, var.encode(), _ptr(f), bp, _ptr(st[mass]),
                                                 _ptr(st[visc]), _ptr(o), stream), "wrf_horizontal_diffusion")

    def bwd(cg, saved, bars, const, stream):
        if bars.get(tend) is None:
            return
        b = bars.need(saved)
        tab, bp = _table({k: const[k] for k in HDIFF_DATA}), None if base is None else _ptr(const[base])
        for f, gk, fb in zip(each(saved[field]), each(bars[tend]), each(b[field])):
            _rc(N.lib().wrf_horizontal_diffusion_adj(ctypes.byref(cg), tab, var.encode(), _ptr(f), bp,
                                                     _ptr(saved[mass]), _ptr(saved[visc]), _ptr(gk), _ptr(fb),
                                                     _ptr(b[mass]), _ptr(b[visc]), stream),
                "wrf_horizontal_diffusion_adj")

    return _ChainOp((field, mass, visc), (tend,), fwd, bwd, HDIFF_DATA + (() if base is None else (base,)))


def _coef_w_op(dts):
    names = ("a", "alpha", "gamma")

    def fwd(cg, st, out, const, stream):
        for k in names:
            out[k].zero_()
        _rc(N.lib().wrf_coef_w(ctypes.byref(cg), _ptr(st["mut"]), _ptr(st["cqw"]), _ptr(st["c2a"]),
                               _ptr(const["rdn"]), _ptr(const["rdnw"]), float(dts), *[_ptr(out[k]) for k in names],
                               stream), "wrf_coef_w")

    def bwd(cg, saved, bars, const, stream):
        gs = bars.need({k: saved["cqw"] for k in names})
        b = bars.need(saved)
        _rc(N.lib().wrf_coef_w_adj(ctypes.byref(cg), _ptr(saved["mut"]), _ptr(saved["cqw"]), _ptr(saved["c2a"]),
                                   _ptr(const["rdn"]), _ptr(const["rdnw"]), float(dts), *[_ptr(gs[k]) for k in names],
                                   _ptr(b["mut"]), _ptr(b["cqw"]), _ptr(b["c2a"]), stream), "wrf_coef_w_adj")
        for k in names:
            del bars[k]

    return _ChainOp(("mut", "cqw", "c2a"), names, fwd, bwd, ("rdn", "rdnw"), fresh=True, fill="cqw")


def _substep_ops(iteration: int, nsub: int, dts: float) -> list:
    """The operators of one acoustic substep, in the reference's order."""
    L = N.lib()
    by = ctypes.byref
    field = lambda names, ren: tuple(ren.get(k, k) for k in names)  # noqa: E731

    def with_work(tab_adj, **size):
        return lambda cg, tab, btab, stream: tab_adj(cg, tab, btab, _ptr(_scratch_like(cg, **size)), stream)

    uv = _CallOp("wrf_advance_uv", UV_INPUTS, ("u", "v"), UV_DATA,
                 lambda cg, tab, s: L.wrf_advance_uv(by(cg), tab, dts, s),
                 lambda cg, tab, b, s: L.wrf_advance_uv_adj(by(cg), tab, b, dts, s))
    mt = _CallOp("wrf_advance_mu_t", field(MUT_INPUTS, _MUT_FIELD), field(MUT_OUTPUTS, _MUT_FIELD), MUT_DATA,
                 lambda cg, tab, s: L.wrf_advance_mu_t(by(cg), tab, dts, s),
                 with_work(lambda cg, tab, b, w, s: L.wrf_advance_mu_t_adj(by(cg), tab, b, dts, 0, w, s), per_point=1))
    aw = _CallOp("wrf_advance_w", field(AW_INPUTS, _AW_FIELD), field(AW_OUTPUTS, _AW_FIELD), AW_DATA,
                 lambda cg, tab, s: L.wrf_advance_w(by(cg), tab, dts, s),
                 with_work(lambda cg, tab, b, w, s: L.wrf_advance_w_adj(by(cg), tab, b, dts, w, s), per_column=1))
    sf = _CallOp("wrf_sumflux", SF_INPUTS, SF_INPUTS[:3], SF_DATA,
                 lambda cg, tab, s: L.wrf_sumflux(by(cg), tab, iteration, nsub, s),
                 lambda cg, tab, b, s: L.wrf_sumflux_adj(by(cg), tab, b, iteration, nsub, s))
    sp = _CallOp("wrf_spec_bdyupdate_ph", SPH_INPUTS, ("ph",), (),
                 lambda cg, tab, s: L.wrf_spec_bdyupdate_ph(by(cg), tab, dts, s),
                 lambda cg, tab, b, s: L.wrf_spec_bdyupdate_ph_adj(by(cg), tab, b, dts, s))
    ops = [_table_chain_op(uv), _table_chain_op(mt)]
    ops += [_spec_update_op("t", "t_tend", dts, "t"), _spec_update_op("mu", "mu_tend", dts, "m"),
            _spec_update_op("muts", "mu_tend", dts, "m")]
    ops += [_table_chain_op(aw), _table_chain_op(sf), _table_chain_op(sp), _p_rho_op(iteration)]
    ops.append(_halo_op(("w", "ph", "al", "p", "muts", "mu", "mudf"), "Zwppttt"))
    return ops


def _p_rho_op(step: int):
    ren = tuple(_PRHO_FIELD.get(k, k) for k in PRHO_INPUTS)
    return _table_chain_op(_CallOp("wrf_calc_p_rho", ren, ("al", "p", "pm1"), ("rdnw",),
                                   lambda cg, tab, s: N.lib().wrf_calc_p_rho(ctypes.byref(cg), tab, step, s),
                                   lambda cg, tab, b, s: N.lib().wrf_calc_p_rho_adj(ctypes.byref(cg), tab, b, step,
                                                                                    s)))


def _chain_grid(shape, rdx, rdy, **scal):
    cg = scalar_grid(shape, rdx, rdy)
    for k, v in scal.items():
        setattr(cg, k, v if k == "top_lid" else float(v))
    return cg


class _SmallStepPrep:
    name = "wrf_small_step_prep"
    fields = ("mu", "mu_1", "mub", "mudf", "muts", "mu_save", "muu", "muv", "muus", "muvs", "mut", "u", "u_1",
              "u_save", "v", "v_1", "v_save", "t", "t_1", "t_save", "w", "w_1", "w_save", "ph", "ph_1", "ph_save",
              "ww", "ww1", "c2a", "pb", "p", "alt")
    outputs = ("mu", "mu_1", "mudf", "muts", "mu_save", "muus", "muvs", "u", "u_1", "u_save", "v", "v_1", "v_save",
               "t", "t_1", "t_save", "w", "w_1", "w_save", "ph", "ph_1", "ph_save", "ww1", "c2a")
    data = ("msfuy", "msfvx_inv", "msfty")

    def __init__(self, rk_step):
        self.rk_step = rk_step

    def fwd(self, cg, tab, stream):
        return N.lib().wrf_small_step_prep(ctypes.byref(cg), tab, self.rk_step, stream)

    def adj(self, cg, tab, btab, stream):
        work = _scratch_like(cg, per_column=3)
        return N.lib().wrf_small_step_prep_adj(ctypes.byref(cg), tab, btab, self.rk_step, _ptr(work), stream)


class _SmallStepFinish:
    name = "wrf_small_step_finish"
    fields = ("u", "u_save", "v", "v_save", "w", "w_save", "ph", "ph_save", "ww", "ww1", "t", "t_save", "h_diabatic",
              "mu", "mu_save", "mut", "muts", "muu", "muv", "muus", "muvs")
    outputs = ("u", "v", "w", "ph", "ww", "t", "mu", "muus", "muvs")
    data = ("msfuy", "msfvx", "msfty")

    def __init__(self, dts, nsub, rk_step):
        self.dts, self.nsub, self.rk_step = dts, nsub, rk_step

    def fwd(self, cg, tab, stream):
        return N.lib().wrf_small_step_finish(ctypes.byref(cg), tab, self.dts, self.nsub, self.rk_step, stream)

    def adj(self, cg, tab, btab, stream):
        work = _scratch_like(cg, per_column=2)
        return N.lib().wrf_small_step_finish_adj(ctypes.byref(cg), tab, btab, self.dts, self.nsub, self.rk_step,
                                                 _ptr(work), stream)


def small_step_prep(st: dict, data: dict, rk_step: int, rdx, rdy) -> dict:
    """Differentiable small_step_prep (pywrf/wrf_dynamics.py:3152-3266):
    returns ``st`` with the fields it updates replaced."""
    op = _SmallStepPrep(rk_step)
    cg = scalar_grid(st["u"].shape, rdx, rdy)
    outs = _TableOp.apply(op, cg, *[st[k] for k in op.fields], *[data[k] for k in op.data])
    return {**st, **dict(zip(op.outputs, outs))}


def small_step_finish(st: dict, data: dict, dts: float, nsub: int, rk_step: int, rdx, rdy) -> dict:
    """Differentiable calc_mu_uv_1 + small_step_finish
    (pywrf/wrf_dynamics.py:3844-3930): returns ``st`` with the fields they
    update replaced."""
    op = _SmallStepFinish(dts, nsub, rk_step)
    cg = scalar_grid(st["u"].shape, rdx, rdy)
    outs = _TableOp.apply(op, cg, *[st[k] for k in op.fields], *[data[k] for k in op.data])
    return {**st, **dict(zip(op.outputs, outs))}


# the fields the acoustic part of an RK stage reads (state) and its constant
# arrays (data)
STAGE_STATE = SUBSTEP_STATE + ("h_diabatic", "mu_1", "mu_save", "mub", "muus", "muvs", "ph_1", "t_1", "u_1", "v_1",
                               "w_1")
STAGE_DATA = SUBSTEP_DATA


def acoustic_stage(st: dict, data: dict, rk_step: int, nsub: int, dts: float, *, epssm: float, emdiv: float,
                   smdiv: float, cf1: float, cf2: float, cf3: float, rdx: float, rdy: float,
                   top_lid: bool = False) -> dict:
    """The acoustic part of one RK stage composed from the operators'
    Functions, in the reference's order (pywrf/solver.py:1258-1492):
    small_step_prep, calc_p_rho at step 0, calc_coef_w, the halo copies that
    follow them, ``nsub`` substeps (:func:`acoustic_substep`), calc_mu_uv_1
    with small_step_finish, and at the last stage the halo copies of the
    averaged fluxes and column masses.  ``st`` maps every field these read;
    returns the state after the stage."""
    cg = _chain_grid(st["u"].shape, rdx, rdy, epssm=epssm, emdiv=emdiv, smdiv=smdiv, cf1=cf1, cf2=cf2, cf3=cf3,
                     top_lid=int(bool(top_lid)))
    return _run_chain(_acoustic_ops(rk_step, nsub, dts), cg, st, data)


def _acoustic_ops(rk_step: int, nsub: int, dts: float) -> list:
    """The operators of :func:`acoustic_stage`."""
    ops = [_table_chain_op(_SmallStepPrep(rk_step)), _p_rho_op(0), _coef_w_op(dts),
           _halo_op(("ru_tend", "rv_tend", "ph", "al", "p", "t_1", "t_save", "mu_1", "mu", "mudf"), "uvwppttttt")]
    for it in range(1, nsub + 1):
        ops += _substep_ops(it, nsub, dts)
    ops.append(_table_chain_op(_SmallStepFinish(dts, nsub, rk_step)))
    if rk_step == 3:
        ops.append(_halo_op(("ru_m", "rv_m", "ww_m", "mut", "muts"), "uvwtt"))
    return ops


class _Addtend:
    name = "wrf_addtend"
    fields = ("ru_tend", "rv_tend", "rw_tend", "ph_tend", "t_tend", "mu_tend", "ru_tendf", "rv_tendf", "rw_tendf",
              "ph_tendf", "t_tendf", "mu_tendf", "u_save", "v_save", "w_save", "ph_save", "t_save", "h_diabatic", "mut")
    outputs = ("ru_tend", "rv_tend", "rw_tend", "ph_tend", "t_tend", "mu_tend", "ru_tendf", "rv_tendf", "rw_tendf",
               "ph_tendf", "t_tendf")
    data = ("msfty", "msfuy", "msfvx", "msfvx_inv")

    def __init__(self, rk_step):
        self.rk_step = rk_step

    def fwd(self, cg, tab, stream):
        return N.lib().wrf_addtend(ctypes.byref(cg), tab, self.rk_step, stream)

    def adj(self, cg, tab, btab, stream):
        return N.lib().wrf_addtend_adj(ctypes.byref(cg), tab, btab, self.rk_step, stream)


def addtend(st: dict, data: dict, rk_step: int, rdx, rdy) -> dict:
    """Differentiable rk_addtend_dry (pywrf/wrf_dynamics.py:3100-3148):
    returns ``st`` with the tendencies (and at stage 1 the physics
    tendencies) replaced."""
    op = _Addtend(rk_step)
    cg = scalar_grid(st["ru_tend"].shape, rdx, rdy)
    outs = _TableOp.apply(op, cg, *[st[k] for k in op.fields], *[data[k] for k in op.data])
    return {**st, **dict(zip(op.outputs, outs))}


class SpecBdytend(torch.autograd.Function):
    """tend' = spec_bdytend(tend, boundary tendencies, var): the specified
    rows take the boundary file's tendency (data); ``scal`` = (var, rdx,
    rdy), then the x-start, x-end, y-start, y-end boundary tendencies."""

    @staticmethod
    def forward(ctx, scal, tend, txs, txe, tys, tye):
        _cuda_only(tend, txs, txe, tys, tye)
        var = str(scal[0])
        shape = (12,) + tuple(tend.shape) if tend.dim() == 2 else tend.shape
        cg = scalar_grid(shape, float(scal[1]), float(scal[2]))
        out = tend.detach().clone()
        stream = _stream(tend)
        with _on(tend):
            rc = N.lib().wrf_spec_bdytend(ctypes.byref(cg), _ptr(out), _ptr(txs), _ptr(txe), _ptr(tys), _ptr(tye),
                                          var.encode(), stream)
        N.check(rc, "wrf_spec_bdytend")
        ctx.cg, ctx.var = cg, var
        return out

    @staticmethod
    def backward(ctx, gout):
        gin = gout.contiguous().clone()
        stream = _stream(gin)
        with _on(gin):
            rc = N.lib().wrf_spec_bdytend_adj(ctypes.byref(ctx.cg), _ptr(gin), ctx.var.encode(), stream)
        N.check(rc, "wrf_spec_bdytend_adj")
        return None, gin, None, None, None, None


def spec_bdytend(tend, bt: dict, var: str, rdx, rdy):
    """Differentiable spec_bdytend; ``bt`` maps txs txe tys tye to the
    variable's boundary tendencies (solver layout)."""
    return SpecBdytend.apply((var, rdx, rdy), tend, bt["txs"], bt["txe"], bt["tys"], bt["tye"])


HDIFF_DATA = ("msfux", "msfuy", "msfvx", "msfvy", "msftx", "msfty", "msfvx_inv")


class HorizontalDiffusion(torch.autograd.Function):
    """tend' = tend + horizontal_diffusion(field) (pywrf/wrf_dynamics.py:
    2623-2915): ``scal`` = (var, rdx, rdy) with var 'u', 'v', 'w' or 'm' (a
    mass-point scalar; with ``base``, the diffusion of field - base as
    horizontal_diffusion_3dmp forms it), then the field, the incoming
    tendency, the column mass, the eddy viscosity, ``base`` (data, or None)
    and the seven map factors of HDIFF_DATA; gradients with respect to the
    field, the tendency, the mass and the viscosity."""

    @staticmethod
    def forward(ctx, scal, field, tend, mut, xk, base, *maps):
        _cuda_only(field, tend, mut, xk, base, *maps)
        var = str(scal[0])
        cg = scalar_grid(field.shape, float(scal[1]), float(scal[2]))
        out = tend.detach().clone()
        tab = _table(dict(zip(HDIFF_DATA, maps)))
        stream = _stream(field)
        bp = None if base is None else _ptr(base)
        with _on(field):
            rc = N.lib().wrf_horizontal_diffusion(ctypes.byref(cg), tab, var.encode(), _ptr(field), bp, _ptr(mut),
                                                  _ptr(xk), _ptr(out), stream)
        N.check(rc, "wrf_horizontal_diffusion")
        ctx.cg, ctx.var, ctx.has_base = cg, var, base is not None
        ctx.save_for_backward(field, mut, xk, *(() if base is None else (base,)), *maps)
        return out

    @staticmethod
    def backward(ctx, gout):
        saved = ctx.saved_tensors
        field, mut, xk = saved[:3]
        base = saved[3] if ctx.has_base else None
        maps = saved[4:] if ctx.has_base else saved[3:]
        gout = gout.contiguous()
        fb, mb, kb = _zeros(field, mut, xk)
        tab = _table(dict(zip(HDIFF_DATA, maps)))
        stream = _stream(field)
        bp = None if base is None else _ptr(base)
        with _on(field):
            rc = N.lib().wrf_horizontal_diffusion_adj(ctypes.byref(ctx.cg), tab, ctx.var.encode(), _ptr(field), bp,
                                                      _ptr(mut), _ptr(xk), _ptr(gout), _ptr(fb), _ptr(mb), _ptr(kb),
                                                      stream)
        N.check(rc, "wrf_horizontal_diffusion_adj")
        return (None, fb, gout, mb, kb, None) + (None,) * len(HDIFF_DATA)


def horizontal_diffusion(var: str, field, tend, mut, xk, data: dict, rdx, rdy, base=None):
    """Differentiable ``tend + horizontal_diffusion(field)``; ``data`` maps
    the map factors of HDIFF_DATA."""
    return HorizontalDiffusion.apply((var, rdx, rdy), field, tend, mut, xk, base, *[data[k] for k in HDIFF_DATA])


class MassWeight(torch.autograd.Function):
    """out = field * mut on levels below nk of the mass points, zero elsewhere
    (mass_weight, pywrf/wrf_boundary.py:408-414); ``scal`` = (nk, rdx, rdy)."""

    @staticmethod
    def forward(ctx, scal, field, mut):
        _cuda_only(field, mut)
        nk = int(scal[0])
        cg = scalar_grid(field.shape, float(scal[1]), float(scal[2]))
        out = torch.zeros_like(field)
        stream = _stream(field)
        with _on(field):
            N.check(N.lib().wrf_mass_weight(ctypes.byref(cg), _ptr(field), _ptr(mut), _ptr(out), nk, stream),
                    "wrf_mass_weight")
        ctx.cg, ctx.nk = cg, nk
        ctx.save_for_backward(field, mut)
        return out

    @staticmethod
    def backward(ctx, gout):
        field, mut = ctx.saved_tensors
        gout = gout.contiguous()
        fb, mb = _zeros(field, mut)
        stream = _stream(field)
        with _on(field):
            rc = N.lib().wrf_mass_weight_adj(ctypes.byref(ctx.cg), _ptr(field), _ptr(mut), _ptr(gout), _ptr(fb),
                                             _ptr(mb), ctx.nk, stream)
        N.check(rc, "wrf_mass_weight_adj")
        return None, fb, mb


def mass_weight(field, mut, nk: int, rdx, rdy):
    """Differentiable mass_weight on levels below ``nk``."""
    return MassWeight.apply((nk, rdx, rdy), field, mut)


class _EddyViscosity:
    name = "wrf_eddy_viscosity"
    fields = ("u", "v", "ph", "xkmh", "xkhh")
    outputs = ("xkmh", "xkhh")
    data = ("phb", "msfux", "msfuy", "msfvx", "msfvy", "msftx", "msfty", "fnm", "fnp", "dn", "dnw")
    scratch = ("rdzw", "zx", "zy", "defor11", "defor22", "defor12")

    def _metrics(self, cg, tab):
        """The metrics and deformations, which each direction forms anew."""
        buf, at, n3 = _scratch_like(cg, per_point=len(self.scratch)), _field_index(), cg.nz * cg.ny * cg.nx
        for q, k in enumerate(self.scratch):
            tab[at[k]] = buf.data_ptr() + 4 * q * n3
        return buf

    def fwd(self, cg, tab, stream):
        buf = self._metrics(cg, tab)  # noqa: F841 (held through the call)
        return N.lib().wrf_eddy_viscosity(ctypes.byref(cg), tab, stream)

    def adj(self, cg, tab, btab, stream):
        buf, work = self._metrics(cg, tab), _scratch_like(cg, per_point=6)  # noqa: F841
        return N.lib().wrf_eddy_viscosity_adj(ctypes.byref(cg), tab, btab, _ptr(work), stream)


def eddy_viscosity(st: dict, data: dict, rdx, rdy, cf1: float, cf2: float, cf3: float):
    """Differentiable first-stage eddy viscosities (compute_diff_metrics,
    cal_deform_and_div, calculate_km_kh: pywrf/wrf_dynamics.py:491-995) from
    u, v and ph; returns (xkmh, xkhh).  ``st`` also maps the incoming xkmh
    and xkhh (which survive outside the formula's region)."""
    op = _EddyViscosity()
    cg = scalar_grid(st["u"].shape, rdx, rdy)
    cg.cf1, cg.cf2, cg.cf3 = float(cf1), float(cf2), float(cf3)
    return _TableOp.apply(op, cg, *[st[k] for k in op.fields], *[data[k] for k in op.data])


# the fields the dynamics part of an RK stage reads (state) beyond the
# acoustic stage's, and its constant arrays (data)
DYN_STATE = tuple(dict.fromkeys(STAGE_STATE + PREP_FIELDS + FORCES_INPUTS + _Addtend.fields +
                                ("moist", "xkmh", "xkhh", "moist_tend")))
DYN_DATA = tuple(dict.fromkeys(STAGE_DATA + PREP_DATA + FORCES_DATA + _Addtend.data + _EddyViscosity.data +
                               HDIFF_DATA + ("t_init",)))


def _first_stage_ops(bdy: dict, dtbc: float, nz: int) -> list:
    """The first stage's horizontal diffusion of u, v, w and theta into the
    physics tendencies and the lateral relaxation into the saved fields
    (pywrf/solver.py:1112-1203)."""
    ops = [_diffusion_op(k, k, f"r{k}_tendf", "mut", "xkmh") for k in ("u", "v", "w")]
    ops.append(_diffusion_op("m", "t", "t_tendf", "mut", "xkhh", base="t_init"))
    ops += [_relax_op("ru", "u_save", bdy["u"], "u", dtbc), _relax_op("rv", "v_save", bdy["v"], "v", dtbc)]
    for k, var in (("ph", "h"), ("t", "t")):
        ops += [_mass_weight_op(k, "mut", "_mass", nz), _relax_op("_mass", f"{k}_save", bdy[var], var, dtbc)]
    ops.append(_relax_op("mu", "mu_tend", bdy["m"], "m", dtbc))
    return ops


def dynamics_stage(st: dict, data: dict, bt: dict, rk_step: int, nsub: int, dts: float, *, epssm: float,
                   emdiv: float, smdiv: float, cf1: float, cf2: float, cf3: float, cfn: float, cfn1: float,
                   rdx: float, rdy: float, dtbc: float | None = None, theta_bias=None) -> dict:
    """The dynamics of one RK stage composed from the operators' Functions,
    in the reference's order (pywrf/solver.py:736-1492): rk_step_prep and
    its halo copies; at the first stage the physics tendencies from zero, the
    eddy viscosities and their halo copies; the advection of u, v, w and
    theta, the tendency terms; at the first stage the horizontal diffusion
    and the lateral relaxation; rk_addtend_dry (then ``theta_bias``, when
    given, added to t_tend); spec_bdytend of u, v, ph, t, mu; and the
    acoustic part (:func:`acoustic_stage`).  ``bt`` maps 'u', 'v', 'h', 't',
    'm' to dicts of their boundary arrays (txs txe tys tye; at the first
    stage also xs xe ys ye, with ``dtbc`` the boundary time); returns the
    state after the acoustic steps."""
    if rk_step not in (1, 2, 3):
        raise ValueError("rk_step is 1, 2 or 3")
    if rk_step == 1 and dtbc is None:
        raise ValueError("the first stage's relaxation needs dtbc")
    L, by = N.lib(), ctypes.byref
    cg = _chain_grid(st["u"].shape, rdx, rdy, epssm=epssm, emdiv=emdiv, smdiv=smdiv, cf1=cf1, cf2=cf2, cf3=cf3,
                     cfn=cfn, cfn1=cfn1)
    ops = [_table_chain_op(_CallOp("wrf_prep", PREP_FIELDS, PREP_OUTPUTS, PREP_DATA,
                                   lambda c, tab, s: L.wrf_prep(by(c), tab, 127, s),
                                   lambda c, tab, b, s: L.wrf_prep_adj(by(c), tab, b, 127, s))),
           _halo_op(("ru", "rv", "rw", "ww", "php", "alt", "p", "muu", "muv", "mut", "al", "ph"), "uvwwwtpuvtpw")]
    zeros = ("ru_tend", "rv_tend", "rw_tend", "t_tend", "ph_tend", "u_save", "v_save", "w_save", "ph_save", "t_save",
             "mu_tend", "mu_save")
    if rk_step == 1:
        tendf = ("ru_tendf", "rv_tendf", "rw_tendf", "ph_tendf", "t_tendf", "mu_tendf", "moist_tend")
        ops += [_zero_op(k, k) for k in tendf]
        ops += [_table_chain_op(_EddyViscosity()), _halo_op(("xkmh", "xkhh"), "tt")]
    ops += [_zero_op(k, k) for k in zeros]
    ops += [_advect_momentum_op(0, "u", "ru_tend"), _advect_momentum_op(1, "v", "rv_tend"),
            _advect_momentum_op(2, "w", "rw_tend"), _advect_scalar_op("t", "t_tend")]
    ops.append(_table_chain_op(_CallOp("wrf_forces", FORCES_INPUTS, FORCES_OUTPUTS, FORCES_DATA,
                                       lambda c, tab, s: L.wrf_forces(by(c), tab, 31, s),
                                       lambda c, tab, b, s: L.wrf_forces_adj(by(c), tab, b, 31, s))))
    if rk_step == 1:
        ops += _first_stage_ops(bt, dtbc, st["u"].shape[0])
    ops.append(_table_chain_op(_Addtend(rk_step)))
    s = _run_chain(ops, cg, st, data)
    if theta_bias is not None:
        s["t_tend"] = s["t_tend"] + theta_bias
    ops = [_spec_tend_op(k, bt[var], var) for k, var in (("ru_tend", "u"), ("rv_tend", "v"), ("ph_tend", "h"),
                                                         ("t_tend", "t"), ("mu_tend", "m"))]
    return _run_chain(ops + _acoustic_ops(rk_step, nsub, dts), cg, s, data)


class _MoistUpdate:
    name = "wrf_moist_update"
    fields = ("moist", "moist_old", "moist_tend", "advect_tend", "mu", "mu_1", "mub", "al", "alb", "muts", "ph", "p",
              "pb", "t")
    outputs = ("moist", "moist_old", "al", "p")
    data = ("msfty", "ru_m", "rv_m", "rdnw")

    def __init__(self, rk_step, dt_rk):
        self.rk_step, self.dt_rk = rk_step, float(dt_rk)

    def fwd(self, cg, tab, stream):
        status = _scratch_like(cg, per_column=1)  # counts NaN points for nobody
        tab[_field_index()["status"]] = status.data_ptr()
        return N.lib().wrf_moist_update(ctypes.byref(cg), tab, self.rk_step, self.dt_rk, stream)

    def adj(self, cg, tab, btab, stream):
        work = _scratch_like(cg, per_point=1)
        tab[_field_index()["status"]] = work.data_ptr()  # the reverse counts nothing
        return N.lib().wrf_moist_update_adj(ctypes.byref(cg), tab, btab, self.rk_step, self.dt_rk, _ptr(work), stream)


def moist_stage(st: dict, data: dict, rk_step: int, dt_rk: float, rdx, rdy, bt: dict | None = None,
                dtbc: float | None = None) -> dict:
    """The moisture part of an RK stage after its acoustic steps, composed
    from the operators' Functions (pywrf/solver.py:1548-1712): advection of
    qv .. qg by the averaged fluxes; at the first stage the horizontal
    diffusion of each species (mass muts, viscosity xkhh), and the relaxation
    and specified tendency of qv (``bt['q']``: its eight boundary arrays,
    ``dtbc`` the boundary time); rk_update_scalar, flow_dep_bdy of qc .. qg,
    calc_p_rho_phi and, before the last stage, the halo copies."""
    if rk_step == 1 and (bt is None or dtbc is None):
        raise ValueError("the first stage's qv relaxation needs its boundary arrays and dtbc")
    cg = scalar_grid(st["u"].shape, rdx, rdy)
    ops = [_advect_moist_op()]
    if rk_step == 1:
        ops.append(_diffusion_op("m", "moist", "moist_tend", "muts", "xkhh"))
        ops += _relax_qv_ops(st["u"].shape[0], bt["q"], dtbc)
    # (the averaged fluxes enter flow_dep_bdy by their sign alone)
    ops.append(_table_chain_op(_MoistUpdate(rk_step, dt_rk), held=("ru_m", "rv_m")))
    if rk_step < 3:
        ops.append(_halo_op(("u", "v", "w", "t", "ph", "mu", "moist"), "UVwpwtM"))
    return _run_chain(ops, cg, st, data)


def _relax_qv_ops(nz: int, bdy: dict, dtbc: float) -> list:
    """qv's lateral relaxation and specified tendency into its slot of
    moist_tend (pywrf/solver.py:1600-1640)."""
    L, by = N.lib(), ctypes.byref
    arrays = [bdy[k] for k in BDY_NAMES]

    def fwd(cg, st, out, const, stream):
        arr = (ctypes.c_void_p * 8)(*[_ptr(v) for v in arrays])
        tend = out["moist_tend"][1]
        mass = torch.zeros_like(tend)
        _rc(L.wrf_mass_weight(by(cg), _ptr(st["moist"][1]), _ptr(st["mut"]), _ptr(mass), nz - 1, stream),
            "wrf_mass_weight")
        _rc(L.wrf_relax_bdytend(by(cg), _ptr(mass), _ptr(tend), arr, b"t", float(dtbc), stream), "wrf_relax_bdytend")
        _rc(L.wrf_spec_bdytend(by(cg), _ptr(tend), *[_ptr(bdy[k]) for k in ("txs", "txe", "tys", "tye")], b"t",
                               stream), "wrf_spec_bdytend")

    def bwd(cg, saved, bars, const, stream):
        if bars.get("moist_tend") is None:
            return
        b, gk = bars.need(saved), bars["moist_tend"][1]
        _rc(L.wrf_spec_bdytend_adj(by(cg), _ptr(gk), b"t", stream), "wrf_spec_bdytend_adj")
        mass = torch.zeros_like(gk)
        _rc(L.wrf_relax_bdytend_adj(by(cg), _ptr(gk), _ptr(mass), b"t", stream), "wrf_relax_bdytend_adj")
        _rc(L.wrf_mass_weight_adj(by(cg), _ptr(saved["moist"][1]), _ptr(saved["mut"]), _ptr(mass),
                                  _ptr(b["moist"][1]), _ptr(b["mut"]), nz - 1, stream), "wrf_mass_weight_adj")

    return [_ChainOp(("moist", "mut"), ("moist_tend",), fwd, bwd)]


RK_STATE = tuple(dict.fromkeys(DYN_STATE + _MoistUpdate.fields + ("ru_m", "rv_m", "ww_m")))
RK_DATA = tuple(dict.fromkeys(DYN_DATA + ("msftx", "fnm", "fnp", "rdnw")))


def rk_stage(st: dict, data: dict, bt: dict, rk_step: int, nsub: int, dts: float, dt_rk: float, **sc) -> dict:
    """One RK stage of the step, composed: :func:`dynamics_stage` then
    :func:`moist_stage`; ``sc`` as for :func:`dynamics_stage` (at the first
    stage ``bt`` also holds 'q', qv's boundary arrays)."""
    s = dynamics_stage(st, data, bt, rk_step, nsub, dts, **sc)
    return moist_stage(s, data, rk_step, dt_rk, sc["rdx"], sc["rdy"], bt, sc.get("dtbc"))


BDY_FINAL_ARRAYS = tuple(f"{v}_{n}" for v in ("u", "v", "t", "ph", "qv")
                         for n in ("bxs", "bxe", "bys", "bye", "btxs", "btxe", "btys", "btye"))


class _BdyFinal:
    name = "wrf_bdy_final"
    fields = ("u", "v", "t", "ph", "moist", "w", "muus", "muvs", "muts")
    outputs = ("u", "v", "t", "ph", "moist", "w")
    data = ("msfuy", "msfvx", "msftx", "msfty", "ht", "dscal") + BDY_FINAL_ARRAYS

    def fwd(self, cg, tab, stream):
        return N.lib().wrf_bdy_final(ctypes.byref(cg), tab, stream)

    def adj(self, cg, tab, btab, stream):
        return N.lib().wrf_bdy_final_adj(ctypes.byref(cg), tab, btab, stream)


def boundary_arrays(bdy: dict) -> dict:
    """The state table's boundary-array fields (u_bxs .. qv_btye) from
    per-variable dicts in the solver layout ('u', 'v', 't', 'ph', 'qv' each
    mapping xs xe ys ye txs txe tys tye)."""
    out = {}
    for v in ("u", "v", "t", "ph", "qv"):
        for n, key in (("bxs", "xs"), ("bxe", "xe"), ("bys", "ys"), ("bye", "ye"), ("btxs", "txs"),
                       ("btxe", "txe"), ("btys", "tys"), ("btye", "tye")):
            out[f"{v}_{n}"] = bdy[v][key]
    return out


def step_end(st: dict, data: dict, bdy: dict, dtbc: float, *, cf1: float, cf2: float, cf3: float, rdx: float,
             rdy: float) -> dict:
    """The end of a step after its microphysics, composed
    (pywrf/solver.py:1776-1910): the halo copies of u_1, u, v_1, v, w_1, w,
    t_1, t, ph_1, ph, mu_1, mu and qv .. qg, spec_bdy_final of u, v, t, ph,
    qv and set_w_surface.  ``bdy`` maps 'u', 'v', 't', 'ph', 'qv' to their
    boundary arrays (xs .. tye)."""
    s = dict(st)
    names = ("u_1", "u", "v_1", "v", "w_1", "w", "t_1", "t", "ph_1", "ph", "mu_1", "mu", "moist")
    s.update(zip(names, halos([s[k] for k in names], "UUVVwwppwwttM", rdx, rdy)))
    op = _BdyFinal()
    cg = scalar_grid(s["u"].shape, rdx, rdy)
    cg.cf1, cg.cf2, cg.cf3 = float(cf1), float(cf2), float(cf3)
    dscal = torch.zeros(16, dtype=torch.float32, device=s["u"].device)
    dscal[:1].fill_(float(dtbc))  # a fill launch, not a host copy: the step stays capturable in a CUDA graph
    dd = {**{k: data[k] for k in ("msfuy", "msfvx", "msftx", "msfty", "ht")}, "dscal": dscal,
          **boundary_arrays(bdy)}
    outs = _TableOp.apply(op, cg, *[s[k] for k in op.fields], *[dd[k] for k in op.data])
    s.update(dict(zip(op.outputs, outs)))
    return s


class _Microphysics:
    """The step's microphysics (moist_physics_prep_em, WSM6,
    moist_physics_finish_em, calc_p_rho_phi) as a table operator; the
    precipitation accumulators and the diagnostic tendencies it also writes
    go to scratch (they do not feed back into the state)."""
    name = "wrf_microphysics_op"
    fields = ("t", "moist", "al", "p", "ph", "h_diabatic", "mu", "muts")
    outputs = ("t", "moist", "al", "p", "h_diabatic")
    data = ("alb", "pb", "phb", "rdnw")
    scratch3 = ("qv_diabatic", "qc_diabatic", "wsm_t", "wsm_qr0s")
    scratch2 = ("rainnc", "rainncv", "snownc", "snowncv", "graupelnc", "graupelncv", "sr")

    def _scratch(self, cg, tab):
        """The diagnostics and accumulators the block writes, in ``tab``."""
        at, n2, n3 = _field_index(), cg.ny * cg.nx, cg.nz * cg.ny * cg.nx
        buf = _scratch_like(cg, per_point=len(self.scratch3), per_column=len(self.scratch2))
        for q, k in enumerate(self.scratch3):
            tab[at[k]] = buf.data_ptr() + 4 * q * n3
        for q, k in enumerate(self.scratch2):
            tab[at[k]] = buf.data_ptr() + 4 * (len(self.scratch3) * n3 + q * n2)
        return buf

    def fwd(self, cg, tab, stream):
        buf = self._scratch(cg, tab)  # noqa: F841 (held through the call)
        return N.lib().wrf_microphysics_op(ctypes.byref(cg), tab, stream)

    def reverse(self, cg, named, bars, stream):
        # the state after the block, recomputed from clones of the inputs it
        # updates (the other fields are the same tensors)
        post = {k: named[k].clone() for k in self.outputs}
        ptab = _table({**named, **post})
        buf = self._scratch(cg, ptab)  # noqa: F841
        rc = N.lib().wrf_microphysics_op(ctypes.byref(cg), ptab, stream)
        if rc:
            return rc
        # the base state's cotangents, which the block accumulates and nobody takes
        dropped = dict(zip(("alb", "pb"), _zeros(named["t"], named["t"])))
        n = ctypes.c_size_t(0)
        rc = N.lib().wrf_microphysics_adj_work(ctypes.byref(cg), ctypes.byref(n))
        if rc:
            return rc
        work = torch.empty(int(n.value), dtype=torch.float32, device=named["t"].device)
        return N.lib().wrf_microphysics_adj(ctypes.byref(cg), _table(named), ptab, _table({**bars, **dropped}),
                                            _ptr(work), n, None, stream)


def microphysics(st: dict, data: dict, dt: float, rdx, rdy) -> dict:
    """Differentiable microphysics of the step (pywrf/solver.py:1714-1766):
    returns ``st`` with t, moist, al, p and h_diabatic replaced.  Its reverse
    is the equation of state's exact reverse, then that of prep + WSM6 + finish
    over a restatement of the scheme.  With one time-split loop (dt up to 240 s)
    the falls of a column run once on taped scalars, reversed by one sweep of
    their tapes, and all else takes forward-mode tangents per level; with several
    loops the whole column is taped.  A column whose tape outgrows the capacity
    takes tangents of the whole restatement."""
    op = _Microphysics()
    cg = scalar_grid(st["t"].shape, rdx, rdy)
    cg.dt = float(dt)
    outs = _TableOp.apply(op, cg, *[st[k] for k in op.fields], *[data[k] for k in op.data])
    return {**st, **dict(zip(op.outputs, outs))}


STEP_DATA = tuple(dict.fromkeys(RK_DATA + ("msfuy", "msfvx", "msftx", "msfty", "ht")))


def step(st: dict, data: dict, bdy: dict, dtbc: float, *, dt: float, soundsteps: int, microphysics=None,
         theta_bias=None, **sc) -> dict:
    """One time step composed from the operators' Functions
    (pywrf/solver.py:709-1910): the three RK stages (:func:`rk_stage`), then
    ``microphysics`` (a differentiable callable on the state dict, or None
    for none: the step of a model without microphysics), then
    :func:`step_end`.  ``bdy`` maps 'u', 'v', 'ph', 't', 'mu', 'qv' to their
    boundary arrays (xs .. tye); ``sc`` holds epssm, emdiv, smdiv, cf1, cf2,
    cf3, cfn, cfn1, rdx, rdy; ``theta_bias`` is added to t_tend in every
    stage."""
    bt = {"u": bdy["u"], "v": bdy["v"], "h": bdy["ph"], "t": bdy["t"], "m": bdy["mu"], "q": bdy["qv"]}
    s = dict(st)
    for rk in (1, 2, 3):
        nsub = {1: 1, 2: soundsteps // 2, 3: soundsteps}[rk]
        dts = dt / 3.0 if rk == 1 else dt / soundsteps
        dt_rk = {1: dt / 3.0, 2: 0.5 * dt, 3: dt}[rk]
        s = rk_stage(s, data, bt, rk, nsub, dts, dt_rk, dtbc=dtbc, theta_bias=theta_bias, **sc)
    if microphysics is not None:
        s = microphysics(s)
    return step_end(s, data, bdy, dtbc, cf1=sc["cf1"], cf2=sc["cf2"], cf3=sc["cf3"], rdx=sc["rdx"], rdy=sc["rdy"])
