"""Kernels and dispatch branches at the sizes where they can go wrong: tile
and warp remainders, the smallest and largest depths, rows that are and are
not whole 16-byte words."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from pywrf_b200 import _native as N
from pywrf_b200 import adjoint as A
from pywrf_b200 import synthetic
from pywrf_b200.config import Grid
from pywrf_b200.solver import Integrator
from pywrf_b200.state import DeviceState, make_cgrid

pytestmark = pytest.mark.gpu


def _cg(nx, ny, nz, dt=45.0):
    return make_cgrid(Grid.make(nx, ny, nz, 9000.0, 9000.0, dt),
                      {"cf1": 0.0, "cf2": 0.0, "cf3": 0.0, "cfn": 0.0, "cfn1": 0.0})


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n,nz", [(316, 12), (317, 17)], ids=["316x12", "317x17"])
def test_marching_acoustic_columns_equal_the_tiled_form_bitwise(n, nz):
    """Domains wide enough for the one-thread-per-column acoustic kernel
    against the point forms (which keep the tiled kernel), every field."""
    spec = synthetic.CaseSpec(n=n, nz=nz, nsteps=1, bdy_tend_amp=1.0e-4, seed=5)
    g = synthetic.grid_for(spec)
    inputs, bdy = synthetic.build(spec)
    states = []
    for form in (N.WRF_FORM_FAST, N.WRF_FORM_POINT):
        prev = N.lib().wrf_set_kernel_form(form)
        try:
            st = DeviceState.from_inputs(g, inputs, bdy, device="cuda")
            it = Integrator(st)
            it.run(1, graph=False)
            torch.cuda.synchronize()
            assert it.status()["wait_timeouts"] == 0
        finally:
            N.lib().wrf_set_kernel_form(prev)
        states.append(st)
    fast, point = states
    bad = [k for k in fast.names if not torch.equal(fast[k].view(torch.int32), point[k].view(torch.int32))]
    assert not bad, bad


@pytest.mark.parametrize("ncol,nz", [(1, 3), (33, 12), (1000, 41), (31, 64)])
def test_implicit_w_solve_and_its_reverse(ncol, nz):
    """The column solve and its transposed solve against float64 loops.  The
    coefficients are those of a diagonally dominant system (|a alpha|, |gamma|
    < 1/2), whose rounding stays within a few ulp per level: 64 levels of
    half an ulp each way and twice that for the reverse, 1e-5 of the norm."""
    gen = torch.Generator(device="cuda").manual_seed(ncol + nz)
    x, a, al, ga, cot = (torch.randn(nz, ncol, generator=gen, device="cuda") for _ in range(5))
    a, al, ga = 0.3 * torch.tanh(a), 1.0 + 0.2 * torch.tanh(al), 0.3 * torch.tanh(ga)
    args = [v.clone().requires_grad_(True) for v in (x, a, al, ga)]
    w = A.vsolve_w(*args)
    grads = torch.autograd.grad(w, args, grad_outputs=cot)
    ref = [v.double().cpu().requires_grad_(True) for v in (x, a, al, ga)]
    y = [ref[0][0]]
    for k in range(1, nz):
        y.append((ref[0][k] - ref[1][k] * y[k - 1]) * ref[2][k])
    z = list(y)
    for k in range(nz - 2, 0, -1):
        z[k] = y[k] - ref[3][k] * z[k + 1]
    z = torch.stack(z)
    want = (z.detach(),) + torch.autograd.grad(z, ref, grad_outputs=cot.double().cpu())
    for got, exact in zip((w.detach(),) + grads, want):
        err = (got.double().cpu() - exact).norm() / exact.norm().clamp_min(1e-30)
        assert float(err) < 1e-5


@pytest.mark.parametrize("nx,ny,nz,dt", [(24, 25, 12, 45.0), (41, 30, 48, 150.0), (37, 24, 64, 45.0),
                                         (24, 24, 20, 250.0)])
def test_wsm6_with_caller_scratch_equals_the_fused_kernel_bitwise(nx, ny, nz, dt):
    """Columns that hold nothing, one species, or all of them side by side."""
    gen = torch.Generator(device="cuda").manual_seed(nx * nz)
    rnd = lambda *s: torch.rand(*s, generator=gen, device="cuda")  # noqa: E731
    k = torch.linspace(0.0, 1.0, nz, device="cuda")[:, None, None]
    p = 1.0e5 * torch.exp(-1.6 * k) * (1.0 + 0.001 * rnd(nz, ny, nx))
    pii = (p / 1.0e5) ** 0.2857143
    th = 295.0 + 45.0 * k + rnd(nz, ny, nx)
    f = dict(th=th, qv=0.012 * torch.exp(-5.0 * k) * (0.7 + 0.6 * rnd(nz, ny, nx)))
    for i, q in enumerate(("qc", "qr", "qi", "qs", "qg")):
        col = (rnd(ny, nx) < 0.4).float() * (rnd(nz, ny, nx) < 0.5).float()
        f[q] = 1.0e-3 * col * rnd(nz, ny, nx) ** 4 - (1.0e-9 if i == 0 else 0.0)
    f |= dict(rho=p / (287.0 * th * pii), pii=pii, p=p, dz=200.0 + 400.0 * k.expand(nz, ny, nx))
    f = {a: b.contiguous() for a, b in f.items()}
    cg, L = _cg(nx, ny, nz, dt), N.lib()
    n = ctypes.c_size_t(0)
    N.check(L.wrf_wsm6_work_floats(ctypes.byref(cg), dt, ctypes.byref(n)), "work")
    assert (n.value == 0) == (dt >= 240.0)
    outs = []
    for split in (False, True):
        d = {a: b.clone() for a, b in f.items()}
        flat = [torch.zeros(ny, nx, device="cuda") for _ in range(7)]
        args = [ctypes.byref(cg)] + [_p(d[a]) for a in d] + [ctypes.c_float(dt)] + [_p(v) for v in flat]
        if split:
            work = torch.full((max(n.value, 1),), float("nan"), device="cuda")
            N.check(L.wrf_wsm6_work(*args, _p(work), n.value, _stream()), "wrf_wsm6_work")
        else:
            N.check(L.wrf_wsm6(*args, _stream()), "wrf_wsm6")
        torch.cuda.synchronize()
        outs.append(list(d.values()) + flat)
    assert float(outs[0][11].max()) > 0.0  # it rained
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    if n.value:
        rc = L.wrf_wsm6_work(*args, _p(work), n.value - 1, _stream())
        assert rc == N.WRF_EINVAL


LETTERS = "uvwtpdefUVxyZ"


@pytest.mark.parametrize("nx,ny", [(24, 24), (32, 27), (45, 30), (61, 38), (132, 70)])
def test_batched_halos_and_their_adjoint(nx, ny):
    """One launch for a batch of fields against the in-place copies of each
    (bitwise), and the adjoint against the transposed copy (dot products of
    integers, exact in float64)."""
    nz = 12
    gen = torch.Generator(device="cuda").manual_seed(nx)
    num = lambda *s: torch.randint(-8, 9, s, generator=gen, device="cuda").float()  # noqa: E731
    fields = [num(nz, ny, nx) for _ in LETTERS] + [num(7, nz, ny, nx)] + [num(ny, nx) for _ in "tuv"]
    letters = LETTERS + "M" + "tuv"
    leaves = [f.clone().requires_grad_(True) for f in fields]
    outs = A.halos(leaves, letters)
    for f, v, o in zip(fields, letters, outs):
        if v == "Z":
            want = A.zero_grad_w(f)
        elif v == "M":
            want = torch.stack([f[0]] + [A.halo(f[m], "p") for m in range(1, 7)])
        else:
            want = A.halo(f, v)
        assert torch.equal(o.detach(), want), v
    cots = [num(*f.shape) for f in fields]
    grads = torch.autograd.grad(outs, leaves, grad_outputs=cots)
    for f, v, o, c, gr in zip(fields, letters, outs, cots, grads):
        assert float((o.detach().double() * c).sum()) == float((f.double() * gr).sum()), v


@pytest.mark.parametrize("rows,cols", [(1, 7), (3, 256), (5, 264), (6, 2560), (130, 8192), (2, 8190)])
def test_row_sums_of_bf16_rows(rows, cols):
    """Row sums against float64 (float32 partial sums of at most 64 terms and
    two trees of eight levels: 80 roundings of half an ulp of the row's
    absolute sum)."""
    gen = torch.Generator(device="cuda").manual_seed(cols)
    a = torch.randn(rows, cols, generator=gen, device="cuda").to(torch.bfloat16)
    out = torch.empty(rows, device="cuda")
    N.check(N.lib().wrf_rowsum_bf16(_p(a), rows, cols, _p(out), _stream()), "rowsum")
    want = a.double().sum(1)
    assert bool(((out.double() - want).abs() <= 80 * 6e-8 * a.double().abs().sum(1)).all())


@pytest.mark.parametrize("r,c", [(64, 62), (33, 40), (1, 5), (130, 258)])
def test_transpose_and_adam_tiles(r, c):
    """The transposed bf16 copy (both element widths) and one Adam step of a
    batch of two matrices, one of them without copies, against float64 (a
    handful of float32 roundings of the update, 1e-6 of its size)."""
    gen = torch.Generator(device="cuda").manual_seed(r)
    a = torch.randn(r, c, generator=gen, device="cuda").to(torch.bfloat16)
    out = torch.empty(c, r, dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().wrf_transpose_bf16(_p(a), r, c, _p(out), _stream()), "transpose")
    assert torch.equal(out, a.t())
    w, m, v = (torch.randn(r, c, generator=gen, device="cuda") for _ in range(3))
    v = v.abs()
    gp = torch.randn(3, r, c, generator=gen, device="cuda")
    bias, bm, bv, bg = torch.randn(4, c, generator=gen, device="cuda")
    bv = bv.abs()
    wb, wtb = torch.empty_like(a), torch.empty_like(out)
    lr, b1, b2, eps = (ctypes.c_float(q).value for q in (1e-2, 0.9, 0.999, 1e-8))  # as the entry takes them
    exact = []
    for x, y, z, g in ((w, m, v, gp.double().sum(0)), (bias, bm, bv, bg.double())):
        mm, vv = b1 * y.double() + (1 - b1) * g, b2 * z.double() + (1 - b2) * g * g
        step = (mm / (1 - b1 ** 3)) / ((vv / (1 - b2 ** 3)).sqrt() + eps)
        exact.append(x.double() - lr * step)
    items = (N.WrfAdamItemC * 2)(
        N.WrfAdamItemC(w.data_ptr(), gp.data_ptr(), m.data_ptr(), v.data_ptr(), wb.data_ptr(), wtb.data_ptr(), r * c,
                       3, r, c, 0.0),
        N.WrfAdamItemC(bias.data_ptr(), bg.data_ptr(), bm.data_ptr(), bv.data_ptr(), None, None, c, 1, 1, c, 0.0))
    N.check(N.lib().wrf_adam_batch(2, items, lr, b1, b2, eps, 3, _stream()), "adam")
    for got, want in zip((w, bias), exact):
        assert float((got.double() - want).abs().max()) <= 1e-6 * float(want.abs().max()) + 1e-6
    assert torch.equal(wb, w.to(torch.bfloat16)) and torch.equal(wtb, w.to(torch.bfloat16).t())


@pytest.mark.parametrize("n,nz", [(28, 12), (37, 20), (64, 33)])
def test_horizontal_diffusion_of_every_stagger(n, nz):
    """The stand-alone diffusion of each variable against its reverse: both
    are bilinear, <D(f), c> = <f, D^T c> (float32 products summed in float64:
    1e-5 of the sum of their sizes)."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    data = {k: 1.0 + 0.1 * torch.rand(n, n, generator=gen, device="cuda") for k in A.HDIFF_DATA}
    mut, xk = 9.0e4 + 100.0 * rnd(n, n), 1.0e3 * (1.0 + 0.1 * rnd(nz, n, n))
    for var in "uvwm":
        f, c = rnd(nz, n, n).requires_grad_(True), rnd(nz, n, n)
        out = A.horizontal_diffusion(var, f, torch.zeros_like(f), mut, xk, data, 1 / 9000.0, 1 / 9000.0)
        (g,) = torch.autograd.grad(out, f, grad_outputs=c)
        lhs, rhs = (out.detach().double() * c).sum(), (f.detach().double() * g).sum()
        size = (out.detach().double() * c).abs().sum()
        assert float(size) > 0 and abs(float(lhs - rhs)) <= 1e-5 * float(size), var




@pytest.mark.parametrize("n,nz", [(24, 12), (37, 16), (64, 17), (33, 41)])
def test_advance_uv_reverse_at_the_ends_of_its_level_chunks(n, nz):
    """The pressure-gradient part A B + C D is homogeneous in its factors: of
    degree one in (muu, muv, php), of (ph, alt, al) in B, of (p, mu) in D and
    of (alt p, al pb) pairwise, so by Euler's identity the products of the
    values and their cotangents agree in four ways (float32 terms of some ten
    roundings summed in float64: 1e-5 of the sum of their sizes)."""
    gen = torch.Generator(device="cuda").manual_seed(n * nz)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    two_d = {"mu", "muu", "muv", "mudf"}
    x = {k: rnd(*((n, n) if k in two_d else (nz, n, n))).requires_grad_(True) for k in A.UV_INPUTS}
    data = {k: (rnd(nz) if k in ("fnm", "fnp", "rdnw") else 1.0 + 0.1 * rnd(n, n)) for k in A.UV_DATA}
    u, v = A.advance_uv(x, data, 9.0, 0.01, 2.0, -1.5, 0.5, 1 / 9000.0, 1 / 9000.0)
    grads = torch.autograd.grad((u, v), list(x.values()), grad_outputs=[rnd(nz, n, n), rnd(nz, n, n)])
    prod = {k: (x[k].detach().double() * gk) for k, gk in zip(x, grads)}

    def agree(left, right):
        a, b = (sum(prod[k].sum() for k in side) for side in (left, right))
        size = sum(prod[k].abs().sum() for k in left + right)
        assert float(size) > 0 and abs(float(a - b)) <= 1e-5 * float(size), (left, right)

    agree(("cqu", "cqv"), ("muu", "muv", "php"))
    agree(("muu", "muv"), ("ph", "alt", "al"))
    agree(("p", "mu"), ("alt", "php"))
    agree(("pb",), ("al",))


@pytest.mark.parametrize("n,nz", [(24, 12), (41, 15), (50, 40)])
def test_advect_scalar_reverse_is_its_transpose(n, nz):
    """The advection is linear in the field, and in the fluxes for fixed
    signs: <A q, c> = <q, A^T c> = the fluxes' products (1e-5 of the sum of
    the sizes)."""
    gen = torch.Generator(device="cuda").manual_seed(n + nz)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    q, ru, rv, rom = (rnd(nz, n, n).requires_grad_(True) for _ in range(4))
    c = rnd(nz, n, n)
    out = A.advect_scalar(q, torch.zeros_like(c), ru, rv, rom, 1.0 + 0.1 * rnd(n, n), rnd(nz), rnd(nz), rnd(nz),
                          1 / 9000.0, 1 / 9000.0)
    grads = torch.autograd.grad(out, (q, ru, rv, rom), grad_outputs=c)
    prods = [a.detach().double() * b for a, b in zip((out, q, ru, rv, rom), (c,) + grads)]
    lhs, field, fluxes = prods[0].sum(), prods[1].sum(), sum(p.sum() for p in prods[2:])
    size = float(prods[0].abs().sum() + prods[1].abs().sum() + sum(p.abs().sum() for p in prods[2:]))
    assert size > 0 and abs(float(lhs - field)) <= 1e-5 * size and abs(float(lhs - fluxes)) <= 1e-5 * size


@pytest.mark.parametrize("n", [300, 61], ids=["sorted", "own"])
def test_microphysics_reverse_by_levels_against_the_tangents(n):
    """Domains on either side of the line from which a block sorts its points
    before their tangents: the column, sedimentation tapes and all, against
    forward-mode tangents of the whole column (the tape capacity at 1), to the
    float32 summation order that the small case is held to (relative L2 1e-5)."""
    from test_gpu_adjoint import MP_OUT, _microphysics_state_before_step2

    g, snap = _microphysics_state_before_step2()
    pick = 6 + np.arange(n) % 16

    def wide(v):
        v = np.asarray(v, np.float32)
        if v.ndim >= 2 and v.shape[-2:] == (g.ny, g.nx):
            v = v[..., pick[:, None], pick[None, :]]
        return torch.tensor(np.ascontiguousarray(v), device="cuda")

    st = {k: wide(snap[k]) for k in A._Microphysics.fields}
    data = {k: wide(snap[k]) for k in A._Microphysics.data}
    st["t"] += 0.2 * torch.sin(torch.arange(st["t"].numel(), device="cuda").view_as(st["t"]).float())
    dt = float(g.dt)
    out = A.microphysics(st, data, dt, g.rdx, g.rdy)
    cg = A.scalar_grid(st["t"].shape, g.rdx, g.rdy)
    cg.dt = dt
    tab = A._table({**st, **data})
    post = A._table({**st, **data, **{k: out[k].detach() for k in ("t", "moist", "al", "p")}})
    gen = torch.Generator(device="cuda").manual_seed(n)
    seeds = {k: torch.randn(st[k].shape, generator=gen, device="cuda") for k in MP_OUT}

    def reverse(capacity):
        prev = ctypes.c_int(-1)
        N.check(N.lib().wrf_set_microphysics_tape_capacity(capacity, ctypes.byref(prev)), "capacity")
        try:
            bars = {k: torch.zeros_like(st[k]) for k in ("t", "moist", "al", "p", "ph", "mu", "muts", "h_diabatic")}
            bars.update({k: torch.zeros_like(st["t"]) for k in ("alb", "pb")})
            for k in MP_OUT:
                bars[k].copy_(seeds[k])
            words = ctypes.c_size_t(0)
            N.check(N.lib().wrf_microphysics_adj_work(ctypes.byref(cg), ctypes.byref(words)), "work")
            work = torch.empty(int(words.value), dtype=torch.float32, device="cuda")
            N.check(N.lib().wrf_microphysics_adj(ctypes.byref(cg), tab, post, A._table(bars), _p(work), words, None,
                                                 _stream()), "adj")
            torch.cuda.synchronize()
            return bars
        finally:
            N.check(N.lib().wrf_set_microphysics_tape_capacity(prev.value, None), "restore")

    taped, tangents = reverse(0), reverse(1)
    for k in ("t", "moist", "al", "p", "ph"):
        a, b = taped[k].double(), tangents[k].double()
        assert float((a - b).norm()) <= 1e-5 * float(b.norm()), k
    assert float(taped["moist"][3].abs().max()) > 0.0


def _column_operator(name, x, data, sc):
    """The operator's outputs on CUDA tensors, in the order of its fixture's
    cotangents."""
    rd = (1.0 / sc["dx"], 1.0 / sc["dy"])
    if name == "coefw":
        return A.coef_w(x["mut"], x["cqw"], x["c2a"], data["rdn"], data["rdnw"], sc["dts"], epssm=sc["epssm"])
    if name == "prho":
        return A.calc_p_rho(x, data["rdnw"], sc["smdiv"], 1, *rd)
    if name == "mut":
        out = A.advance_mu_t(x, data, sc["dts"], sc["epssm"], *rd)
        return [out[k] for k in A.MUT_OUTPUTS]
    out = A.advance_w(x, data, sc["dts"], sc["epssm"], sc["cf1"], sc["cf2"], sc["cf3"], *rd)
    return [out[k] for k in A.AW_OUTPUTS]


def _column_oracle(name, g, x, data, sc):
    from oracle import dynamics as OD

    x = {k: v.copy() for k, v in x.items()}
    if name == "coefw":
        out = [np.zeros_like(x["cqw"]) for _ in range(3)]
        OD.calc_coef_w(g, *out, x["mut"], x["cqw"], data["rdn"], data["rdnw"], x["c2a"], sc["dts"], sc["epssm"])
        return out
    if name == "prho":
        pm1 = OD.calc_p_rho(g, *[x[k] for k in A.PRHO_INPUTS], data["rdnw"], sc["smdiv"], 1)
        return [x["al"], x["p"], pm1]
    names, outs = (A._MUT_FIELD, A.MUT_OUTPUTS) if name == "mut" else (A._AW_FIELD, A.AW_OUTPUTS)
    st = {names.get(k, k): v for k, v in x.items()} | data
    if name == "mut":
        OD.advance_mu_t(g, st, sc["dts"], sc["epssm"], 1)
    else:
        OD.advance_w(g, st, sc["dts"], sc["epssm"], sc["cf1"], sc["cf2"], sc["cf3"])
    return [st[names.get(k, k)] for k in outs]


@pytest.mark.parametrize("name,inputs,data", [("coefw", ("mut", "cqw", "c2a"), ("rdn", "rdnw")),
                                              ("prho", A.PRHO_INPUTS, ("rdnw",)),
                                              ("mut", A.MUT_INPUTS, A.MUT_DATA), ("advw", A.AW_INPUTS, A.AW_DATA)],
                         ids=["coef_w", "calc_p_rho", "advance_mu_t", "advance_w"])
def test_column_reverses_at_the_greatest_depth(name, inputs, data):
    """64 levels, the deepest accepted column and so the largest shared
    memory: the operator against the float64 oracle on its fixture's profiles
    stretched over the column, and the reverse's derivative along one random
    direction per input against the oracle's central differences (the
    fixtures' tolerance, of the gradient's size: a sum of 64 levels' terms in
    float32)."""
    from helpers import load_npz, rel_l2

    z, nz = load_npz(f"{name}_adj_ref64.npz"), 64
    sc = {k: float(z[k]) for k in ("dts", "epssm", "smdiv", "cf1", "cf2", "cf3") if k in z}
    g = synthetic.grid_for(synthetic.CaseSpec(n=24, nz=nz))
    sc |= {"dx": g.dx, "dy": g.dy}

    def deep(v):
        if v.ndim == 2:
            return v.astype(np.float32)
        at = np.linspace(0.0, v.shape[0] - 1.0, nz)
        lo = np.minimum(at.astype(int), v.shape[0] - 2)
        w = (at - lo).reshape((nz,) + (1,) * (v.ndim - 1))
        return ((1.0 - w) * v[lo] + w * v[lo + 1]).astype(np.float32)

    x, dd = {k: deep(z[k]) for k in inputs}, {k: deep(z[k]) for k in data}
    xg = {k: torch.tensor(v, device="cuda").requires_grad_(True) for k, v in x.items()}
    outs = _column_operator(name, xg, {k: torch.tensor(v, device="cuda") for k, v in dd.items()}, sc)
    x64, d64 = ({k: v.astype(np.float64) for k, v in q.items()} for q in (x, dd))
    want = _column_oracle(name, g, x64, d64, sc)
    rng = np.random.default_rng(64)
    cots = [rng.standard_normal(o.shape).astype(np.float32) for o in want]
    for o, ref in zip(outs, want):
        assert rel_l2(o.detach().cpu().numpy(), ref) < 1e-5
    grads = torch.autograd.grad(outs, list(xg.values()), grad_outputs=[torch.tensor(c, device="cuda") for c in cots])

    def loss(v):
        return sum(float((o * c).sum()) for o, c in zip(_column_oracle(name, g, v, d64, sc), cots))

    for k, gk in zip(inputs, grads):
        gr, d = gk.double().cpu().numpy(), rng.standard_normal(x64[k].shape)
        eps = float(z[f"fd_eps_{k}"]) if f"fd_eps_{k}" in z else 1e-4 * float(np.abs(x64[k]).max())
        fd = (loss({**x64, k: x64[k] + eps * d}) - loss({**x64, k: x64[k] - eps * d})) / (2.0 * eps)
        assert abs(float((gr * d).sum()) - fd) <= 2e-4 * float(np.sqrt((gr * gr).sum())) + 1e-9, k


@pytest.mark.parametrize("nx,ny", [(6120, 24), (6121, 24), (24, 6122), (30000, 24), (24, 30001)])
def test_halo_copies_of_long_rows_and_columns(nx, ny):
    """Either side of the length whose edges fit the halo kernel's shared
    memory, and past the largest a block can have: the in-place copies against
    the gathered ones, every stagger, bitwise."""
    nz = 12
    gen = torch.Generator(device="cuda").manual_seed(nx)
    fields = [torch.rand(nz, ny, nx, generator=gen, device="cuda") for _ in LETTERS]
    fields += [torch.rand(ny, nx, generator=gen, device="cuda") for _ in "tuv"]
    letters = LETTERS + "tuv"
    for f, v, want in zip(fields, letters, A.halos(fields, letters)):
        assert torch.equal(A.zero_grad_w(f) if v == "Z" else A.halo(f, v), want), v


@pytest.mark.parametrize("op,outputs", [(0, ("ph_tend", "ru_tend", "rv_tend", "rw_tend", "cqw")), (1, ("advect_tend",)),
                                        (2, ("ru_tend", "rv_tend", "rw_tend")), (3, ("u", "v"))],
                         ids=["forces", "advect_moist", "advect_momentum", "advance_uv"])
@pytest.mark.parametrize("counted", [True, False], ids=["status", "no_status"])
def test_waits_that_ran_out_leave_no_plausible_result(op, outputs, counted):
    """A tensor-map kernel whose waits on its tiles ran out: NaN at every point
    that the kernel updates otherwise, the rest untouched, with and without
    the status words that count the blocks; the context stays usable."""
    n, nz = 40, 14
    cg, L = A.scalar_grid((nz, n, n), 1 / 9000.0, 1 / 9000.0), N.lib()
    gen = torch.Generator(device="cuda").manual_seed(op)
    three = set(A.FORCES_INPUTS) | set(A.UV_INPUTS) | {"ru_m", "rv_m", "ww_m", "rw_tend"}
    three -= {"mu", "muu", "muv", "mudf", "mut", "mub"}
    rnd = lambda *s: 1.0 + torch.rand(*s, generator=gen, device="cuda")  # noqa: E731
    st = {k: rnd(nz, n, n) for k in three} | {k: rnd(7, nz, n, n) for k in ("moist", "advect_tend")}
    st |= {k: rnd(n, n) for k in ("mu", "muu", "muv", "mudf", "mut", "mub", *A.FORCES_DATA, *A.UV_DATA)}
    st |= {k: rnd(nz) for k in ("fnm", "fnp", "rdn", "rdnw")}
    status = torch.zeros(16, dtype=torch.int32, device="cuda")

    def run(expired):
        d = {k: v.clone() for k, v in st.items()}
        tab = A._table(d)
        if counted:
            tab[N.field_names().index("status")] = status.data_ptr()
        by, s = ctypes.byref(cg), _stream()
        if expired:
            rc = L.wrf_expired_waits(by, tab, op, s)
        elif op == 0:
            rc = L.wrf_forces(by, tab, 31, s)
        elif op == 1:
            rc = L.wrf_advect_moist(by, *[_p(d[k]) for k in ("moist", "advect_tend", "ru_m", "rv_m", "ww_m", "msftx",
                                                              "fnm", "fnp", "rdnw")], s)
        elif op == 2:
            rc = 0
            for c, (q, t, m) in enumerate((("u", "ru_tend", "msfux"), ("v", "rv_tend", "msfvy"),
                                           ("w", "rw_tend", "msftx"))):
                rc |= L.wrf_advect_momentum(by, c, *[_p(d[k]) for k in (q, t, "ru", "rv", "ww", m, "msfvx", "fnm", "fnp",
                                                                        "rdn" if c == 2 else "rdnw")], 0, s)
        else:
            rc = L.wrf_advance_uv(by, tab, 1.0, s)
        N.check(rc, "operator")
        torch.cuda.synchronize()
        return d

    good, left = run(False), run(True)
    assert int(status[N.WRF_ST_WAIT]) > 0 if counted else int(status.abs().sum()) == 0
    for k in good:
        if k not in outputs:
            assert torch.equal(left[k], st[k]), k
            continue
        assert bool(torch.isfinite(good[k]).all())
        updated = good[k] != st[k]
        assert bool(updated.any()) and bool(left[k][updated].isnan().all()), k
        same = ~left[k].isnan()
        assert torch.equal(left[k][same], st[k][same]), k
    prev = L.wrf_set_kernel_form(N.WRF_FORM_POINT)
    try:
        assert L.wrf_expired_waits(ctypes.byref(cg), A._table(st), op, _stream()) == N.WRF_EINVAL
    finally:
        L.wrf_set_kernel_form(prev)


def _chain_case():
    """A small moist state, its constants and boundary arrays, and the
    scalars of a step."""
    spec = synthetic.CaseSpec(n=28, nz=16, dt=45.0, soundsteps=4, bdy_tend_amp=1.0e-4, seed=11)
    inputs, bdy = synthetic.build(spec)
    g = synthetic.grid_for(spec)
    st = DeviceState.from_inputs(g, inputs, bdy, device="cuda")
    names = dict.fromkeys(A.RK_STATE + ("u_1", "w_1", "ph_1", "mu_1", "t_1", "v_1"))
    state = {k: st[k].clone() for k in names}
    data = {k: st[k].clone() for k in dict.fromkeys(A.STEP_DATA + ("alb", "pb", "phb", "rdnw"))}
    keys = (("bxs", "xs"), ("bxe", "xe"), ("bys", "ys"), ("bye", "ye"), ("btxs", "txs"), ("btxe", "txe"), ("btys", "tys"),
            ("btye", "tye"))
    bd = {f: {key: st[f"{f}_{n}"].clone() for n, key in keys} for f in ("u", "v", "ph", "t", "mu", "qv")}
    sc = dict(epssm=g.epssm, emdiv=g.emdiv, smdiv=g.smdiv, rdx=g.rdx, rdy=g.rdy, **st.scal)
    return g, state, data, bd, sc


def _first_stage(state, data, bd, sc):
    bt = {"u": bd["u"], "v": bd["v"], "h": bd["ph"], "t": bd["t"], "m": bd["mu"], "q": bd["qv"]}
    return A.rk_stage(state, data, bt, 1, 1, 15.0, 15.0, dtbc=45.0, **sc)


@pytest.mark.parametrize("name", ["msftx", "msfty", "msfux", "msfuy", "msfvx", "msfvx_inv", "msfvy", "fnm", "rdn", "rdnw",
                                  "dnw", "t_init"])
def test_a_constant_changed_before_the_reverse_is_refused(name):
    """The reverse of an RK stage reads its constant arrays again: one changed
    in place since the forward raises, as a changed state field does."""
    _, state, data, bd, sc = _chain_case()
    state["t"].requires_grad_(True)
    out = _first_stage(state, data, bd, sc)
    data[name].mul_(1.01)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        (out["t"].sum() + out["moist"].sum()).backward()


def test_all_that_a_stage_reverses_with_passes_the_saved_tensor_hooks():
    """Saved-tensor hooks that copy: with every array of the caller overwritten
    after the forward, the copies alone give the same gradients (sums by
    atomics in some order: 1e-5 of the norm)."""
    grads = []
    for hooked in (False, True):
        _, state, data, bd, sc = _chain_case()
        leaves = [state[k].requires_grad_(True) for k in ("u", "t", "ph", "mu", "moist")]
        if hooked:
            with torch.autograd.graph.saved_tensors_hooks(lambda v: v.detach().clone(), lambda v: v):
                out = _first_stage(state, data, bd, sc)
            with torch.no_grad():
                for v in [*state.values(), *data.values(), *[b for d in bd.values() for b in d.values()]]:
                    v.fill_(float("nan"))
        else:
            out = _first_stage(state, data, bd, sc)
        grads.append(torch.autograd.grad([out[k] for k in ("u", "w", "t", "p", "moist")], leaves,
                                         grad_outputs=[torch.ones_like(out[k]) for k in ("u", "w", "t", "p", "moist")]))
    for a, b in zip(*grads):
        assert float(a.norm()) > 0.0 and float((a - b).norm()) <= 1e-5 * float(a.norm())


def test_a_checkpointed_rollout_holds_one_state_per_step():
    """What the forward of a checkpointed rollout leaves allocated: the states
    at the segments' starts, and no operator's scratch or intermediates (one
    percent of a state per step for the small arrays of the step's end)."""
    g, state, data, bd, sc = _chain_case()
    names = tuple(state)

    def one(*xs):
        out = A.step(dict(zip(names, xs)), data, bd, 45.0, dt=45.0, soundsteps=4,
                     microphysics=lambda q: A.microphysics(q, data, 45.0, g.rdx, g.rdy), **sc)
        return tuple(out[k] for k in names)

    def held(n):
        xs = tuple(state[k].clone().requires_grad_(k == "t") for k in names)
        before = torch.cuda.memory_allocated()
        out = A.rollout(one, xs, n)
        torch.cuda.synchronize()
        return torch.cuda.memory_allocated() - before, out

    held(1)
    size = sum(v.numel() * 4 for v in state.values())
    first, last = held(1)[0], held(4)[0]
    assert last - first <= 3 * 1.01 * size + 4096 * len(names), (first / size, last / size)


def test_arrays_with_gaps_where_only_their_slots_or_shapes_are_used():
    """Species that lie together slot by slot in a larger array (step_end's
    moist, the first stage's moist_tend) and tendencies whose shape alone is
    read: the same values as from packed arrays; where an operator reads the
    whole array, or a slot has gaps of its own, it is refused."""
    g, state, data, bd, sc = _chain_case()
    bt = {"u": bd["u"], "v": bd["v"], "h": bd["ph"], "t": bd["t"], "m": bd["mu"], "q": bd["qv"]}

    def slots(v):
        big = torch.full((2 * v.shape[0],) + tuple(v.shape[1:]), 7.0, device="cuda")
        big[::2] = v
        return big[::2]

    def inner(v):
        return torch.full(tuple(v.shape[:-1]) + (2 * v.shape[-1],), 7.0, device="cuda")[..., :v.shape[-1]].copy_(v)

    def end(s):
        return A.step_end(s, data, bd, 45.0, cf1=sc["cf1"], cf2=sc["cf2"], cf3=sc["cf3"], rdx=g.rdx, rdy=g.rdy)

    def moist(s, rk=1):
        return A.moist_stage(s, data, rk, 15.0, g.rdx, g.rdy, bt, 45.0)

    def dynamics(s):
        return A.dynamics_stage(s, data, bt, 2, 2, 9.0, **sc)

    for run, name, gaps in ((end, "moist", slots), (moist, "moist_tend", slots), (dynamics, "ru_tend", inner)):
        want, got = run(state), run({**state, name: gaps(state[name])})
        for k in want:
            assert torch.equal(want[k].view(torch.int32), got[k].contiguous().view(torch.int32)), (name, k)
    for run, name, gaps in ((end, "moist", inner), (moist, "moist_tend", inner), (moist, "moist", slots),
                            (lambda s: moist(s, 2), "moist_tend", slots), (dynamics, "u", inner)):
        with pytest.raises(TypeError):
            run({**state, name: gaps(state[name])})


@pytest.mark.parametrize("name", ["advance_mu_t", "coef_w_adj"])
def test_column_tiles_on_more_rows_than_a_grid_dimension(name):
    """70000 rows (a grid's second dimension takes 65535): the last inner rows
    against the same rows as a domain of their own, bitwise (nothing sums over
    rows)."""
    nz, nx, rows, crop = 12, 24, 70000, 64
    gen = torch.Generator(device="cuda").manual_seed(7)
    fld = {True: {}, False: {}}

    def field(k, two_d):
        if k not in fld[two_d]:
            fld[two_d][k] = 1.0 + 0.1 * torch.rand(*((rows, nx) if two_d else (nz, rows, nx)), generator=gen, device="cuda")
        return fld[two_d][k]

    prof = {k: torch.linspace(0.9, 1.1, nz, device="cuda") for k in ("fnm", "fnp", "rdn", "rdnw", "dnw")}

    def run(cut):
        def get(k, two_d=False):
            v = field(k, two_d)
            return (v[..., rows - crop:, :] if cut else v).clone()

        ny = crop if cut else rows
        if name == "coef_w_adj":
            cg = A.scalar_grid((nz, ny, nx), 1 / 9000.0, 1 / 9000.0)
            out = [torch.zeros(ny, nx, device="cuda")] + [torch.zeros(nz, ny, nx, device="cuda") for _ in range(2)]
            ops = [get("mut", True), get("cqw"), get("c2a"), prof["rdn"], prof["rdnw"]]
            cots = [get(k) for k in ("ca", "calpha", "cgamma")]
            N.check(N.lib().wrf_coef_w_adj(ctypes.byref(cg), *map(_p, ops), 0.01, *map(_p, cots), *map(_p, out),
                                           _stream()), "coef_w_adj")
        else:
            two = {"mu", "mut", "muave", "muts", "muu", "muv", "mudf", "mu_tend"}
            x = {k: get(k, k in two).requires_grad_(True) for k in A.MUT_INPUTS}
            data = {k: prof[k] if k in prof else get(k, True) for k in A.MUT_DATA}
            res = A.advance_mu_t(x, data, 0.1, 0.1, 1 / 9000.0, 1 / 9000.0)
            out = [v.detach() for v in res.values()]
            out += torch.autograd.grad(list(res.values()), list(x.values()),
                                       grad_outputs=[get("cot_" + k, k in two) for k in res])
        torch.cuda.synchronize()
        return [v[..., ny - 32:ny - 12, :].clone() for v in out]

    for a, b in zip(run(True), run(False)):
        assert float(a.abs().max()) > 0.0 and torch.equal(a, b)


def test_marching_acoustic_columns_from_a_sector_and_deep():
    """Rows of whole sectors, whose blocks start left of the first column, and
    the depth the marching kernel was made for."""
    test_marching_acoustic_columns_equal_the_tiled_form_bitwise(320, 61)


@pytest.mark.parametrize("n,nz,rk", [(64, 17, 1), (140, 41, 1), (140, 41, 2), (130, 38, 1)])
def test_tendency_accumulation_at_both_depths_per_thread(n, nz, rk):
    """The step's fused accumulation, at one level a thread and (from 606208
    points on) at four with a remainder, against the stand-alone accumulation
    and the specified rows on the fields the step had before it, bitwise (its
    divisions are correctly rounded)."""
    spec = synthetic.CaseSpec(n=n, nz=nz, nsteps=1, bdy_tend_amp=1.0e-4, seed=n)
    g = synthetic.grid_for(spec)
    inputs, bdy = synthetic.build(spec)
    st = DeviceState.from_inputs(g, inputs, bdy, device="cuda")
    before, after = {}, {}

    def probe(name):
        if name == ("s1.diff" if rk == 1 else f"s{rk}.forces"):
            before.update({k: st[k].clone() for k in A._Addtend.fields})
        if name == f"s{rk}.tend":
            after.update({k: st[k].clone() for k in A._Addtend.outputs})

    Integrator(st).step(probe)
    torch.cuda.synchronize()
    want = A.addtend(before, {k: st[k] for k in A._Addtend.data}, rk, g.rdx, g.rdy)
    for k, var, f in (("ru_tend", "u", "u"), ("rv_tend", "v", "v"), ("ph_tend", "h", "ph"), ("t_tend", "t", "t"),
                      ("mu_tend", "m", "mu")):
        bt = {key: st[f"{f}_{b}"] for b, key in (("btxs", "txs"), ("btxe", "txe"), ("btys", "tys"), ("btye", "tye"))}
        want[k] = A.spec_bdytend(want[k], bt, var, g.rdx, g.rdy)
    for k in A._Addtend.outputs:
        assert torch.equal(after[k], want[k]), k
    assert float(after["ru_tend"].abs().max()) > 0.0


def test_a_chain_whose_names_share_a_tensor():
    """One tensor under two names of the state: its gradient is the sum of
    those of two equal tensors (sums by atomics in some order: 1e-5 of the
    norm)."""
    pairs = (("u", "u_1"), ("t", "t_1"), ("mu", "mu_1"))
    got = []
    for shared in (True, False):
        _, state, data, bd, sc = _chain_case()
        state["t"] += 0.1 * torch.sin(torch.arange(state["t"].numel(), device="cuda").view_as(state["t"]).float())
        leaves = []
        for a, b in pairs:
            state[a].requires_grad_(True)
            state[b] = state[a] if shared else state[a].detach().clone().requires_grad_(True)
            leaves += [state[a]] if shared else [state[a], state[b]]
        out = _first_stage(state, data, bd, sc)
        names = ("u", "w", "t", "p", "t_1", "mu_1")
        grads = torch.autograd.grad([out[k] for k in names], leaves,
                                    grad_outputs=[torch.cos(torch.arange(out[k].numel(), device="cuda").view_as(out[k])
                                                            .float()) for k in names])
        got.append(grads if shared else [a + b for a, b in zip(grads[::2], grads[1::2])])
    for a, b in zip(*got):
        assert float(a.norm()) > 0.0 and float((a - b).norm()) <= 1e-5 * float(a.norm())
