"""Stand-alone operators on fields of more than 2^31 points: a level's offset
does not fit 32 bits there."""
from __future__ import annotations

import ctypes
import math

import pytest
import torch

from pywrf_b200 import _native as N
from pywrf_b200 import adjoint as A

pytestmark = pytest.mark.gpu

NZ, TILE = 64, 100
SMALL, LARGE = 3 * TILE, 59 * TILE  # levels 62 and 63 of the large domain start past 2^31 points
RD = 1.0 / 9000.0


class Domain:
    """Periodic copies of one tile of columns, so that a point away from the
    sides has the same value in every domain."""

    def __init__(self, n):
        self.n, self.cg = n, A.scalar_grid((NZ, n, n), RD, RD)
        self.cg.smdiv, self.cg.emdiv, self.cg.cf1, self.cg.cf2, self.cg.cf3 = 0.1, 0.01, 2.0, -1.5, 0.5

    def field(self, seed, two_d=False):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        nz, t = 1 if two_d else NZ, TILE
        tile = 1.0 + 0.1 * torch.rand(nz, t, t, generator=gen, device="cuda")
        out = torch.empty(nz, self.n // t, t, self.n // t, t, device="cuda")
        out.copy_(tile[:, None, :, None, :].expand_as(out))
        return out.view((self.n, self.n) if two_d else (nz, self.n, self.n))

    def zeros(self, two_d=False):
        return torch.zeros((self.n, self.n) if two_d else (NZ, self.n, self.n), device="cuda")

    def tile(self, a):
        """The last tile that no side reaches."""
        o = self.n - 2 * TILE
        return a[..., o:o + TILE, o:o + TILE].clone()

    def call(self, name, *args):
        """A library call; a dict becomes a state table, and lives through the call."""
        vals = [A._ptr(a) if isinstance(a, torch.Tensor) else A._table(a) if isinstance(a, dict) else a for a in args]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        N.check(getattr(N.lib(), name)(ctypes.byref(self.cg), *vals, stream), name)
        torch.cuda.synchronize()


def profiles():
    return {k: torch.linspace(0.9, 1.1, NZ, device="cuda") for k in ("fnm", "fnp", "rdn", "rdnw", "dn", "dnw")}


def maps(d):
    return {k: d.field(100 + q, True) for q, k in enumerate(("msfux", "msfuy", "msfvx", "msfvx_inv", "msfvy", "msftx",
                                                            "msfty"))}


def coef_w(d):
    p, mut, x = profiles(), d.field(1, True), d.field(2)
    out = [d.zeros() for _ in range(3)]
    d.call("wrf_coef_w", mut, x, x, p["rdn"], p["rdnw"], 0.01, *out)
    return out


def coef_w_adj(d):
    p, mut, x, c = profiles(), d.field(1, True), d.field(2), d.field(3)
    out = [d.zeros(True), d.zeros(), d.zeros()]
    d.call("wrf_coef_w_adj", mut, x, x, p["rdn"], p["rdnw"], 0.01, c, c, c, *out)
    return out


def diffusion(d):
    tab, x, out = maps(d), d.field(2), d.zeros()
    d.call("wrf_horizontal_diffusion", tab, b"m", x, None, d.field(1, True), x, out)
    return [out]


def diffusion_adj(d):
    tab, x, c, out = maps(d), d.field(2), d.field(3), [d.zeros(), d.zeros(True), d.zeros()]
    d.call("wrf_horizontal_diffusion_adj", tab, b"w", x, None, d.field(1, True), x, c, *out)
    return out


def operands(d, three_d, two_d, own):
    """A table whose read-only 3-D operands share one array; ``own`` are the
    operator's to write."""
    x = d.field(4)
    named = {k: x for k in three_d} | {k: d.field(20 + q, True) for q, k in enumerate(two_d)}
    return named | {k: (d.field(50 + q, True) if k in two_d else d.field(50 + q)) for q, k in enumerate(own)}


UV3 = [k for k in A.UV_INPUTS if k not in ("mu", "muu", "muv", "mudf")]


def advance_uv(d):
    prev = N.lib().wrf_set_kernel_form(N.WRF_FORM_POINT)  # the form of rows that are not whole 16-byte words
    try:
        t = operands(d, UV3, ("mu", "muu", "muv", "mudf"), ("u", "v"))
        d.call("wrf_advance_uv", t | maps(d) | profiles(), 9.0)
    finally:
        N.lib().wrf_set_kernel_form(prev)
    return [t["u"], t["v"]]


MUT2 = ("mu", "mut", "muave", "muts", "muu", "muv", "mudf", "mu_tend")
MUT3 = [A._MUT_FIELD.get(k, k) for k in A.MUT_INPUTS if k not in MUT2]


def advance_mu_t(d):
    own = ("ww", "t", "t_2save", "muave", "muts", "mudf", "mu")
    t = operands(d, MUT3, MUT2, own)
    d.call("wrf_advance_mu_t", t | maps(d) | profiles(), 0.1)
    return [t[k] for k in own]


def advance_mu_t_adj(d):
    t = operands(d, MUT3, MUT2, ())
    bars = {k: d.field(70 + q) for q, k in enumerate(MUT3)} | {k: d.field(90 + q, True) for q, k in enumerate(MUT2)}
    d.call("wrf_advance_mu_t_adj", t | maps(d) | profiles(), bars, 0.1, 0, d.zeros())
    return list(bars.values())


PR3 = [A._PRHO_FIELD.get(k, k) for k in A.PRHO_INPUTS if k not in ("mu", "mut")]


def calc_p_rho_adj(d):
    t = operands(d, PR3, ("mu", "muts"), ()) | profiles()
    bars = {k: d.field(70 + q) for q, k in enumerate(PR3)} | {k: d.field(90 + q, True) for q, k in enumerate(("mu", "muts"))}
    d.call("wrf_calc_p_rho_adj", t, bars, 1)
    return list(bars.values())


@pytest.mark.parametrize("op,arrays", [(coef_w, 4), (coef_w_adj, 4), (diffusion, 2), (diffusion_adj, 4), (advance_uv, 3),
                                       (advance_mu_t, 4), (advance_mu_t_adj, 12), (calc_p_rho_adj, 9)],
                         ids=lambda v: getattr(v, "__name__", ""))
def test_operator_past_32_bit_offsets(op, arrays):
    """The last inner tile against the middle one of three: the same operations
    but for sums by atomics in some order, of at most 200 float32 terms whose
    partial sums stay below ten times the level's largest total (half an ulp
    each: 200 * 6e-8 * 10, below 2e-4 of that total)."""
    need = 4 * NZ * LARGE ** 2 * arrays + (4 << 30)
    if torch.cuda.mem_get_info()[0] < need:
        pytest.skip(f"{math.ceil(need / 1e9)} GB of free device memory needed")
    assert NZ * LARGE ** 2 > 2 ** 31 and 62 * LARGE ** 2 > 2 ** 31
    got = []
    for n in (SMALL, LARGE):
        d = Domain(n)
        got.append([d.tile(a) for a in op(d)])
        torch.cuda.empty_cache()
    for a, b in zip(*got):
        assert bool(torch.isfinite(a).all())
        assert bool(((a - b).abs() <= 2e-4 * a.abs().amax((-2, -1), keepdim=True)).all())
