"""Sizes that an entry point refuses before it touches the device."""
from __future__ import annotations

import ctypes

import pytest

from pywrf_b200 import _native as N
from pywrf_b200.config import Grid
from pywrf_b200.state import make_cgrid


def _cgrid(n, nz=64):
    return make_cgrid(Grid.make(n, n, nz, 9000.0, 9000.0, 45.0),
                      {"cf1": 1.0, "cf2": 0.0, "cf3": 0.0, "cfn": 1.0, "cfn1": 0.0})


@pytest.mark.parametrize("n,refused", [(5900, True), (5700, False)])
def test_entries_with_32_bit_offsets_refuse_larger_fields(n, refused):
    """The step, its phases and the eddy viscosities on either side of 2^31
    points, on a table without fields (which the smaller size is refused for);
    an operator with 64-bit offsets takes both."""
    L, by = N.lib(), ctypes.byref
    assert (64 * n * n >= 2 ** 31) == refused
    cg, tab = _cgrid(n), (ctypes.c_void_p * N.lib().wrf_field_count())()
    tab = ctypes.cast(tab, ctypes.c_void_p)
    for name, args in (("wrf_rk3_step", (None, N.PROBE_FN(), None)), ("wrf_rk_prep", (1, None)),
                       ("wrf_acoustic_substep", (3, 1, None)), ("wrf_eddy_viscosity", (None,)),
                       ("wrf_eddy_viscosity_adj", (tab, tab, None))):
        assert getattr(L, name)(by(cg), tab, *args) == N.WRF_EINVAL, name
        assert ("2^31" in L.wrf_last_error().decode()) == refused, (name, L.wrf_last_error())
    words = ctypes.c_size_t(0)
    assert L.wrf_advect_scalar_adj_work(by(cg), by(words)) == 0 and words.value == 6 * 64 * n * n
