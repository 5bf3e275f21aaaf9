"""Calls refused for a missing argument take no copy of the caller's arrays (or
of the staging buffer) before they look: with molecular cut-offs, force_calc
without centres of mass and ewald before any force_calc.  The next call, with
other arrays in other memory and more sites, has its own result: that of a
fresh context, the same launches (1e-12 leaves room for rounding)."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pointers(a):
    return (C.POINTER(C.c_double) * 3)(*[a[k].ctypes.data_as(C.POINTER(C.c_double)) for k in range(3)])


@pytest.mark.parametrize("nside", [5, 36])   # staged, and straight from the caller's arrays
def test_refused_call_then_another(nside):
    from moldy_gb300 import ForceField, system
    from moldy_gb300.forcefield import _dp
    small, s = (system.water(nside=n, seed=3) for n in (4, nside))
    small, s = (dataclasses.replace(x, control=dataclasses.replace(x.control, molpbc=True)) for x in (small, s))
    ff = ForceField(small, precision="mixed")
    h = np.ascontiguousarray(small.h, float).reshape(9)
    out = np.zeros(1), np.zeros(9)
    for call in ("mdgpu_ewald", "mdgpu_force_calc"):
        x, f = np.full((3, small.nsites), 1e9), np.full((3, small.nsites), 7.0)
        args = [_dp(h), pointers(x), pointers(f)] + ([None] if call == "mdgpu_force_calc" else [])
        assert getattr(ff.L, call)(ff.ctx, *args, _dp(out[0]), _dp(out[1])) == 1      # MDGPU_E_ARG
        assert b"centres of mass" in ff.L.mdgpu_last_error(ff.ctx)
        assert (f == 7.0).all() and out[0][0] == 0.0
        del x, f
    ff.set_system(s)
    got = ff.force_calc()
    ff.close()
    fresh = ForceField(s, precision="mixed")
    want = fresh.force_calc()
    fresh.close()
    assert np.abs(got[0] - want[0]).max() <= 1e-12 * np.abs(want[0]).max()
    assert abs(got[1] - want[1]) <= 1e-12 * abs(want[1])
