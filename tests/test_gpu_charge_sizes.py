"""Charges of very different size in the reciprocal space: a few large ones among
many small, on both sides of the ratio (largest to root mean square, 16) from
which the digits on the grid of the largest do not serve.  Forces on the large
and on the small ions apart.

FP64: against the CUDA-core passes; beyond the ratio it is those, so the same
to rounding (1e-15 of the group's RMS force), and below it the 1e-12 of the
other comparisons.  Mixed: against the FP64 result, with the error that the form
had with its former operands (24 bits of every charge) as the bound: measured
2.8e-6 and 1.8e-6, 1.7e-6 and 1.4e-6, 2.7e-6 and 2.5e-6, 4.8e-5 and 2.8e-6,
5.0e-3 and 4.0e-6 of the RMS force on the large and the small ions."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ions(n, nbig, ratio, seed=7):
    from moldy_gb300 import system as S
    rng = np.random.default_rng(seed)
    L = 20.0
    x = rng.uniform(-0.499, 0.499, (3, n)) * L
    sp = [S.Species("A", nbig, np.array([1], np.int32), np.zeros((1, 3))),
          S.Species("B", n - nbig, np.array([2], np.int32), np.zeros((1, 3)))]
    q = np.array([0.0, 1.0, -1.0 / ratio]) / S.CONV_Q
    return S.System(h=np.diag([L] * 3), species=sp, ptype=S.LJPOT, potpar=np.zeros((9, 8)), site_charge=q, site=x,
                    c_of_m=(x / L).T, control=S.Control(cutoff=3.0, alpha=0.45, k_cutoff=2.0))


CASES = [(1000, 10, 100, 1e-12, 2.8e-6, 1.8e-6), (1000, 1, 10, 1e-12, 1.7e-6, 1.4e-6),
         (4000, 4, 30, 1e-15, 2.7e-6, 2.5e-6), (1000, 1, 1000, 1e-15, 4.8e-5, 2.8e-6),
         (4000, 1, 1e5, 1e-15, 5.0e-3, 4.0e-6)]


@pytest.mark.parametrize("n,nbig,ratio,tol64,tolbig,tolsmall", CASES)
def test_forces_on_large_and_small_charges(n, nbig, ratio, tol64, tolbig, tolsmall, monkeypatch):
    from moldy_gb300 import ForceField
    s = ions(n, nbig, ratio)
    res = {}
    for form, tc in (("fp64", "0"), ("fp64", "1"), ("mixed", "1")):
        monkeypatch.setenv("MDGPU_KSPACE_TC", tc)
        ff = ForceField(s, precision=form)
        res[form, tc] = ff.ewald() + (ff.energy_grad()[1]["chg"],)
        ff.close()
    f0, e0, s0, g0 = res["fp64", "0"]

    def err(f, part):
        return np.sqrt(((f - f0)[:, part] ** 2).mean()) / np.sqrt((f0[:, part] ** 2).mean())
    big, small = slice(0, nbig), slice(nbig, n)
    for form, tb, ts, te in (("fp64", tol64, tol64, 1e-12), ("mixed", tolbig, tolsmall, 1e-5)):
        f, e, st, g = res[form, "1"]
        assert err(f, big) <= tb and err(f, small) <= ts, form
        assert abs(e - e0) <= te * abs(e0) and np.abs(st - s0).max() <= te * np.abs(s0).max(), form
        assert np.abs(g - g0).max() <= 2 * te * np.abs(g0).max(), form


def test_large_system_runs_its_pairs_with_either_passes(monkeypatch):
    """From some thousand sites on, the pair kernel waits for the tensor-core
    passes' tables; with the CUDA-core ones it must not.  Whole forces of one
    large charge among 8000."""
    from moldy_gb300 import ForceField
    s = dataclasses.replace(ions(8000, 1, 1000), site_charge=ions(8000, 1, 1000).site_charge * 0.01)
    res = []
    for tc in ("0", "1"):
        monkeypatch.setenv("MDGPU_KSPACE_TC", tc)
        ff = ForceField(s, precision="fp64")
        res.append(ff.forces())
        ff.close()
    for a, b in zip(*res):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()
