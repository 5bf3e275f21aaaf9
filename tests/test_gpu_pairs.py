"""The column-walk pair kernels where their branches can go wrong: every
potential form with a pair whose parameters are all zero (the FP64 kernel
leaves that part out), with and without charges, one and two interaction
classes, and site counts on both sides of the sort's one-block limits.

Tolerances: the bounds of the other comparisons with the FP64 oracle, 1e-12
(FP64) and 1e-5 (mixed) of the RMS force and of the energy."""
import dataclasses
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PARS = {0: [400.0, 2.3], 1: [9.0e3, 3.0e6, 3.4], 2: [4.0e5, 3.1, 8.0e3, 1.9],
        3: [5.0e4, 3.2, 1.0e3, 10.0, 20.0, 30.0], 4: [-50.0, -300.0, 4.0e5],
        6: [20.0, 3.0, 3.5, 300.0, 5.0, 1.8, 2.6]}
CASES = [(pt, 343, True, (1, 2)) for pt in PARS] + [(0, 343, False, (1, 2)), (0, 343, True, (1, 1, 2, 2)),
         (0, 1728, True, (1, 2)), (0, 2197, True, (2, 2)), (1, 4913, False, (1, 2))]


def build(ptype, n, charged, zero):
    """Ions on a jittered lattice; the pairs of species listed two by two in
    `zero` interact by their charges alone."""
    from moldy_gb300 import system as S
    s = S.generic_ions(S.GENPOT, n=n, L=3.4 * round(n ** (1 / 3)))
    p = np.zeros((3, 3, 8))
    for a, b in ((1, 1), (1, 2), (2, 2)):
        p[a, b, :len(PARS[ptype])] = p[b, a, :len(PARS[ptype])] = np.array(PARS[ptype]) * (1 + 0.01 * (a + b))
    for a, b in zip(zero[::2], zero[1::2]):
        p[a, b] = p[b, a] = 0.0
    ctl = s.control if charged else dataclasses.replace(s.control, alpha=0.0)
    return dataclasses.replace(s, ptype=ptype, potpar=p.reshape(9, 8), control=ctl)


@pytest.mark.parametrize("ptype,n,charged,zero", CASES)
def test_pairs_against_the_oracle(port_built, ptype, n, charged, zero):
    from moldy_gb300 import ForceField
    from oracle import port
    s = build(ptype, n, charged, zero)
    r = port.force_calc(s, nthreads=os.cpu_count() or 1)
    for form, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
        ff = ForceField(s, precision=form)
        f, pe, _ = ff.force_calc()
        ff.close()
        assert np.sqrt(((f - r.force) ** 2).mean()) <= tol * np.sqrt((r.force ** 2).mean()), form
        assert abs(pe - r.pe) <= tol * abs(r.pe), form
