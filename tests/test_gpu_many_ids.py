"""Potential tables that fill a block's 48 KB of shared memory next to what
the pair kernels hold themselves: the numbers of site identifiers around which
a launch needs the larger limit, by columns and cell by cell (molecular
cut-off).  Two species of the same ions with identifiers 1 and M - 1; the
result is that of the smallest table, the same arithmetic, so 1e-12 (FP64) and
1e-6 (mixed) of the largest force only leave room for rounding."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ions(M, molpbc):
    from moldy_gb300 import system as S
    s = S.generic_ions(S.HIWPOT, n=343, L=22.0)
    small = np.asarray(s.potpar).reshape(3, 3, 8)
    p = np.zeros((M, M, 8))
    q = np.zeros(M)
    at = {1: 1, 2: M - 1}
    for a in (1, 2):
        q[at[a]] = s.site_charge[a]
        for b in (1, 2):
            p[at[a], at[b]] = small[a, b]
    sp = [dataclasses.replace(x, site_id=np.array([at[int(x.site_id[0])]], np.int32)) for x in s.species]
    return dataclasses.replace(s, species=sp, potpar=p.reshape(M * M, 8), site_charge=q,
                               control=dataclasses.replace(s.control, molpbc=molpbc))


@pytest.mark.parametrize("molpbc", [False, True])
@pytest.mark.parametrize("form,M", [("mixed", m) for m in (23, 30, 31, 32, 36, 37, 38, 39, 40, 54, 55)] +
                         [("fp64", m) for m in (16, 17, 25, 26, 27, 28, 39, 40)])
def test_number_of_identifiers(form, M, molpbc):
    from moldy_gb300 import ForceField
    res = []
    for m in (3, M):
        ff = ForceField(ions(m, molpbc), precision=form)
        f, pe, _ = ff.force_calc()
        ff.close()
        res.append((f, pe))
    tol = 1e-12 if form == "fp64" else 1e-6
    (f0, e0), (f, e) = res
    assert np.abs(f - f0).max() <= tol * np.abs(f0).max()
    assert abs(e - e0) <= tol * abs(e0)
