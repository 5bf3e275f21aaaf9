"""The FP64 column walk's cheaper square root and exponential where rounding shows
most: rock salt near its lattice, whose forces are a thousandth of the pair
terms that they are sums of, with an exponential of r.  Its error against
extended precision is to be no larger than that of the cell-by-cell kernel with
correctly rounded operations (MDGPU_PAIRS_COLUMNS=0, read once per process: a
process of its own); 10 % leaves room for another order of the sums."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RUN = """
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from moldy_gb300 import ForceField, system
s = system.rock_salt(ncell=6, seed=int(sys.argv[2]))
s.control.strict_cutoff = True
ff = ForceField(s, precision="fp64")
np.save(sys.argv[3], ff.force_calc()[0])
ff.close()
"""


def extended(s):
    """Forces of the pairs within the cut-off (strict: others are taken at 100 times it)."""
    L = np.longdouble
    x, q, ids = np.asarray(s.site).astype(L), s.chg().astype(L), s.site_ids()
    box, rc, a = L(np.asarray(s.h)[0, 0]), L(s.control.cutoff), L(s.control.alpha)
    pot = np.asarray(s.potpar).reshape(s.max_id, s.max_id, 8).astype(L)
    f = np.zeros_like(x)
    for i in range(s.nsites):
        r = x - x[:, i:i + 1]
        r -= box * np.rint(r / box)
        r2 = (r * r).sum(0)
        near = (r2 <= rc * rc) & (np.arange(s.nsites) != i)
        r, r2, p, qq = r[:, near], r2[near], pot[ids[i], ids[near]], q[i] * q[near]
        d = np.sqrt(r2)
        t = 1 / (1 + L("0.3275911") * a * d)
        poly = L("-1.453152027") + t * L("1.061405429")
        poly = t * (L("0.254829592") + t * (L("-0.284496736") + t * (L("1.421413741") + t * poly)))
        g = np.exp(-a * a * r2) * qq
        e = poly * g / d + 2 / np.sqrt(L("3.14159265358979323846264338")) * a * g
        fr = -6 * p[:, 0] / r2 ** 4 + p[:, 1] * p[:, 2] * np.exp(-p[:, 2] * d) / d + e / r2
        f[:, i] = -(fr * r).sum(1)
    return f


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_rock_salt_forces(seed, tmp_path):
    from moldy_gb300 import system
    if np.finfo(np.longdouble).nmant < 60:
        pytest.skip("no extended precision")
    s = system.rock_salt(ncell=6, seed=seed)
    want, err = extended(s), {}
    for columns in "01":
        out = str(tmp_path / (columns + ".npy"))
        subprocess.run([sys.executable, "-c", RUN, ROOT, str(seed), out], check=True,
                       env={**os.environ, "MDGPU_PAIRS_COLUMNS": columns})
        err[columns] = np.sqrt(((np.load(out) - want) ** 2).sum() / (want ** 2).sum())
    assert err["1"] <= 1.1 * err["0"], err
