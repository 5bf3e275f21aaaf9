"""Link-cell grids beyond what the column walk's packed words hold (cell indices
of 26 bits and more, z indices of 16): the cell-by-cell kernels serve them.
The mixed form against the FP64 form: 1e-5 of the RMS force, 2e-5 of the largest
gradient entry, the bounds of its other comparisons."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ions(h, subcell, cutoff, alpha, n=500, seed=3):
    from moldy_gb300 import system as S
    rng = np.random.default_rng(seed)
    h = np.asarray(h, float)
    g = [max(2, int(v)) for v in h * (n / h.prod()) ** (1 / 3) + 1]
    cells = np.stack(np.meshgrid(*[(np.arange(v) + 0.5) / v - 0.5 for v in g], indexing="ij"), -1).reshape(-1, 3)
    cells = cells[rng.permutation(len(cells))[:n]]
    x = (cells + rng.uniform(-0.02, 0.02, cells.shape) / g).T * h[:, None]
    n = x.shape[1]
    sp = [S.Species("A", n // 2, np.array([1], np.int32), np.zeros((1, 3))),
          S.Species("B", n - n // 2, np.array([2], np.int32), np.zeros((1, 3)))]
    p = np.zeros((3, 3, 8))
    p[1:, 1:, 0], p[1:, 1:, 1] = 300.0, 2.4
    q = np.array([0.0, 1.0, -1.0]) / S.CONV_Q
    ctl = S.Control(cutoff=cutoff, alpha=alpha, k_cutoff=2.0, subcell=subcell, strict_cutoff=False)
    return S.System(h=np.diag(h), species=sp, ptype=S.LJPOT, potpar=p.reshape(9, 8), site_charge=q, site=x,
                    c_of_m=(x / h[:, None]).T, control=ctl)


@pytest.mark.parametrize("case", [dict(h=(30, 30, 30), subcell=30 / 410, cutoff=4.5, alpha=0.5),
                                  dict(h=(8, 8, 13200), subcell=0.4, cutoff=7.0, alpha=0.0)],
                         ids=["cells", "z"])
def test_mixed_matches_fp64(case):
    from moldy_gb300 import ForceField
    s = ions(**case)
    res = {}
    for form in ("fp64", "mixed"):
        ff = ForceField(s, precision=form)
        f, pe, _ = ff.forces()
        info = ff.info()
        g = ff.fm_loss_grad(np.zeros((3, s.nsites)))[1]
        ff.close()
        res[form] = f, pe, g, info["npairs"]
    assert info["nx"] * info["ny"] * info["nz"] > 1 << 26 or info["nz"] > 1 << 15
    (f0, e0, g0, n0), (f, e, g, n) = res["fp64"], res["mixed"]
    assert n0 == n > 0
    assert np.sqrt(((f - f0) ** 2).mean()) <= 1e-5 * np.sqrt((f0 ** 2).mean())
    for k in ("potpar", "chg"):
        assert np.abs(g[k] - g0[k]).max() <= 2e-5 * np.abs(g0[k]).max()
