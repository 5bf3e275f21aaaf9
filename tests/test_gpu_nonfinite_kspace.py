"""Values that are not finite in the fixed-point digits of the reciprocal space:
they hold none, and the result has to be NaN where the sums over them are, not
a saturated number."""
import dataclasses

import numpy as np
import pytest

from test_gpu_quads import ions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("species", [1, 2])
def test_charge_not_finite(form, value, species):
    from moldy_gb300 import ForceField
    s = ions(200, (9, 9, 9), 4.0)
    q = np.array(s.site_charge)
    q[species] = value
    s = dataclasses.replace(s, site_charge=q)
    ff = ForceField(s, precision=form)
    f, pe, _ = ff.ewald()
    ff.close()
    assert np.isnan(f).all()
    assert not np.isfinite(pe)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_residual_not_finite(form, value):
    from moldy_gb300 import ForceField
    s = ions(200, (9, 9, 9), 4.0)
    ff = ForceField(s, precision=form)
    fref = np.zeros((3, s.nsites))
    fref[1, 17] = value
    loss, g = ff.fm_loss_grad(fref, 0.3)
    ff.close()
    assert not np.isfinite(loss)
    assert np.isnan(g["chg"]).all() and np.isnan(g["alpha"])


@pytest.mark.parametrize("size", [1e120, 1e60, 1.0, 1e-60, 1e-200])
def test_residual_sizes(size, monkeypatch):
    """FP64 weights over the exponent's range, against the CUDA-core passes (as
    test_gpu_quads: 1e-9 of the largest entry); with 1e120 and 1e60 from one
    site's reference force, with the others from the loss's weight."""
    from moldy_gb300 import ForceField
    s = ions(200, (9, 9, 9), 4.0)
    fref = np.zeros((3, s.nsites))
    if size > 1:
        fref[2, 5] = size
    res = []
    for tc in ("0", "1"):
        monkeypatch.setenv("MDGPU_KSPACE_TC", tc)
        ff = ForceField(s, precision="fp64")
        res.append(ff.fm_loss_grad(fref, min(size, 1.0))[1])
        ff.close()
    g0, g = res
    assert np.isfinite(g0["chg"]).all() and np.abs(g0["chg"]).max() > 0
    assert np.abs(g["chg"] - g0["chg"]).max() <= 1e-9 * np.abs(g0["chg"]).max()
    assert abs(g["alpha"] - g0["alpha"]) <= 1e-9 * (abs(g0["alpha"]) + np.abs(g0["chg"]).max())
