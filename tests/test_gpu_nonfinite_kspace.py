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
