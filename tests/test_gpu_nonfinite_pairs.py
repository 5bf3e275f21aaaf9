"""Pairs at no distance and coordinates that are not numbers, FP64 form: the
column walk's cheaper square root and its comparisons by bits give what the
oracle's arithmetic gives.  Two like charges at one place have an infinite
energy and no defined force; without charges the exponential potential of
the MCY form has a finite one.  A site whose coordinate is NaN makes the energy
NaN, with the strict cut-off too (a NaN distance is not beyond it), and the
call reports it as out of range.  Finite values: the 1e-12 of the other
comparisons with the oracle."""
import dataclasses
import os

import numpy as np
import pytest

from test_gpu_pairs import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("charged", [True, False])
def test_coincident_sites(port_built, charged):
    from moldy_gb300 import ForceField
    from oracle import port
    s = build(2, 343, charged, ())
    x = np.array(s.site)
    x[:, 1] = x[:, 0]
    s = dataclasses.replace(s, site=x, c_of_m=(np.linalg.inv(np.asarray(s.h, float)) @ x).T)
    with np.errstate(all="ignore"):
        r = port.force_calc(s, nthreads=os.cpu_count() or 1)
    ff = ForceField(s, precision="fp64")
    f, pe, _ = ff.force_calc()
    close = ff.info()["too_close"]
    ff.close()
    assert (0, 1) in close
    assert np.array_equal(np.isnan(f), np.isnan(r.force)) and np.isnan(f[:, :2]).all()
    fine = ~np.isnan(f)
    assert np.sqrt(((f - r.force)[fine] ** 2).mean()) <= 1e-12 * np.sqrt((r.force[fine] ** 2).mean())
    if charged:
        assert np.isposinf(r.pe) and np.isposinf(pe)
    else:
        assert np.isfinite(r.pe) and abs(pe - r.pe) <= 1e-12 * abs(r.pe)


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("strict", [True, False])
def test_coordinate_not_a_number(strict, sign):
    import torch
    from moldy_gb300 import ForceField
    from moldy_gb300._lib import MdgpuError
    s = build(0, 343, True, ())
    s = dataclasses.replace(s, control=dataclasses.replace(s.control, strict_cutoff=strict))
    ff = ForceField(s, precision="fp64")
    x = np.ascontiguousarray(s.site)
    x[1, 7] = np.copysign(np.nan, sign)
    stream = torch.cuda.Stream()
    ff.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        d = torch.from_numpy(x).cuda()
        f = torch.zeros_like(d)
        e = torch.zeros(11, dtype=torch.float64, device="cuda")
        stream.synchronize()
        ff.forces_device(d.data_ptr(), f.data_ptr(), e.data_ptr(), e.data_ptr() + 16)
    with pytest.raises(MdgpuError):
        ff.synchronize()
    assert np.isnan(float(e[0])) and np.isnan(f[:, 7].cpu().numpy()).all()
    assert ff.info()["n_too_close"] == 0
    ff.close()
