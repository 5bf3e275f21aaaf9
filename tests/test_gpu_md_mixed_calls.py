"""Dynamics on a context that other calls use as well.  A run replays a
captured step; a gradient (over all sites instead of the charged ones) or an
evaluation in another cell in between moves buffers and makes other work
ranges, and the trajectory has to be that of the same run alone.  Sizes:
charged and all site tiles give the FP64 force pass 2 and 1 runs (10), the
mixed one twice as many work ranges as tiles and as many (14).

Tolerance: every sum is taken in a fixed order, so the two runs agree to the
last bit where nothing differs; 1e-11 (FP64) and 1e-6 (mixed) of the largest
element, a few rounding errors of each form's forces, leaves room for another
split of a sum."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def start(n, form):
    from moldy_gb300 import ForceField, system
    from moldy_gb300.dynamics import MolecularDynamics, species_dynamics, thermal_state
    sysm = system.water(nside=n, seed=9)
    dyn = species_dynamics(sysm, 0.002)
    ff = ForceField(sysm, precision=form)
    return ff, MolecularDynamics(ff, dyn, thermal_state(sysm, dyn, 300.0, 4))


def gradient(ff):
    ff.energy_grad()


def loss_gradient(ff):
    ff.fm_loss_grad(np.zeros((3, ff.sysm.nsites)))


def other_cell(ff):
    """A wider cell: more link cells and k-vectors, larger tables."""
    own = ff.sysm
    h = np.asarray(own.h, float) * 1.3
    x = np.asarray(own.site) + np.repeat(0.3 * np.asarray(own.h) @ np.asarray(own.c_of_m).T, 4, axis=1)
    ff.sysm = dataclasses.replace(own, h=h, site=x)
    ff.forces()
    ff.sysm = own


CASES = [(n, call) for n in (10, 14) for call in (gradient, loss_gradient)] + [(6, gradient), (6, other_cell)]


@pytest.mark.parametrize("form,tol", [("fp64", 1e-11), ("mixed", 1e-6)])
@pytest.mark.parametrize("before", [3, 1])   # replayed already, and run directly only
@pytest.mark.parametrize("n,call", CASES, ids=lambda v: getattr(v, "__name__", str(v)))
def test_run_between_other_calls(n, call, before, form, tol):
    out = []
    for between in (False, True):
        ff, md = start(n, form)
        e = [md.run(before)]
        if between:
            call(ff)
        e.append(md.run(3))
        if between:
            call(ff)
        e.append(md.run(1))
        s = md.state()
        out.append([np.concatenate(e), s.c_of_m, s.mom, s.quat, s.amom])
        ff.close()
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= tol * np.abs(a).max()


@pytest.mark.parametrize("form,tol", [("fp64", 1e-11), ("mixed", 1e-6)])
@pytest.mark.parametrize("before", [3, 1])
@pytest.mark.parametrize("call", [gradient, other_cell], ids=lambda v: v.__name__)
def test_run_between_other_calls_cuda_core_passes(call, before, form, tol, monkeypatch):
    """The k-list tables of the CUDA-core passes are the run's own again."""
    monkeypatch.setenv("MDGPU_KSPACE_TC", "0")
    test_run_between_other_calls(6, call, before, form, tol)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("call", [None, gradient, other_cell], ids=lambda v: getattr(v, "__name__", "info"))
def test_pair_count_after_replayed_steps(call, form):
    """The count is taken from the slots as the last step left them: class by
    class, where a gradient leaves them in plain order, and again for steps
    after one that has been counted.  Exact."""
    counts = []
    for between in (False, True):
        ff, md = start(6, form)
        md.run(3)
        if between:
            assert ff.info()["npairs"] > 0
            if call:
                call(ff)
        md.run(2)
        counts.append(ff.info()["npairs"])
        ff.close()
    assert counts[0] == counts[1] > 0
