"""The tensor-core reciprocal space of both forms (products of per-axis trig
tables, kspace_q.cu, and the mixed force pass, kspace_tc.cu) against the
CUDA-core passes at the sizes where its tiling can go wrong: charged-site
counts around the 32-site stages and 128-site tiles, |l| ranges around the
column blocks (8, 16, 32, 40, 64), row tiles that span several blocks of h,
triclinic cells (|l| not symmetric about a column's middle) and net charge.

Tolerances.  FP64: both paths are FP64-accurate sums (operands to 2^-55, the
CUDA-core recurrence a few 2^-53 per term), held to the parity tests' 1e-12
of the RMS force.  Mixed: 1e-5 of the FP64 result, the form's bound."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ions(n, box, kc, tilt=0.0, seed=1, net=False):
    from moldy_gb300 import system as S
    rng = np.random.default_rng(seed)
    h = np.diag(np.asarray(box, float))
    h[0, 1], h[0, 2], h[1, 2] = tilt * box[1], 0.7 * tilt * box[2], -tilt * box[2]
    x = h @ rng.uniform(-0.499, 0.499, (3, n))
    half = n // 2
    species = [S.Species("A", half, np.array([1], np.int32), np.zeros((1, 3))),
               S.Species("B", n - half, np.array([2], np.int32), np.zeros((1, 3)))]
    species = [s for s in species if s.nmols]
    q = np.array([0.0, 1.0, 0.7 if net else -1.0]) / S.CONV_Q
    return S.System(h=h, species=species, ptype=S.LJPOT, potpar=np.zeros((9, 8)), site_charge=q, site=x,
                    c_of_m=(np.linalg.inv(h) @ x).T, control=S.Control(cutoff=3.0, alpha=0.45, k_cutoff=kc))


def lbox(trange, kc):
    return 2 * math.pi * (trange - 0.5) / kc


CASES = [dict(n=n, box=(9, 9, 9), kc=4.0) for n in (1, 2, 31, 32, 33, 127, 128, 129, 1025, 4097)]
CASES += [dict(n=65, box=(7, 8, lbox(t, 3.0)), kc=3.0) for t in (3, 8, 9, 16, 17, 32, 33, 40, 41, 64, 65, 81, 130)]
CASES += [dict(n=200, box=(lbox(t, 3.0), 7, 8), kc=3.0) for t in (33, 70)]
CASES += [dict(n=200, box=(7, lbox(t, 3.0), 8), kc=3.0) for t in (33, 70)]
CASES += [dict(n=300, box=(20, 22, 24), kc=3.0, tilt=t, net=net) for t in (0.1, -0.25) for net in (False, True)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(
    str(round(v, 1) if isinstance(v, float) else v) for v in c.values()).replace(" ", ""))
def test_matches_cuda_core_passes(case, monkeypatch):
    from moldy_gb300 import ForceField
    sysm = ions(**case)
    res = {}
    for form in ("fp64", "mixed"):
        for tc in ("1", "0"):
            monkeypatch.setenv("MDGPU_KSPACE_TC", tc)
            ff = ForceField(sysm, precision=form)
            res[form, tc] = ff.ewald()
            self_e = abs(ff.info()["self_energy"])
            ff.close()
    f0, e0, s0 = res["fp64", "0"]
    # a single site feels no net force: the terms' own size is the scale
    scale = max(np.sqrt((f0 ** 2).mean()), 1e-3 * self_e / sysm.nsites)
    for form, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
        f, e, s = res[form, "1"]
        assert np.sqrt(((f - f0) ** 2).mean()) <= tol * scale, form
        assert abs(e - e0) <= tol * (abs(e0) + self_e), form
        assert np.abs(s - s0).max() <= tol * (np.abs(s0).max() + self_e), form


@pytest.mark.parametrize("case", [CASES[k] for k in (1, 4, 8, 13, 18, 23, 29)], ids=lambda c: "-".join(
    str(round(v, 1) if isinstance(v, float) else v) for v in c.values()).replace(" ", ""))
@pytest.mark.parametrize("loss", [False, True])
def test_adjoint_matches_cuda_core_passes(case, loss, monkeypatch):
    """Charge and alpha gradients at the tiling's edges.  The reference forces
    are zero, so the residual is the force itself (random positions: over
    several decades) and the mixed form's relative force error carries over:
    the bounds of the adjoint's oracle tests, FP64 1e-9 and mixed 2e-5 of the
    largest entry, twice that for the loss."""
    from moldy_gb300 import ForceField
    sysm = ions(**case)
    fref = np.zeros((3, sysm.nsites))
    res = {}
    for form, tc in (("fp64", "0"), ("fp64", "1"), ("mixed", "1")):
        monkeypatch.setenv("MDGPU_KSPACE_TC", tc)
        ff = ForceField(sysm, precision=form)
        res[form, tc] = ff.fm_loss_grad(fref, 0.3) if loss else ff.energy_grad()
        ff.close()
    v0, g0 = res["fp64", "0"]
    for form, tol in (("fp64", 1e-9), ("mixed", 2e-5)):
        v, g = res[form, "1"]
        if form == "fp64" or loss:
            assert abs(v - v0) <= 2 * tol * abs(v0), form
        assert np.abs(g["chg"] - g0["chg"]).max() <= tol * np.abs(g0["chg"]).max(), form
        if form == "fp64":
            assert abs(g["alpha"] - g0["alpha"]) <= tol * (abs(g0["alpha"]) + np.abs(g0["chg"]).max())


@pytest.mark.parametrize("nside,nwall,wall_charge,water_charge", [
    (6, 7, 0.4, True), (7, 8, 0.4, True), (8, 12, 0.3, True), (6, 5, 0.0, True), (6, 7, 0.4, False)])
def test_framework_matches_cuda_core_passes(nside, nwall, wall_charge, water_charge, monkeypatch):
    """A framework molecule: its charged sites in tiles of their own, fewer
    and more than one, none, and nothing else charged."""
    import dataclasses

    from moldy_gb300 import ForceField
    from moldy_gb300 import system as S
    sysm = S.water_on_framework(nside=nside, nlayers=nside - 2, nwall=nwall, seed=3, wall_charge=wall_charge)
    if not water_charge:
        q = np.array(sysm.site_charge)
        q[1:4] = 0.0
        sysm = dataclasses.replace(sysm, site_charge=q)
    res = {}
    for form in ("fp64", "mixed"):
        for tc in ("1", "0"):
            monkeypatch.setenv("MDGPU_KSPACE_TC", tc)
            ff = ForceField(sysm, precision=form)
            res[form, tc] = ff.ewald() + (ff.forces(),)
            self_e = abs(ff.info()["self_energy"])
            ff.close()
    f0, e0, s0, t0 = res["fp64", "0"]
    scale = max(np.sqrt((f0 ** 2).mean()), 1e-3 * self_e / sysm.nsites)
    for form, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
        f, e, s, t = res[form, "1"]
        assert np.sqrt(((f - f0) ** 2).mean()) <= tol * scale, form
        assert abs(e - e0) <= tol * (abs(e0) + self_e), form
        assert np.abs(s - s0).max() <= tol * (np.abs(s0).max() + self_e), form
        assert np.abs(t[1] - t0[1]).max() <= tol * (np.abs(t0[1]).max() + self_e), form
