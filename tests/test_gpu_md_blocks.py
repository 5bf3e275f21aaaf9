"""The molecular correction of the stress (k_md_virc, k_md_virc2) over the
numbers of blocks where its second reduction changes shape: up to 32 blocks,
up to 64, more (a wider block), and the larger first-level blocks of large
systems.  From a state at rest and a vanishing time step the dump record's
stress is that of the start: the force field's, mirrored, less
sum f (x) (x - R).  The distant-potential term sits on the diagonal alone and
equally, so off-diagonal elements and differences of diagonal ones are
compared.

Tolerance: the record holds float32 (2^-24 of each element, two in a
difference), the rest is FP64: 4e-7 of the largest element."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside", [4, 6, 7, 8, 9, 17])   # 8, 27, 43, 64, 92 and 77 (of 256 sites) blocks
def test_dump_stress_molecular_correction(nside):
    from moldy_gb300 import ForceField, system
    from moldy_gb300.dumpfile import split_record
    from moldy_gb300.dynamics import MolecularDynamics, MDState, species_dynamics, thermal_state
    sysm = system.water(nside=nside, seed=5)
    dyn = species_dynamics(sysm, 1e-9)
    st = thermal_state(sysm, dyn, 0.0, 1)
    ff = ForceField(sysm, precision="fp64")
    f, _, s = ff.forces()
    s = np.triu(np.asarray(s).reshape(3, 3))
    s = s + np.triu(s, 1).T
    md = MolecularDynamics(ff, dyn, MDState(st.c_of_m, 0 * st.mom, st.quat, 0 * st.amom))
    _, rec = md.run_dump(1, 1, 8)
    ff.close()
    got = split_record(rec[0], 8, sysm.nmols, md.nq)["stress"].astype(float)
    h = np.asarray(sysm.h, float)
    d = np.asarray(sysm.site) - np.repeat(h @ np.asarray(sysm.c_of_m).T, 4, axis=1)
    d -= h @ np.rint(np.linalg.inv(h) @ d)
    want = s - np.asarray(f).reshape(3, -1) @ d.T
    scale = np.abs(want).max()

    def parts(a):
        return np.array([a[0, 1], a[0, 2], a[1, 0], a[1, 2], a[2, 0], a[2, 1], a[0, 0] - a[1, 1], a[1, 1] - a[2, 2]])
    assert np.abs(parts(got) - parts(want)).max() <= 4e-7 * scale
