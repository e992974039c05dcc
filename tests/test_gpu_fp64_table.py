"""FP64 mode: pair forces without energies (the Coulomb term from a table of
polynomials, 1/r by iteration) against those with energies (exp and divide as
written), over the tables' piece counts and where no table is accurate enough."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, synth

pytestmark = pytest.mark.gpu


# a rc = 1 (16 pieces), 2.4 (32), 3.09 (64, real-space Ewald), 12 (no table); RF
@pytest.mark.parametrize("lkspace,alpha", [(1, 0.1), (1, 0.24), (2, None), (1, 1.2), (0, None)])
@pytest.mark.parametrize("natom", [998, 2744])
def test_forces_with_and_without_energies(lkspace, alpha, natom):
    a = synth.to_arrays(synth.nacl_replica(natom, seed=3, rc=10.0, alpha=alpha or 0.2))
    a["lkspace"] = lkspace
    if lkspace == 2:
        a["alfa"] = float(np.float32(3.09 / np.sqrt(a["rcutsq"])))
    if lkspace == 0:
        a["reacf"] = float(np.float32(0.9 / np.sqrt(a["rcutsq"]) ** 3))
    with MDSystem.from_arrays(**a) as sim:
        sim.set_precision(64)
        out = []
        for energy in (False, True):
            sim.compute_forces(energy=energy)
            out.append(sim.forces()[:, :3])
    # 8 lane sums, each rounded to 2^-32 on both sides, and 2e-14 of the sum of
    # the pair forces' sizes (under 1.5e5 kJ/mol/A per atom)
    assert np.abs(out[0] - out[1]).max() <= 8 * 2.0 ** -32 + 2e-14 * 1.5e5
    assert np.abs(out[1]).max() > 1.0
