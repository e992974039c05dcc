"""The warp-per-part list builder against the lanes-per-atom builder, which
shares none of its candidate handling: the same neighbours, and (through
bit-equal forces, summed in list order) in the same order."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, synth

pytestmark = pytest.mark.gpu

# groups of more than 32 atoms and more than one 1024-candidate chunk (dense
# ions), one warp per atom (few cells), per-pair shifts and image cells, cell
# counts below and above the one-block scan (2048 cells), exclusions, a row
# count at the capacity's edge (nmaxlist)
CASES = {
    "dense": lambda: synth.nacl_replica(4096, seed=1, density=9.0, rc=9.0, nmaxlist=1600, jitter=0.1),
    "few_cells": lambda: synth.nacl_replica(512, seed=2),
    "odd": lambda: synth.nacl_replica(2702, seed=3),
    "images": lambda: synth.nacl_replica(9602, seed=4),
    "many_cells": lambda: synth.argon_fcc(ncell=18, seed=5),
    "full_rows": lambda: synth.nacl_replica(4096, seed=6, nmaxlist=32),
    "water": lambda: synth.water_grid(nside=11, seed=7),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_parts_match_lanes_per_atom(name, tmp_path):
    sys_ = CASES[name]()
    base = synth.write_case(sys_, str(tmp_path), "s")
    out = []
    for list_tpa in (0, 8):
        with MDSystem.from_files(base) as sim:
            sim.set_tuning(8, list_tpa)
            sim.update_neighbors(True)
            nmax = sim.info()["max_neighbors"]
            nn, nm = sim.neighbor_list(nmax)
            sim.compute_forces()
            out.append((nn, nm, sim.forces(), sim.order()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
