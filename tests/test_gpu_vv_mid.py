"""Step graphs of velocity Verlet without a thermostat run the second half of a
step and the first half of the next as one kernel (k_vv_mid, k_vv_mid_b): bit
for bit the run of the separate kernels launched step by step."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, synth

pytestmark = pytest.mark.gpu


def _nacl(natom, seed=4, **kw):
    return synth.to_arrays(synth.nacl_replica(natom=natom, seed=seed, **kw))


# one step (no middle), an even and an odd run, one with steps after its last
# graph, energies between (runs that start between two of them too); the batch
# has replicas of one block, of a last block of one atom pair and of several
@pytest.mark.parametrize("steps,every", [(1, 0), (2, 0), (19, 0), (45, 0), (24, 5), (9, 1)])
@pytest.mark.parametrize("kind", ["single", "fp64", "batch"])
def test_fused_halves_match_separate_kernels(kind, steps, every):
    out = []
    for graphs in (True, False):
        if kind == "batch":
            sim = MDSystem.from_batch([_nacl(n, rc=6.0) for n in (120, 258, 1000)])
        else:
            sim = MDSystem.from_arrays(**_nacl(9800 if kind == "single" else 500, rc=8.0))
        with sim:
            if kind == "fp64":
                sim.set_precision(64)
            sim.set_graphs(graphs)
            for _ in range(3):
                sim.step(steps, every)
            out.append([sim.positions(), sim.velocities(), sim.forces(), sim.order(), sim.history(3 * steps),
                        sim.thermo()])
    for a, b in zip(*out):
        assert np.array_equal(a, b) if isinstance(a, np.ndarray) else a == b
