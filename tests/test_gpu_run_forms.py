"""Which form the steps of a small single system take, and that every form
gives the same bits."""
import threading

import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, synth

pytestmark = pytest.mark.gpu


def _nacl(natom, seed=4, **kw):
    return synth.to_arrays(synth.nacl_replica(natom=natom, seed=seed, integrator="leapfrog", ensemble="nvt", **kw))


@pytest.mark.parametrize("tpa,depth", [(8, 2), (8, 4), (16, 1), (16, 2), (32, 1)])
def test_every_depth_matches_separate_kernels(tpa, depth):
    """One entry at a time (an odd depth) and two round differently: the run
    takes the form of the context's depth."""
    out = []
    for graphs in (True, False):
        with MDSystem.from_arrays(**_nacl(982)) as s:
            s.set_tuning(tpa, 0, depth if (tpa, depth) not in ((8, 4), (16, 2), (32, 1)) else 0)
            assert (s.info()["pair_tpa"], s.info()["pair_depth"]) == (tpa, depth)
            s.set_graphs(graphs)
            s.step(40, 15)
            out.append((s.positions(), s.velocities(), s.forces()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
