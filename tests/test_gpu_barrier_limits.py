"""The bounded waits of the kernels that hold grid barriers: a block that
leaves before the first one (test hook, the wait shortened to 2 ms) makes the
others give up, set the sticky status and return; the calls report it and the
GPU runs on.  (The single systems' rebuild kernel is in test_gpu_faults.py.)"""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, synth
from md_gpu_gb300.system import MDError, library

pytestmark = pytest.mark.gpu


def _nacl(natom, seed=4, **kw):
    return synth.to_arrays(synth.nacl_replica(natom=natom, seed=seed, **kw))


def _times_out(call):
    with pytest.raises(MDError) as e:
        call()
    assert e.value.status == 4 and "grid barrier" in str(e.value)


@pytest.mark.parametrize("drop", [0, 5, 123])   # first, middle, the bookkeeping block
@pytest.mark.parametrize("integrator", ["vv", "leapfrog"])
def test_run_of_steps(integrator, drop):
    """982 ions at 32 lanes: 123 blocks of atoms and the bookkeeping block."""
    a = _nacl(982, integrator=integrator)
    sim = MDSystem.from_arrays(**a)
    try:
        sim.set_tuning(32, 0)
        sim.step(8)
        step0, builds = sim.thermo()["step"], sim.info()["builds"]
        sim.update_neighbors(force=True)      # no rebuild is due in the next steps
        assert library().md_debug_rebuild_barrier(sim._ctx, 2.0, drop) == 0
        _times_out(lambda: sim.step(4))
        assert sim.thermo()["step"] == step0 and sim.info()["builds"] == builds + 1
        assert library().md_debug_rebuild_barrier(sim._ctx, 0.0, -1) == 0
        _times_out(lambda: sim.step(4))       # sticky
    finally:
        sim.close()
    with MDSystem.from_arrays(**a) as sim:
        sim.step(8)
        assert np.isfinite(sim.thermo()["temper"])


def test_batch_rebuild():
    reps = [_nacl(998, seed=k) for k in (4, 5)]
    sim = MDSystem.from_batch(reps)
    try:
        sim.step(4)
        order, builds = sim.order(), sim.info()["builds"]
        assert library().md_debug_rebuild_barrier(sim._ctx, 2.0, 0) == 0
        _times_out(lambda: sim.update_neighbors(force=True))
        assert np.array_equal(sim.order(), order) and sim.info()["builds"] == builds
        _times_out(lambda: sim.step(4))
    finally:
        sim.close()
    with MDSystem.from_batch(reps) as sim:
        sim.step(8)
        assert np.isfinite(sim.thermo()["temper"])
