"""The adjoint over kept frames against the one that runs the trajectory again
from checkpoints, and the property the latter rests on: pair forces of the Wolf
form have the same bits with and without energies."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, library, synth

pytestmark = pytest.mark.gpu


def _reps(sizes):
    return [synth.to_arrays(synth.nacl_replica(n, seed=5 + k, charge_scale=1.0 - 0.05 * k))
            for k, n in enumerate(sizes)]


# one atom past a 16-atom block; segments that do and do not divide the run
@pytest.mark.parametrize("lkspace,sizes,steps,checkpoint", [
    (1, (514,), 12, 4), (1, (512, 978), 11, 5), (1, (998, 510, 512), 7, 7), (0, (512, 514), 11, 5)])
def test_kept_frames_match_recompute(lkspace, sizes, steps, checkpoint):
    out = []
    reps = _reps(sizes)
    for a in reps:
        a.update(lkspace=lkspace, reacf=1e-3 if lkspace == 0 else 0.0)
    for keep in (1, 0):
        with MDSystem.from_batch(reps) as sim:
            assert library().md_debug_adjoint_frames(sim._ctx, keep) == 0
            o = sim.adjoint(steps, checkpoint=checkpoint, nbins=100)
            out.append((o, sim.positions(), sim.velocities()))
    (a, xa, va), (b, xb, vb) = out
    assert np.array_equal(a["loss"], b["loss"]) and np.array_equal(a["gbar"], b["gbar"])
    assert np.array_equal(xa, xb) and np.array_equal(va, vb)
    # the rows of a frame may be summed in another order: FP32 sums of a few
    # hundred terms that nearly cancel, against the sum of their sizes
    for k in ("dlj1", "dlj2", "dlns"):
        assert np.abs(a[k] - b[k]).max() <= 2e-5 * np.abs(a[k]).max()


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("tpa,depth", [(8, 2), (8, 4), (4, 4), (16, 2)])
def test_forces_same_with_energies(batch, tpa, depth):
    reps = _reps((998, 1728))
    sim = MDSystem.from_batch(reps) if batch else MDSystem.from_arrays(**reps[1])
    with sim:
        sim.set_tuning(tpa, 0, depth)
        sim.compute_forces(energy=False)
        f = sim.forces()
        sim.compute_forces(energy=True)
        assert np.array_equal(f, sim.forces())
