"""Many steps of a small system in one launch (k_run_steps): bit for bit the
run of the separate kernels launched step by step (md_set_graphs off)."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, synth

pytestmark = pytest.mark.gpu

# (system, lanes per atom, steps, energy_every): block edges (256 / lanes atoms
# per block), one atom more and less than a block, the largest system that runs
# this way, odd and even step counts (position buffers), energy steps between
CASES = [
    ("argon", dict(ncell=4), 8, 41, 0),
    ("argon", dict(ncell=5), 16, 40, 7),
    ("argon", dict(ncell=9), 32, 33, 16),
    ("nacl", dict(natom=510), 8, 64, 0),
    ("nacl", dict(natom=514), 16, 31, 10),
    ("nacl", dict(natom=9602), 8, 24, 0),
    ("water", dict(nside=8), 8, 40, 0),
    ("water", dict(nside=9), 16, 37, 12),
    ("water", dict(nside=8), 32, 24, 0),
]


def _system(kind, kw, tmp_path):
    if kind == "argon":
        return MDSystem.from_arrays(**synth.to_arrays(synth.argon_fcc(seed=3, integrator="vv", **kw)))
    if kind == "nacl":
        return MDSystem.from_arrays(**synth.to_arrays(synth.nacl_replica(
            seed=4, integrator="leapfrog", ensemble="nvt", **kw)))
    return MDSystem.from_files(synth.write_case(synth.water_grid(seed=5, **kw), str(tmp_path), "w"))


@pytest.mark.parametrize("kind,kw,tpa,steps,every", CASES)
def test_small_run_matches_separate_kernels(kind, kw, tpa, steps, every, tmp_path):
    out = []
    for graphs in (True, False):
        with _system(kind, kw, tmp_path) as sim:
            sim.set_tuning(tpa, 0)
            sim.set_graphs(graphs)
            sim.step(steps, every)
            mid = [sim.positions(), sim.velocities(), sim.forces()]
            sim.step(steps, every)
            out.append(mid + [sim.positions(), sim.velocities(), sim.forces(), sim.order(), sim.history(2 * steps),
                              sim.info()["builds"]])
    for k, (a, b) in enumerate(zip(*out)):
        if isinstance(a, np.ndarray):
            assert np.array_equal(a, b), f"output {k} differs by {np.abs(a - b).max()}"
        else:
            assert a == b
    assert out[0][-1] >= 2


def test_two_small_systems_interleaved():
    """Runs of two contexts in turn do not see each other's barrier state."""
    def make(seed):
        return MDSystem.from_arrays(**synth.to_arrays(synth.argon_fcc(ncell=5, seed=seed, integrator="vv")))

    alone = []
    for seed in (1, 2):
        with make(seed) as s:
            for n in (5, 8, 21):
                s.step(n)
            alone.append(s.positions())
    with make(1) as a, make(2) as b:
        for n in (5, 8, 21):
            a.step(n)
            b.step(n)
        assert np.array_equal(a.positions(), alone[0]) and np.array_equal(b.positions(), alone[1])


def test_list_after_creation():
    """The first list build waits for the uploads and memsets of the creation
    (they run on another stream): many creations, always the same list."""
    a = synth.to_arrays(synth.argon_fcc(ncell=7, seed=3, integrator="vv"))
    counts = []
    for _ in range(60):
        with MDSystem.from_arrays(**a) as sim:
            counts.append(sim.neighbor_list(128)[1])
    assert counts[0][:1372].min() > 0
    assert all(np.array_equal(c, counts[0]) for c in counts)


@pytest.mark.parametrize("natom,lanes", [(510, 32), (1208, 32), (1210, 16), (4848, 16), (4850, 8)])
def test_lanes_by_size(natom, lanes):
    """A new single system's lanes per atom follow its size (152 SMs: 1208 and
    4848 atoms are the last of 32 and 16 lanes).  The forces differ from those
    of 8 lanes by the rounding of FP32 sums only: both are within 1e-5 (rms,
    relative) of the FP64 forces, hence within 2e-5 of each other.  A depth
    set first brings the context to the 8 lanes that it was built for."""
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("sizes are for 152 SMs")
    arrays = synth.to_arrays(synth.nacl_replica(seed=6, natom=natom, integrator="leapfrog"))
    F = []
    for first in (lambda s: None, lambda s: s.set_tuning(8, 0), lambda s: s.set_tuning(8, 0, 2)):
        with MDSystem.from_arrays(**arrays) as sim:
            assert sim.info()["pair_tpa"] == lanes
            first(sim)
            sim.compute_forces()
            F.append(sim.forces()[:, :3])
            sim.step(5)
            F.append(sim.forces()[:, :3])
    for k in (0, 1):
        d = np.sqrt(((F[k] - F[2 + k]) ** 2).mean() / (F[2 + k] ** 2).mean())
        assert d <= 2e-5
        assert np.array_equal(F[2 + k], F[4 + k])
    with MDSystem.from_arrays(**arrays) as sim:
        from md_gpu_gb300.system import library
        for depth, ok in ((1, False), (4, True), (2, True)):
            assert (library().md_set_pair_depth(sim._ctx, depth) == 0) == ok
        assert sim.info()["pair_tpa"] == 8 and sim.info()["pair_depth"] == 2


def test_large_forces_match_separate_kernels():
    """Two atoms 0.45 sigma apart: forces above 2^18 take the run's
    general force conversion and still give the separate kernels' bits."""
    a = synth.to_arrays(synth.argon_fcc(ncell=5, seed=3, integrator="vv"))
    a["pos"] = np.array(a["pos"], copy=True)
    a["pos"][1] = a["pos"][0] + np.array([0.45, 0.0, 0.0], a["pos"].dtype)
    out = []
    for graphs in (True, False):
        with MDSystem.from_arrays(**a) as sim:
            sim.set_graphs(graphs)
            assert np.abs(sim.forces()[:2, 0]).min() > 2.0 ** 18
            sim.step(4)
            out.append((sim.positions(), sim.velocities(), sim.forces()))
    for p, q in zip(*out):
        assert np.array_equal(p, q)


def test_short_rows_keep_eight_lanes():
    with MDSystem.from_arrays(**synth.to_arrays(synth.argon_fcc(ncell=5, seed=3, integrator="vv"))) as sim:
        assert sim.info()["pair_tpa"] == 8 and sim.info()["pair_depth"] == 2
