"""A list rebuild asked for before a run of many steps in one launch
(k_run_steps) happens before the run's first forces, with every integrator.
The request comes from md_debug_list_capacity, which also replaces the list."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, synth
from md_gpu_gb300.system import library

pytestmark = pytest.mark.gpu


def _system(kind, tmp_path):
    if kind == "nh":
        return MDSystem.from_files(synth.write_case(synth.water_grid(seed=5, nside=8), str(tmp_path), "w"))
    return MDSystem.from_arrays(**synth.to_arrays(synth.nacl_replica(
        982, seed=6, nmaxlist=512, integrator="vv" if kind == "vv" else "leapfrog")))


@pytest.mark.parametrize("kind", ["vv", "nh", "leapfrog"])
def test_pending_rebuild_comes_first(kind, tmp_path):
    """The list replaced and a rebuild asked for: the run builds it before it
    reads it, as the separate kernels do (same bits, same build count), and
    an overflow in that rebuild grows the list and runs the steps again.
    (Velocity Verlet then builds before its first drift instead of after it:
    another atom order, so FP32 sums rounded otherwise, 1e-6 of forces that
    move an atom by less than 1 A in nine steps.)"""
    L = library()
    out = []
    for graphs, cap in ((True, 1024), (False, 1024), (True, 64)):
        with _system(kind, tmp_path) as s:
            s.set_tuning(16, 0)
            s.set_graphs(graphs)
            s.step(6)
            b0 = s.info()["builds"]
            assert L.md_debug_list_capacity(s._ctx, cap, 1) == 0
            s.step(9)
            i = s.info()
            assert i["builds"] > b0 and i["list_regrows"] == (1 if cap == 64 else 0)
            assert i["capacity"] >= i["max_neighbors"] > 64
            out.append((s.positions(), s.velocities(), s.forces(), s.order(), i["builds"] - b0))
    for a, b in zip(out[0], out[1]):
        assert np.array_equal(a, b)
    if kind == "leapfrog":
        assert all(np.array_equal(out[0][k], out[2][k]) for k in (0, 1, 2))
    else:
        d = out[0][0] - out[2][0]
        assert np.abs(np.where(np.abs(d) > 5.0, 0.0, d)).max() <= 1e-5   # 5: across the periodic wrap
