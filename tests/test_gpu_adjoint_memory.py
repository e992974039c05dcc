"""The adjoint keeps every frame only where that takes little memory (1 GiB):
a longer trajectory holds no more than the checkpoints the caller asked for."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, library, synth

pytestmark = pytest.mark.gpu


def test_long_trajectory_uses_the_callers_checkpoints():
    """8 x 7986 ions, 24 bytes each a frame: 701 frames are the first past
    1 GiB.  The run from checkpoints builds its lists a second time, which the
    build count shows."""
    reps = [synth.to_arrays(synth.nacl_replica(7986, seed=5 + k)) for k in range(8)]
    out = []
    for keep in (1, 0):
        with MDSystem.from_batch(reps) as sim:
            assert library().md_debug_adjoint_frames(sim._ctx, keep) == 0
            o = sim.adjoint(720, checkpoint=60, nbins=100)
            out.append((o["loss"], o["dlj1"], o["dlns"], sim.positions(), sim.info()["builds"]))
    assert out[0][4] == out[1][4]
    for a, b in zip(out[0][:4], out[1][:4]):
        assert np.array_equal(a, b)
