"""The end of a batch's step: each replica's thermostat, pressure and box by
the last of its integrator blocks, the batch's record by the last replica."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem, synth

pytestmark = pytest.mark.gpu

STEPS = 23


# one replica (no sum over replicas), a few, one more than a warp, more than
# an integrator block has threads (384), of one to four blocks each
@pytest.mark.parametrize("nrep", [1, 3, 33, 400])
@pytest.mark.parametrize("integrator,ensemble", [("vv", "nvt"), ("leapfrog", "nvt"), ("leapfrog", "npt")])
def test_records_of_equal_replicas(nrep, integrator, ensemble):
    """Copies of three systems: copies stay equal bit for bit wherever they
    sit in the batch, and the batch's record is the replicas' sum (FP64, up to
    400 terms: 1e-12 is above 400 x 2^-53)."""
    kinds = [synth.to_arrays(synth.nacl_replica(natom=n, seed=n, rc=6.0, integrator=integrator,
                                                    ensemble=ensemble))
             for n in (216, 256, 400)]
    with MDSystem.from_batch([kinds[r % 3] for r in range(nrep)]) as b:
        b.step(STEPS, 5)
        b.step(2, 1)
        th, total, hist = b.replica_thermo(), b.thermo(), b.history(STEPS + 2)
    assert [h["step"] for h in hist] == list(range(hist[0]["step"], hist[0]["step"] + STEPS + 2))
    for r in range(nrep):
        assert th[r] == th[r % 3]
    for key in ("ke", "pe"):
        s = sum(t[key] for t in th)
        assert abs(s - total[key]) <= 1e-12 * abs(s)
        assert hist[-1][key] == total[key]
    assert all(np.isfinite(list(t.values())).all() for t in th)
