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


def test_default_form_follows_the_tuning():
    """Step graphs that nobody chose a form for: rebuild inline and fused step
    wherever the steps do not run in one launch, after every setting that
    changes that; a chosen form stays."""
    def form(s):
        i = s.info()
        return bool(i["rebuild_inline"]), bool(i["fused_step"])

    for natom, tunings in ((982, (((4, 0), True), ((8, 0), False), ((8, 8), True), ((32, 0), False))),
                           (9602, (((16, 0), True), ((8, 0), False), ((8, 4), True))),
                           (13822, (((8, 8), True), ((8, 0), True), ((16, 0), True)))):
        with MDSystem.from_arrays(**_nacl(natom)) as s:
            assert form(s) == ((natom > 9696),) * 2
            for (tpa, ltpa), on in tunings:
                s.set_tuning(tpa, ltpa)
                assert form(s) == (on, on), (natom, tpa, ltpa)
                s.step(6)
            s.set_fused_step(False)
            s.set_graph_rebuild(False)
            s.set_tuning(4, 0)
            assert form(s) == (False, False)
            s.step(6)


@pytest.mark.parametrize("natom", [510, 982, 4080, 9602])
def test_autotuned_small_system_runs_in_one_launch(natom):
    """With a block dropped (test hook) and no rebuild due, steps time out in
    the one launch only: the separate kernels have no wait then."""
    from md_gpu_gb300.system import MDError, library
    with MDSystem.from_arrays(**_nacl(natom)) as s:
        s.step(16)
        s.autotune()
        i = s.info()
        assert i["list_tpa"] == 0 and i["pair_tpa"] >= 8
        s.update_neighbors(force=True)
        assert library().md_debug_rebuild_barrier(s._ctx, 2.0, 0) == 0
        with pytest.raises(MDError):
            s.step(4)


def test_control_of_the_above():
    from md_gpu_gb300.system import library
    with MDSystem.from_arrays(**_nacl(982)) as s:
        s.step(16)
        s.set_tuning(4, 0)
        s.update_neighbors(force=True)
        assert library().md_debug_rebuild_barrier(s._ctx, 2.0, 0) == 0
        s.step(4)


@pytest.mark.parametrize("sizes", [(982, 982, 982), (9602, 9602), (982, 13822)])
def test_contexts_stepped_at_once(sizes):
    """Contexts of several threads at work together, each launch needing its
    blocks resident (9602 ions: nearly the whole device each): the same bits
    as one after the other, runs of more than one launch among them."""
    def make(k, n):
        return MDSystem.from_arrays(**_nacl(n, seed=4 + k))

    def go(s):
        for n in (300, 7, 64):
            s.step(n)

    alone = []
    for k, n in enumerate(sizes):
        with make(k, n) as s:
            go(s)
            alone.append(s.positions())
    sims = [make(k, n) for k, n in enumerate(sizes)]
    errors = []

    def work(s):
        try:
            go(s)
        except Exception as e:   # raised in the test's own thread below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in sims]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    try:
        assert not errors, errors
        for s, p in zip(sims, alone):
            assert np.array_equal(s.positions(), p)
    finally:
        for s in sims:
            s.close()
