"""Populations that outgrow the list form within a call: the lists stop before the frame that might not fit, and
the rest of the frames run in another form over the whole GPU.  Every frame is the oracle's (integer state: the
tolerance is zero), whichever call first sees the stop, and a growing call does not fall behind the in-place
form (a block that stepped the rest of the call over its whole lattice took some ninety times as long)."""
import time

import numpy as np
import pytest

from cell_simulation_gb300 import CellsimError, Ensemble, RNG_PHILOX, configs
from cell_simulation_gb300.simulation import LatticeParams, Simulation
from tests.helpers import LAM
from tests.test_new_forms_gpu import in_place, lists, one_region
from tests.test_prod_gpu import oracle_prod

pytestmark = pytest.mark.gpu

RATES = (30.0, 10.0, 500.0)  # A -> A + A at 500 / s: some 2.5 times the particles in 40 frames


def growing(K, res=(10, 9, 20)):
    return lambda: one_region(res, K, (60, 20, 0), RATES)


def started(mk, K, form=lists):
    sim = mk()
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    sim.set_tiling(form(K))
    return sim


def same(sim, want):
    assert np.array_equal(sim.get_lattice()[0].astype(np.uint8), want[0])
    assert np.array_equal(sim.counts(), want[1])
    assert np.array_equal(sim.diagnostics()[:4], want[2][:4])


@pytest.mark.parametrize("K", [8, 16])
@pytest.mark.parametrize("reader", ["lattice", "counts", "diagnostics", "view", "synchronize", "checkpoint", "tiling", "timed"])
def test_whatever_sees_the_stop_first(orc, K, reader, tmp_path):
    """Several calls are enqueued, then one reader sees the state first; later frames follow on."""
    mk = growing(K)
    want = oracle_prod(orc, mk(), 48, seed=7)
    assert want[1].sum() > 800
    sim = started(mk, K)
    for n in (1, 40, 5, 2):
        sim.step_philox(n, 7)
    if reader == "lattice":
        assert np.array_equal(sim.get_lattice()[0].astype(np.uint8), want[0])
    elif reader == "counts":
        assert np.array_equal(sim.counts(), want[1])
    elif reader == "diagnostics":
        assert np.array_equal(sim.diagnostics()[:4], want[2][:4])
    elif reader == "view":
        got = sim.render_view()
        ref = started(mk, K, in_place)
        ref.step_philox(48, 7)
        assert np.array_equal(got, ref.render_view())
    elif reader == "synchronize":
        sim.synchronize()
        assert sim.get_tiling() != lists(K)
    elif reader == "checkpoint":
        path = tmp_path / "state"
        sim.save_checkpoint(path)
        other = Simulation.load_checkpoint(path)
        assert np.array_equal(other.get_lattice()[0].astype(np.uint8), want[0])
        assert np.array_equal(other.counts(), want[1])
    elif reader == "tiling":
        sim.set_tiling(in_place(K))
    else:
        assert sim.step_philox_timed(4, 7) > 0.0
        want = oracle_prod(orc, mk(), 52, seed=7)
        same(sim, want)
        return
    same(sim, want)
    sim.step_philox(9, 7)
    same(sim, oracle_prod(orc, mk(), 57, seed=7))


@pytest.mark.parametrize("K", [8, 16])
def test_samples_of_a_growing_call(orc, K):
    """Logged counts of one call, before and after the stop, each the oracle's of its frame."""
    mk = growing(K)
    sim = started(mk, K)
    sim.step_philox(46, 7, 3)
    got = {}
    for s in sim.stats:
        got.setdefault(s.iteration_count, []).append(s.value)
    assert sorted(got) == list(range(3, 46, 3))
    for f in got:
        assert got[f] == [int(c) for c in oracle_prod(orc, mk(), f, seed=7)[1][1:]], f
    same(sim, oracle_prod(orc, mk(), 46, seed=7))


@pytest.mark.parametrize("change", ["seed", "precision", "upload"])
def test_changes_after_an_unseen_stop(orc, change):
    """A change of the seed, the precision or the lattice right after the enqueued frames applies to the frames
    after them."""
    mk = growing(16)
    mid = oracle_prod(orc, mk(), 45, seed=7)
    sim = started(mk, 16)
    sim.step_philox(45, 7)
    if change == "upload":
        sim.set_lattice(mk().get_lattice()[0])
        assert np.array_equal(sim.diagnostics()[:4], mid[2][:4])
        sim.step_philox(6, 7)
        want_s, want_c, _ = oracle_prod(orc, mk(), 6, seed=7, frame0=45)
    else:
        if change == "precision":
            sim.set_precision(2)
        sim.step_philox(6, 8 if change == "seed" else 7)
        ref = started(mk, 16, in_place)
        ref.step_philox(45, 7)
        if change == "precision":
            ref.set_precision(2)
        ref.step_philox(6, 8 if change == "seed" else 7)
        want_s, want_c = ref.get_lattice()[0].astype(np.uint8), ref.counts()
    assert np.array_equal(sim.get_lattice()[0].astype(np.uint8), want_s)
    assert np.array_equal(sim.counts(), want_c)


def test_long_growing_call(orc):
    """A call of several launches whose population grows through list lengths and out of the form."""
    mk = lambda: one_region((20, 18, 18), 8, (20, 10, 0), (3.0, 1.0, 8.0))
    n = 3400
    want = oracle_prod(orc, mk(), n, seed=3)
    assert want[1].sum() > 1400
    sim = started(mk, 8)
    sim.step_philox(n, 3)
    same(sim, want)


@pytest.mark.parametrize("K", [8, 16])
def test_list_chosen_for_too_many_particles(orc, K):
    """The particles have grown unseen by the host when the list variant is chosen: more voxels are occupied than
    its lists hold, and the frames run in another form."""
    mk = growing(K, (16, 15, 20))
    want = oracle_prod(orc, mk(), 90, seed=11)
    assert (want[0].reshape(-1, K) > 0).any(1).sum() > 704
    sim = started(mk, K, in_place)
    sim.step_philox(84, 11)
    sim.set_tiling(lists(K))
    sim.step_philox(6, 11)
    same(sim, want)
    assert sim.get_tiling() != lists(K)


@pytest.mark.parametrize("K", [8, 16])
@pytest.mark.parametrize("batched", [True, False])
def test_replicates_outgrow_at_their_own_frames(K, batched):
    """Uneven replicates with rate multipliers from 1/50 to 2: some outgrow their lists early, some late, some never;
    against the in-place form."""
    D = 1e-12
    def template():
        t = Simulation(LatticeParams([8 * LAM] * 3, [8, 8, 8], configs.stable_tau(D), LAM, K))
        t.set_diffusion_rate("background", D)
        t.prepare_regions()
        for s in "ABC":
            t.add_particle_count(s, "background", 0, True, False)
        t.set_diffusion_rate("background", D)
        t.add_reaction(["A", "B"], ["C"], RATES[0])
        t.add_reaction(["C"], ["A", "B"], RATES[1])
        t.add_reaction(["A"], ["A", "A"], RATES[2])
        return t
    res = np.array([[9, 9, 33], [12, 8, 12], [6, 7, 64], [16, 16, 16], [15, 15, 15], [10, 10, 10]], np.uint32)
    out = []
    for form in (lists, in_place):
        ens = Ensemble(template(), res, np.arange(1, 7, dtype=np.uint64),
                       np.array([0.02, 1.0, 0.7, 2.0, 1.5, 0.02], np.float32), np.array([0, 60, 20, 0], np.uint32))
        ens.set_tiling(form(K))
        got = []
        for n in (30, 25, 5, 1, 7):
            ens.step(n, batched=batched)
            if n != 25:
                got += [ens.counts(), ens.slots(), ens.diagnostics()[:4]]
        out.append(got)
    for i, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), i


def test_time_of_a_growing_call():
    """One call in which 20 particles fill a 40 cubed lattice, by default and in place from the start."""
    ms = []
    for tiling in (None, in_place(8)):
        best = np.inf
        for _ in range(2):
            sim = one_region((40, 40, 40), 8, (20, 0, 0), (30.0, 10.0, 300.0))
            sim.prepare_for_gpu(RNG_PHILOX, 0)
            if tiling is None:
                assert sim.get_tiling() == lists(8)
            else:
                sim.set_tiling(tiling)
            t = time.perf_counter()
            sim.step_philox(400, 7)
            total = sim.counts().sum()
            best = min(best, time.perf_counter() - t)
            assert total > 50000
            sim.close()
        ms.append(best * 1e3)
    assert ms[0] < 5.0 * ms[1], ms
