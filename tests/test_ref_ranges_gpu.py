"""The three launches of a reference-RNG frame (and the one block that runs them on small lattices) where
they can go wrong, bit for bit against the serial oracle (integer state: the tolerance is zero): lattices
that end inside a bitmap word or a block's range, slots that are not 4, 8 or 16, rows of voxels whose
occupancy and counts are not those of their slots (uploaded so, or made so by a reaction that takes more
than there is, a reservoir or a rollback), reaction masks of two and three words, tables too large for
shared memory, and contended frames."""
import numpy as np
import pytest

from cell_simulation_gb300 import RNG_REFERENCE, configs
from cell_simulation_gb300.simulation import LatticeParams, Simulation
from tests.helpers import LAM, crowded_model, itime_schedule, multi_region_model, oracle_args, ref_state
from tests.test_ref_parity_gpu import assert_same, run_pair

pytestmark = pytest.mark.gpu


def network(res, K, species, reactions, count, seed=4):
    """species S0 .. on one region, reactions a -> b around the ring, then pairs."""
    D = 1e-12
    sim = Simulation(LatticeParams([r * LAM for r in res], list(res), configs.stable_tau(D), LAM, K))
    sim.seed_placement(seed)
    sim.set_diffusion_rate("background", D)
    sim.prepare_regions()
    names = [f"S{i}" for i in range(species)]
    for n in names:
        sim.add_particle_count(n, "background", count, True, False)
    sim.set_diffusion_rate("background", D)
    for r in range(reactions):
        a, b, c = names[r % species], names[(r * 7 + 1) % species], names[(r * 3 + 2) % species]
        sim.add_reaction([a] if r % 3 else [a, b], [c], 20.0 + r)
    return sim


# voxels: 6,144 is the largest lattice of the one-block form; ranges of 1 .. 128 words above it
@pytest.mark.parametrize("res", [(16, 16, 24), (17, 19, 20), (40, 41, 37), (97, 31, 33), (1, 80, 81), (6200, 1, 1)])
@pytest.mark.parametrize("K", [4, 8, 11, 16])
def test_range_edges(orc, res, K):
    v = int(np.prod(res))
    sim = crowded_model(res=res, K=K, counts=(v // 8, v // 9, v // 20))
    assert_same(*run_pair(orc, sim, 12, chunks=3))


@pytest.mark.parametrize("reservoir,transition", [(False, False), (True, False), (False, True)])
def test_regions_in_launches(orc, reservoir, transition):
    sim = multi_region_model(res=(24, 23, 25), K=16, counts=(400, 300, 200, 100), reservoir=reservoir, transition=transition)
    assert_same(*run_pair(orc, sim, 60, chunks=2))


@pytest.mark.parametrize("res", [(16, 16, 16), (25, 24, 23)])
@pytest.mark.parametrize("K", [4, 8, 16])
def test_contended_frames(orc, res, K):
    v = int(np.prod(res))
    sim = crowded_model(res=res, K=K, counts=(v * K // 4, v * K // 4, v * K // 4))
    ref, gpu = run_pair(orc, sim, 5)
    assert_same(ref, gpu)
    assert gpu[4][2] > 0  # frames resolved in serial order


@pytest.mark.parametrize("res", [(15, 16, 17), (25, 24, 23)])
@pytest.mark.parametrize("K", [8, 16])
def test_voxels_that_are_not_their_slots(orc, res, K):
    """Uploaded occupancies and counts that differ from the slots, slots with holes; the state is read
    back and put in again half way."""
    v = int(np.prod(res))
    sim = multi_region_model(res=res, K=K, counts=(408, 340, 272, 204))  # the shell has a fixed size
    args = oracle_args(sim)
    s, o, c, st = ref_state(sim)
    S1 = len(st)
    rng = np.random.default_rng(9)
    s, c = s.reshape(v, K), c.reshape(v, S1)
    holes = rng.choice(v, v // 6, replace=False)
    s[holes] = np.roll(s[holes], 2, axis=1)
    some = rng.choice(v, v // 9, replace=False)
    c[some, rng.integers(1, S1, some.size)] += rng.integers(0, 3, some.size).astype(np.int32)
    c[rng.choice(v, v // 9, replace=False), 0] = 3
    odd = rng.choice(v, v // 9, replace=False)
    o[odd] = np.minimum(o[odd] + rng.integers(0, 2, odd.size).astype(np.uint32), K)
    s, c = s.reshape(-1), c.reshape(-1)
    st = c.reshape(v, S1).sum(0).astype(np.int32)
    it = itime_schedule(30, 31)
    ref = orc.ref_run(*args, orc.RefState(s.copy(), o.copy(), c.copy(), st.copy()), it, mode=1, threads=8)
    sim.prepare_for_gpu(RNG_REFERENCE, 0)
    sim.set_lattice(s, o, c)
    sim.step(it[:13])
    before = sim.counts()
    sim.set_lattice(*sim.get_lattice())
    assert np.array_equal(sim.counts()[1:], sim.get_lattice()[2].reshape(v, S1).sum(0)[1:])
    sim.step(it[13:])
    gs, go, gc = sim.get_lattice()
    assert np.array_equal(gs, ref.slots), np.flatnonzero(gs != ref.slots)[:10]
    assert np.array_equal(go, ref.occ)
    assert np.array_equal(gc, ref.conc)
    assert before.shape == (S1,)


@pytest.mark.parametrize("res", [(14, 15, 16), (25, 24, 23)])
def test_counts_below_zero(orc, res):
    """A + A -> B counts a lone A twice (its propensity is the product of counts) and takes two: the count
    falls to -1 and the occupancy, as a 32-bit word, to its largest value, which no slots show (the oracle's
    serial form: its parallel one adds arrivals to the occupancy in 32 bits)."""
    v = int(np.prod(res))
    D = 1e-12
    sim = Simulation(LatticeParams([r * LAM for r in res], list(res), configs.stable_tau(D), LAM, 8))
    sim.seed_placement(2)
    sim.set_diffusion_rate("background", D)
    sim.prepare_regions()
    for n in "AB":
        sim.add_particle_count(n, "background", v // 5, True, False)
    sim.set_diffusion_rate("background", D)
    sim.add_reaction(["A", "A"], ["B"], 900.0)
    sim.add_reaction(["B"], ["A"], 500.0)
    args = oracle_args(sim)
    it = itime_schedule(40, 987654321)
    ref = orc.ref_run(*args, orc.RefState(*ref_state(sim)), it, mode=0)
    sim.prepare_for_gpu(RNG_REFERENCE, 0)
    sim.step(it[:20])
    sim.step(it[20:])
    gs, go, gc = sim.get_lattice()
    assert np.array_equal(gs, ref.slots), np.flatnonzero(gs != ref.slots)[:10]
    assert np.array_equal(go, ref.occ)
    assert np.array_equal(gc, ref.conc)
    assert np.array_equal(sim.counts(), ref.stat.astype(np.int64))
    for k in (0, 1, 3, 4):  # the serial form does not count frames resolved in serial order
        assert sim.diagnostics()[k] == ref.diag[k], k
    assert ref.conc.min() < 0


# 3 bits of the last mask word, a full word, words more, and rows of 130 and 255 species (no shared tables)
@pytest.mark.parametrize("species,reactions", [(3, 31), (6, 32), (9, 63), (9, 64), (20, 97), (130, 40), (255, 99)])
@pytest.mark.parametrize("res", [(12, 13, 14), (21, 20, 19)])
def test_reaction_tables(orc, species, reactions, res):
    sim = network(res, 16, species, reactions, max(2, 1500 // species))
    ref, gpu = run_pair(orc, sim, 15, chunks=2)
    assert_same(ref, gpu)
    assert ref.diag[4] > 0
