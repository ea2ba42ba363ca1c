"""The form that the default rule takes on both sides of the lines that decide between the fused sweep stream and
the in-place form on crowded, thin, long and many lattices, and how a handle of the rule's choice follows its
population and the length of its calls.  Every run is compared bit for bit with the column tiles (the general
path) or the oracle."""
import numpy as np
import pytest

from cell_simulation_gb300 import Ensemble, RNG_PHILOX, configs, tiling_kinds, tiling_variants
from cell_simulation_gb300.simulation import LatticeParams, Simulation
from tests.helpers import LAM, multi_region_model
from tests.test_new_forms_gpu import in_place, lists, one_region
from tests.test_prod_gpu import oracle_prod

pytestmark = pytest.mark.gpu

STREAM, IN_PLACE, RESIDENT, LISTS = (2, 0), (2, 2), (3, 0), (4, 0)


def form(handle_tiling):
    kind, ty = tiling_kinds()[handle_tiling][0], tiling_variants()[handle_tiling][1]
    return kind, ty if kind == 2 else 0


def tiles(K):
    return next(i for i, (t, k) in enumerate(zip(tiling_variants(), tiling_kinds())) if t[0] == K and k[0] == 0)


def run(mk, K, tiling, calls, seed=77):
    sim = mk()
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    took = form(sim.get_tiling())
    if tiling is not None:
        sim.set_tiling(tiling)
    for n in calls:
        sim.step_philox(n, seed)
    out = took, sim.get_lattice()[0], sim.counts(), sim.diagnostics()[:4]
    sim.close()
    return out


def check(mk, K, want_form, calls=(1, 3)):
    got = run(mk, K, None, calls)
    assert got[0] == want_form
    want = run(mk, K, tiles(K), calls)
    for a, b in zip(got[1:], want[1:]):
        assert np.array_equal(a, b)


def mixed(res, K, particles):
    """A + B <-> C on one region, that many particles."""
    return lambda: one_region(res, K, (particles // 2, particles - particles // 2, 0), (300.0, 60.0, 0.0))


@pytest.mark.parametrize("res,K,particles,want", [
    ((96, 96, 7), 16, 38000, STREAM),          # fewer than 8 voxels per bitmap word
    ((96, 96, 8), 16, 38000, IN_PLACE),
    ((11, 512, 64), 8, 40000, STREAM),         # 22 Y blocks of 512 words
    ((12, 512, 64), 8, 40000, IN_PLACE),       # 24
    ((11, 510, 64), 8, 40000, IN_PLACE),       # 22 of 510 words
    ((24, 200, 32), 8, 336500, STREAM),        # 24 Y blocks, more than 14,000 particles each
    ((24, 200, 32), 8, 335500, IN_PLACE),      # fewer
    ((384, 384, 16), 8, 250000, STREAM),       # 4,608 groups, 16 voxels per word
    ((384, 384, 20), 8, 250000, IN_PLACE),     # 20 voxels per word
    ((152, 152, 152), 8, 4600000, STREAM),     # 3,952 groups times particles past 1.8e10
    ((152, 152, 152), 8, 4500000, IN_PLACE),
    ((140, 140, 140), 8, 228000, STREAM),      # up to 4.4 M voxels of one region: one particle in twelve voxels
    ((140, 140, 140), 8, 229000, IN_PLACE),
    ((140, 140, 140), 8, 20000, STREAM),       # ... and 20,000 particles
    ((140, 140, 140), 8, 19999, IN_PLACE),
    ((165, 165, 165), 8, 100000, IN_PLACE),    # more voxels
])
def test_lattices(res, K, particles, want):
    check(mixed(res, K, particles), K, want, calls=(1, 2) if particles > 10 ** 6 else (1, 3, 9))


@pytest.mark.parametrize("res,particles", [((64, 64, 1), 50), ((20, 20, 20), 100), ((33, 20, 40), 3000)])
def test_reactions_without_reactants(orc, res, particles):
    """Every voxel may react: in place, against the oracle."""
    def mk():
        sim = one_region(res, 16, (particles // 2, particles - particles // 2, 0), (300.0, 60.0, 0.0))
        sim.add_reaction([], ["A"], 2.0)
        return sim
    want = oracle_prod(orc, mk(), 9, seed=5)
    got = run(mk, 16, None, (1, 8), seed=5)
    assert got[0] == IN_PLACE
    assert np.array_equal(got[1].astype(np.uint8), want[0])
    assert np.array_equal(got[2], want[1])
    assert np.array_equal(got[3], want[2][:4])


@pytest.mark.parametrize("res,want", [((12, 10, 34), IN_PLACE), ((20, 30, 4), STREAM)])
def test_reservoirs(orc, res, want):
    """In place but where voxels per word are few."""
    mk = lambda: multi_region_model(res=res, K=16, counts=(60, 50, 40, 5), reservoir=True)
    ref = oracle_prod(orc, mk(), 12, seed=23)
    got = run(mk, 16, None, (1, 11), seed=23)
    assert got[0] == want
    assert np.array_equal(got[1].astype(np.uint8), ref[0])
    assert np.array_equal(got[2], ref[1])


@pytest.mark.parametrize("n,edge,particles,want", [
    (100, 30, 2000, IN_PLACE),       # 3,000 groups
    (101, 30, 2000, STREAM),         # more, in planes of 30 words
    (16, 90, 2000, IN_PLACE),        # many groups, planes of 270 words
    (16, 90, 126000, STREAM),        # more than 2 M particles
])
def test_replicates(n, edge, particles, want):
    tmpl = configs.c4_ensemble_template(K=8)
    res = np.full((n, 3), edge, np.uint32)
    init = np.array([0, particles // 2, particles - particles // 2, 0], np.uint32)
    out = []
    for tiling in (None, tiles(8)):
        ens = Ensemble(tmpl, res, np.arange(1, n + 1, dtype=np.uint64), np.linspace(0.5, 2.0, n).astype(np.float32), init)
        if tiling is not None:
            ens.set_tiling(tiling)
        for k in (1, 3):
            ens.step(k)
        out.append((ens.slots(), ens.counts(), ens.diagnostics()[:4]))
        if tiling is None:
            items = ens.info()[1]
            rows_per_group = 32 // -(-edge // 32)
            groups = n * edge * -(-edge // rows_per_group)
            assert (items == groups) == (want == STREAM), (items, groups)
        ens.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("K,particles", [(8, 400), (8, 401), (8, 900), (16, 640)])
def test_short_calls_of_a_resident_handle(K, particles):
    """Calls of one frame up to twenty, in the stream or in the resident form, one after another."""
    check(mixed((64, 64, 1), K, particles), K, RESIDENT, calls=(1, 1, 2, 5, 1, 20, 3, 1, 4, 2, 2))


@pytest.mark.parametrize("K", [8, 16])
def test_form_follows_an_upload(K):
    """A handle made with few particles takes the form of the lattice that is uploaded, and back; one whose variant
    was chosen keeps it."""
    few, many = mixed((16, 16, 16), K, 100), mixed((16, 16, 16), K, 16000)
    outs = []
    for tiling in (None, tiles(K), in_place(K)):
        sim = few()
        sim.prepare_for_gpu(RNG_PHILOX, 0)
        if tiling is not None:
            sim.set_tiling(tiling)
        seen = [sim.get_tiling()]
        got = []
        for mk in (many, few, many):
            sim.set_lattice(mk().get_lattice()[0])
            sim.step_philox(7, 3)
            seen.append(sim.get_tiling())
            got += [sim.get_lattice()[0], sim.counts()]
        outs.append(got)
        if tiling is None:
            assert [form(t) for t in seen] == [RESIDENT, IN_PLACE, RESIDENT, IN_PLACE]
        else:
            assert seen == [tiling] * 4
    for a, b, c in zip(*outs):
        assert np.array_equal(a, b) and np.array_equal(a, c)


def test_form_follows_a_population_that_grows(orc):
    """Grown within one long call, and within calls whose counts are read."""
    mk = lambda: one_region((64, 64, 1), 8, (20, 0, 0), (30.0, 10.0, 20.0))
    want = oracle_prod(orc, mk(), 2048, seed=7)
    assert want[1].sum() > 15000
    for calls in ((2048,), (256,) * 8):
        sim = mk()
        sim.prepare_for_gpu(RNG_PHILOX, 0)
        assert form(sim.get_tiling()) == RESIDENT
        for n in calls:
            sim.step_philox(n, 7)
            if len(calls) > 1:
                sim.counts()
        assert np.array_equal(sim.get_lattice()[0].astype(np.uint8), want[0])
        assert np.array_equal(sim.counts(), want[1])
        assert np.array_equal(sim.diagnostics()[:4], want[2][:4])
        assert form(sim.get_tiling()) == STREAM
