"""The list form (one block per replicate keeps the list of its occupied voxels) and the in-place sweep
stream of the production step, bit for bit against the oracle (integer state: the tolerance is zero), at
the sizes where they can go wrong: rows of one word, of a full word, of one voxel more and of several
words; edges of length 1; crowded voxels and refused moves; regions that end inside a word; reservoirs
(in place) and their refusal (lists); a replicate whose particles outgrow its list within a call, which
finishes over the whole lattice; calls of one and of many frames; switches between the forms, each of
which keeps the lattice in a layout of its own; and the view read from those layouts."""
import numpy as np
import pytest

from cell_simulation_gb300 import CellsimError, Ensemble, RNG_PHILOX, configs, tiling_kinds, tiling_variants
from cell_simulation_gb300.simulation import LatticeParams, Simulation
from tests.helpers import LAM, crowded_model, multi_region_model
from tests.test_prod_gpu import gpu_prod, oracle_prod

pytestmark = pytest.mark.gpu


def lists(K):
    return next(i for i, (t, k) in enumerate(zip(tiling_variants(), tiling_kinds())) if t[0] == K and k[0] == 4)


def in_place(K):
    return next(i for i, (t, k) in enumerate(zip(tiling_variants(), tiling_kinds()))
                if t[0] == K and k[0] == 2 and t[1] == 2)


def one_region(res, K, counts, rates, seed=5):
    """A, B, C on one region: A + B -> C, C -> A + B, A -> A + A at the given rates."""
    D = 1e-12
    sim = Simulation(LatticeParams([r * LAM for r in res], list(res), configs.stable_tau(D), LAM, K))
    sim.seed_placement(seed)
    sim.prepare_regions()
    sim.set_diffusion_rate("background", D)
    for n, k in zip("ABC", counts):
        sim.add_particle_count(n, "background", k, True, False)
    sim.set_diffusion_rate("background", D)
    sim.add_reaction(["A", "B"], ["C"], rates[0])
    sim.add_reaction(["C"], ["A", "B"], rates[1])
    if rates[2]:
        sim.add_reaction(["A"], ["A", "A"], rates[2])
    return sim


def check(orc, mk, n, seed, tiling, chunks=(1, 3)):
    want_s, want_c, want_d = oracle_prod(orc, mk(), n, seed=seed)
    for ch in chunks:
        got_s, got_c, got_d = gpu_prod(mk(), n, seed, tiling=tiling, chunks=ch)
        assert np.array_equal(got_s, want_s), (ch, np.flatnonzero(got_s != want_s)[:8])
        assert np.array_equal(got_c, want_c), ch
        assert np.array_equal(got_d[:4], want_d[:4]), (ch, got_d, want_d)
    return want_d


SIZES = [(5, 4, 31), (4, 6, 32), (3, 5, 33), (6, 1, 64), (1, 7, 65), (9, 8, 1), (2, 2, 97)]


@pytest.mark.parametrize("form", [lists, in_place])
@pytest.mark.parametrize("K", [8, 16])
@pytest.mark.parametrize("res", SIZES)
def test_word_edges_match_oracle(orc, form, K, res):
    v = int(np.prod(res))
    mk = lambda: one_region(res, K, (v // 12 + 1, v // 12 + 1, v // 20), (300.0, 60.0, 0.0))
    check(orc, mk, 12, 91, form(K))


@pytest.mark.parametrize("K", [8, 16])
@pytest.mark.parametrize("particles", [128, 129, 350, 351, 600])
def test_threads_of_a_list_block(orc, K, particles):
    """Both sides of the lines between 256, 512 and 768 threads."""
    check(orc, lambda: one_region((11, 13, 17), K, (particles - particles // 2, particles // 2, 0), (300.0, 60.0, 0.0)),
          12, 57, lists(K))


@pytest.mark.parametrize("form", [lists, in_place])
@pytest.mark.parametrize("K", [8, 16])
def test_regions_match_oracle(orc, form, K):
    """Regions that end inside words, transitions between them."""
    mk = lambda: multi_region_model(res=(11, 12, 45), K=K, counts=(60, 70, 50, 30), transition=True)
    d = check(orc, mk, 20, 17, form(K), chunks=(1, 20))
    assert d[0] > 0


def test_crowded_voxels_match_oracle(orc):
    """Nearly full voxels: moves refused for lack of room, in both forms (K = 8) and with more voxels on the
    general path than the in-place form keeps in shared memory (K = 16, one long column per block)."""
    check(orc, lambda: crowded_model(res=(6, 5, 7), K=8, counts=(300, 280, 240)), 25, 5, lists(8))
    check(orc, lambda: crowded_model(res=(6, 5, 7), K=8, counts=(420, 380, 240)), 25, 5, in_place(8))
    check(orc, lambda: crowded_model(res=(40, 9, 33), K=16, counts=(9000, 8000, 6000)), 6, 8, in_place(16), chunks=(2,))


def test_long_lines_match_oracle(orc):
    """Lines of 1024 voxels along x and along y (the in-place form's longest) and rows of 32 words."""
    check(orc, lambda: one_region((1024, 2, 3), 8, (300, 300, 50), (300.0, 60.0, 0.0)), 4, 3, in_place(8), chunks=(2,))
    check(orc, lambda: one_region((2, 1024, 3), 16, (300, 300, 50), (300.0, 60.0, 0.0)), 4, 3, in_place(16), chunks=(2,))
    check(orc, lambda: one_region((2, 3, 1024), 8, (300, 300, 50), (300.0, 60.0, 0.0)), 4, 3, in_place(8), chunks=(2,))


@pytest.mark.parametrize("K", [8, 16])
def test_reservoirs(orc, K):
    mk = lambda: multi_region_model(res=(9, 8, 40), K=K, counts=(60, 50, 40, 30), reservoir=True)
    check(orc, mk, 20, 23, in_place(K))
    sim = mk()
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    before = sim.get_tiling()
    with pytest.raises(CellsimError):
        sim.set_tiling(lists(K))
    assert sim.get_tiling() == before


@pytest.mark.parametrize("K", [8, 16])
def test_outgrown_list_finishes_over_the_lattice(orc, K):
    """A -> A + A multiplies the particles past the list's room within one call: the block finishes the call
    voxel by voxel, and so do the calls enqueued before the host can know; the first call made after the
    results were read takes another form.  Every frame is the oracle's."""
    mk = lambda: one_region((10, 9, 20), K, (60, 20, 0), (30.0, 10.0, 500.0))
    want_s, want_c, want_d = oracle_prod(orc, mk(), 46, seed=7)
    assert want_c.sum() > 800  # past 704 entries for them and their moves
    sim = mk()
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    sim.set_tiling(lists(K))
    for n in (40, 5, 1):
        sim.step_philox(n, 7)
    assert np.array_equal(sim.get_lattice()[0].astype(np.uint8), want_s)
    assert np.array_equal(sim.counts(), want_c)
    assert np.array_equal(sim.diagnostics()[:4], want_d[:4])
    sim.step_philox(1, 7)
    assert sim.get_tiling() != lists(K)
    want_s, want_c, _ = oracle_prod(orc, mk(), 47, seed=7)
    assert np.array_equal(sim.get_lattice()[0].astype(np.uint8), want_s)
    assert np.array_equal(sim.counts(), want_c)


def test_layouts_hand_over(orc):
    """List, in-place, resident and stream frames in one run, with uploads, read-backs and seed changes."""
    mk = lambda: multi_region_model(res=(9, 8, 40), K=16, counts=(70, 60, 50, 40))
    want_s, want_c, _ = oracle_prod(orc, mk(), 40, seed=909)
    sim = mk()
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    kinds = tiling_kinds()
    stream = next(i for i, (t, k) in enumerate(zip(tiling_variants(), kinds)) if t[0] == 16 and k[0] == 2)
    res = next(i for i, (t, k) in enumerate(zip(tiling_variants(), kinds)) if t[0] == 16 and k[0] == 3)
    for i, (ti, n) in enumerate(((lists(16), 3), (in_place(16), 4), (lists(16), 1), (res, 5), (in_place(16), 3),
                                 (stream, 3), (lists(16), 2), (stream, 4), (in_place(16), 1), (res, 2),
                                 (lists(16), 5), (in_place(16), 7))):
        sim.set_tiling(ti)
        sim.step_philox(n, 909)
        view = sim.render_view()       # from the form's own layout
        slots = sim.get_lattice()[0]   # writes the slots
        assert np.array_equal(view, sim.render_view()), i
        if i % 4 == 1:
            sim.set_lattice(slots)
    assert np.array_equal(sim.get_lattice()[0].astype(np.uint8), want_s)
    assert np.array_equal(sim.counts(), want_c)


@pytest.mark.parametrize("K", [8, 16])
@pytest.mark.parametrize("batched", [True, False])
def test_ensemble_of_lists_and_in_place_agree(K, batched):
    """Uneven replicates, stepped batched and replicate by replicate, read back between calls."""
    tmpl = configs.c4_ensemble_template(K=K)
    res = np.array([[9, 9, 33], [12, 3, 12], [1, 7, 64], [16, 16, 16], [5, 5, 5]], np.uint32)
    out = []
    for form in (lists, in_place):
        ens = Ensemble(tmpl, res, np.array([11, 22, 33, 44, 55], np.uint64), np.array([0.5, 1.0, 1.7, 2.0, 1.0], np.float32),
                       np.array([0, 40, 40, 5], np.uint32))
        ens.set_tiling(form(K))
        for n in (1, 9, 10):
            ens.step(n, batched=batched)
            s, c = ens.slots(), ens.counts()
        out.append((s, c))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("res,counts,form", [
    ((56, 56, 56), (7000, 7000, 336), (2, 0)),     # 14,336 particles: fused stream
    ((56, 56, 56), (9000, 9000, 337), (2, 2)),     # more, and more than one in ten voxels: in place
    ((24, 24, 24), (2500, 2500, 500), (2, 0)),     # two fifths of a particle per voxel: fused stream
    ((24, 24, 24), (2500, 2500, 600), (2, 2)),     # more: in place
    ((110, 110, 110), (9000, 9000, 2000), (2, 0)), # at most one in ten voxels: fused stream
    ((136, 136, 136), (900, 900, 200), (2, 2)),    # more than 2.5 M voxels: in place
    ((64, 8, 8), (200, 200, 200), (3, 0)),         # few voxels, up to 640 particles: resident
    ((64, 8, 8), (200, 200, 300), (2, 0)),         # more: fused stream
    ((9, 9, 9), (200, 200, 50), (3, 0)),           # few particles, few voxels: resident
    ((30, 30, 30), (110, 100, 46), (4, 0)),        # few particles (256 at K = 16): lists
    ((30, 30, 30), (111, 100, 46), (2, 0)),        # more: fused stream
])
def test_default_form_matches_general_path(res, counts, form):
    """The form that a new handle takes on both sides of each line of the rule, against the column tiles
    (the general path), bit for bit, in calls of one frame, of a part and of more than a captured graph."""
    def frames(tiling):
        sim = one_region(res, 16, counts, (300.0, 60.0, 0.0))
        sim.prepare_for_gpu(RNG_PHILOX, 0)
        kind, bx = tiling_kinds()[sim.get_tiling()]
        ty = tiling_variants()[sim.get_tiling()][1]
        if tiling is not None:
            sim.set_tiling(tiling)
        for n in (1, 3, 11):
            sim.step_philox(n, 77)
        return (kind, bx if kind == 1 else ty if kind == 2 else 0), sim.get_lattice()[0], sim.counts(), sim.diagnostics()[:4]
    got = frames(None)
    want = frames(0)
    assert got[0] == form
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[2], want[2])
    assert np.array_equal(got[3], want[3])
