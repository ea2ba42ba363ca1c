"""A form that the rule wants and the device has no room for: a handle whose lists no longer hold its particles goes on
in the tile pipeline, any other handle in the form that it has, and every frame is the oracle's (integer state: the
tolerance is zero).  The want of room comes from the hook cs_debug_refuse_tiling."""
import numpy as np
import pytest

from cell_simulation_gb300 import CellsimError, RNG_PHILOX
from tests.test_default_rule_gpu import RESIDENT, STREAM, form, mixed, tiles
from tests.test_growing_lists_gpu import growing, same, started
from tests.test_new_forms_gpu import in_place
from tests.test_prod_gpu import oracle_prod

pytestmark = pytest.mark.gpu

NO_ROOM = 8  # CS_ERR_CAPACITY


def stepped(mk, K, refuse, calls):
    sim = started(mk, K)
    if refuse is not None:
        sim.debug_refuse_tiling(refuse, NO_ROOM)
        with pytest.raises(CellsimError):
            sim.set_tiling(refuse)
    for n in calls:
        sim.step_philox(n, 7)
    return sim


@pytest.mark.parametrize("K", [8, 16])
@pytest.mark.parametrize("res,calls,goes_on", [
    ((20, 20, 20), (30,), None),           # lists, then the stream's turn: the tile pipeline
    ((20, 20, 20), (10, 20), None),
    ((20, 20, 20), (10, 20, 2), None),
    ((10, 9, 20), (48,), RESIDENT),        # lists, the resident form, then another's turn: the resident form
    ((10, 9, 20), (10, 20, 18), RESIDENT),
])
def test_outgrown_lists(orc, K, res, calls, goes_on):
    """The last form is found with a handle that has room."""
    mk, frames = growing(K, res), sum(calls)
    free = stepped(mk, K, None, calls)
    want = oracle_prod(orc, mk(), frames, seed=7)
    same(free, want)
    after = free.get_tiling()
    assert form(after) == STREAM if goes_on is None else form(after) != goes_on
    sim = stepped(mk, K, after, calls)
    same(sim, want)
    assert sim.get_tiling() == tiles(K) if goes_on is None else form(sim.get_tiling()) == goes_on
    sim.debug_refuse_tiling(-1, NO_ROOM)
    sim.step_philox(9, 7)
    same(sim, oracle_prod(orc, mk(), frames + 9, seed=7))


@pytest.mark.parametrize("K", [8, 16])
def test_upload_of_many(K):
    """The resident form goes on where the in-place form has no room."""
    few, many = mixed((16, 16, 16), K, 100), mixed((16, 16, 16), K, 16000)
    outs = []
    for refuse in (False, True):
        sim = few()
        sim.prepare_for_gpu(RNG_PHILOX, 0)
        if refuse:
            sim.debug_refuse_tiling(in_place(K), NO_ROOM)
        sim.set_lattice(many().get_lattice()[0])
        sim.step_philox(7, 3)
        sim.step_philox(300, 3)
        outs.append((sim.get_lattice()[0], sim.counts(), sim.diagnostics()[:4]))
        assert form(sim.get_tiling()) == RESIDENT if refuse else sim.get_tiling() == in_place(K)
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
