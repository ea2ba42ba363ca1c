"""Long step calls.  A call whose particles cannot outgrow the handle's form only enqueues its frames, as short ones
do; one whose particles can, through the dissociation of a complex, ends with the lattice of any other form."""
import time

import numpy as np
import pytest

from cell_simulation_gb300 import RNG_PHILOX
from tests.test_default_rule_gpu import LISTS, RESIDENT, form
from tests.test_new_forms_gpu import in_place, one_region

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,want", [((64, 64, 1), RESIDENT), ((40, 40, 40), LISTS)])
def test_returns_before_its_frames_have_run(res, want):
    """A + B <-> C from A and B alone: no more particles than at the start, whatever happens.  The call takes some
    100 ms on the device; a quarter of that is left for its launches."""
    sim = one_region(res, 8, (200, 200, 0), (30.0, 10.0, 0.0))
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    assert form(sim.get_tiling()) == want
    sim.step_philox(4096, 7)
    sim.synchronize()
    t0 = time.perf_counter()
    sim.step_philox(16384, 7)
    t1 = time.perf_counter()
    sim.synchronize()
    t2 = time.perf_counter()
    assert form(sim.get_tiling()) == want
    assert t1 - t0 < 0.25 * (t2 - t0), (t1 - t0, t2 - t0)
    assert 200 <= sim.counts().sum() <= 400


@pytest.mark.parametrize("K,res,particles", [(8, (40, 40, 40), 500), (16, (40, 40, 40), 250), (8, (64, 64, 1), 1000)])
def test_complexes_fall_apart(K, res, particles):
    """C -> A + B from C alone doubles the particles."""
    outs = []
    for tiling in (None, in_place(K)):
        sim = one_region(res, K, (0, 0, particles), (0.001, 200.0, 0.0))
        sim.prepare_for_gpu(RNG_PHILOX, 0)
        if tiling is not None:
            sim.set_tiling(tiling)
        sim.step_philox(3000, 7)
        outs.append((sim.get_lattice()[0], sim.counts(), sim.diagnostics()[:4]))
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
    assert outs[0][1].sum() > 1.9 * particles
