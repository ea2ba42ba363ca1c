"""A tune in which a variant cannot be set up: the variant is no candidate when it does not fit, any other error
ends the tune, and either way the simulation has not advanced (the lattice, counts and diagnostics are those of
before, and the following frames are the oracle's)."""
import numpy as np
import pytest

from cell_simulation_gb300 import CellsimError, RNG_PHILOX, tiling_variants
from tests.helpers import multi_region_model
from tests.test_prod_gpu import oracle_prod

pytestmark = pytest.mark.gpu

LIMIT, DEVICE_STATUS = 3, 9


@pytest.mark.parametrize("status", [LIMIT, DEVICE_STATUS])
@pytest.mark.parametrize("which", [0, -1])
def test_failed_variant_leaves_the_state(orc, status, which):
    """which: the first and the last variant of this slot count."""
    res = (15, 13 + which, 41 + status)  # a shape that no other tune of this process has had
    mk = lambda: multi_region_model(res=res, K=16, counts=(90, 70, 50, 40))
    want_s, want_c, want_d = oracle_prod(orc, mk(), 12, seed=616)
    sim = mk()
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    sim.step_philox(4, 616)
    tiling, slots, counts, diag = sim.get_tiling(), sim.get_lattice()[0], sim.counts(), sim.diagnostics()
    bad = [i for i, t in enumerate(tiling_variants()) if t[0] == 16][which]
    sim.debug_refuse_tiling(bad, status)
    if status == LIMIT:
        idx, ms = sim.autotune(frames_per_trial=2)
        assert idx != bad and idx == sim.get_tiling() and ms > 0
    else:
        with pytest.raises(CellsimError):
            sim.autotune(frames_per_trial=2)
        assert sim.get_tiling() == tiling or tiling == bad  # the handle's own may be the one that is refused
    assert np.array_equal(sim.get_lattice()[0], slots)
    assert np.array_equal(sim.counts(), counts)
    assert np.array_equal(sim.diagnostics(), diag)
    sim.step_philox(8, 616)
    assert np.array_equal(sim.get_lattice()[0].astype(np.uint8), want_s)
    assert np.array_equal(sim.counts(), want_c)
    assert np.array_equal(sim.diagnostics()[:4], want_d[:4])
