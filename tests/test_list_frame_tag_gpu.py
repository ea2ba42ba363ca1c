"""A call of more than 65,536 frames in the list form, bit for bit against the oracle.  A list entry caches the
random block of its voxel under the low 16 bits of the frame number, and an entry that empties stays in the
list while most entries are occupied.  Here movers leave the plane x = 0 in the first frames and come back
about once in 65,536; with this seed one comes back to a voxel exactly 65,536 frames after the voxel's block
was last computed, and its next move depends on which frame's block is used."""
import numpy as np
import pytest

from cell_simulation_gb300 import RNG_PHILOX, configs
from cell_simulation_gb300.simulation import LatticeParams, RegionType, Simulation
from tests.helpers import LAM
from tests.test_new_forms_gpu import lists
from tests.test_prod_gpu import oracle_prod

pytestmark = pytest.mark.gpu

SEED, FRAMES = 204, 65536 + 24


def model():
    """One mover in every voxel of the plane x = 0, one immobile particle in every voxel of the plane x = 1, where
    movers do not move but back (with probability 2^-16 per frame)."""
    res, K = (2, 300, 2), 8
    tau = configs.stable_tau(1e-12)
    rate = lambda p: p * LAM * LAM / tau  # of probability p per frame
    sim = Simulation(LatticeParams([r * LAM for r in res], list(res), tau, LAM, K))
    sim.add_region(RegionType.Cube("b", [LAM, 0, 0], [r * LAM for r in res]), 0.0)
    sim.prepare_regions()
    for name in ("mover", "keeper"):
        sim.add_particle_count(name, "background", 0, True, False)
    for region in ("background", "b"):
        sim.set_diffusion_rate(region, 0.0)
    sim.set_diffusion_rate_particle("mover", "background", rate(0.3))
    sim.set_transition_rate_particle("mover", "background", "b", rate(0.3))
    sim.set_transition_rate_particle("mover", "b", "background", rate(2.0 ** -16))
    sim.add_reaction(["mover"], ["keeper"], 1e-12)
    V = int(np.prod(res))
    slots = np.zeros((V, K), np.uint32)
    slots[:V // 2, 0] = 1
    slots[V // 2:, 0] = 2
    sim.set_lattice(slots.reshape(-1))
    return sim


def test_frame_tags_of_a_long_call(orc):
    want_s, want_c, _ = oracle_prod(orc, model(), FRAMES, seed=SEED)
    sim = model()
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    sim.set_tiling(lists(8))
    sim.step_philox(FRAMES, SEED)
    got_s, got_c = sim.get_lattice()[0].astype(np.uint8), sim.counts()
    assert sim.get_tiling() == lists(8)  # the particles fit throughout
    assert np.array_equal(got_s, want_s), np.flatnonzero(got_s != want_s)[:8]
    assert np.array_equal(got_c, want_c)
