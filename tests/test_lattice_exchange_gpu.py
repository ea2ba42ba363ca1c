"""Uploads and read-backs of a production handle's lattice against the same conversion in numpy (integers:
the tolerance is zero): slots with holes come back with the particles first, occupancy and counts follow,
reservoir voxels count one of their species; one voxel, odd shapes, and lattices of exactly one piece of
the workspace (1,048,576 voxels) and of more."""
import numpy as np
import pytest

from cell_simulation_gb300 import CellsimError, RNG_PHILOX
from tests.helpers import crowded_model, multi_region_model

pytestmark = pytest.mark.gpu


def packed(slots, V, K, S1):
    s = slots.reshape(V, K)
    order = np.argsort(s == 0, axis=1, kind="stable")  # particles first, in their order
    out = np.take_along_axis(s, order, axis=1)
    conc = np.zeros((V, S1), np.int32)
    for q in range(1, S1):
        conc[:, q] = (s == q).sum(1)
    return out.reshape(-1), (s != 0).sum(1).astype(np.uint32), conc


@pytest.mark.parametrize("res,K", [((1, 1, 1), 8), ((7, 5, 9), 16), ((13, 11, 17), 8), ((13, 11, 17), 16), ((9, 20, 31), 16),
                                   ((128, 128, 64), 8), ((128, 129, 64), 8), ((103, 104, 101), 16)])
def test_upload_and_read_back(res, K):
    V = int(np.prod(res))
    sim = crowded_model(res=res, K=K, counts=(1, 1, 1))
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    rng = np.random.default_rng(V + K)
    for fill in (0.0, 0.3, 1.0):
        slots = np.where(rng.random(V * K) < fill, rng.integers(1, 4, V * K), 0).astype(np.uint32)
        sim.set_lattice(slots)
        want_s, want_o, want_c = packed(slots, V, K, 4)
        s, o, c = sim.get_lattice()
        assert np.array_equal(s, want_s)
        assert np.array_equal(o, want_o)
        assert np.array_equal(c.reshape(V, 4), want_c)
        assert np.array_equal(sim.counts()[1:], want_c.sum(0)[1:])


def test_reservoirs_and_refusals():
    sim = multi_region_model(res=(12, 10, 14), K=8, reservoir=True)
    s0, o0, c0 = sim.get_lattice()  # the host's model
    V, S1 = 1680, c0.size // 1680
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    s, o, c = sim.get_lattice()
    want_s, want_o, want_c = packed(s0, V, 8, S1)
    res = sim.tables().reservoir.reshape(-1).astype(np.int64)
    at = np.flatnonzero(res)
    want_c[at, res[at]] = 1
    assert at.size > 0
    assert np.array_equal(s, want_s) and np.array_equal(o, want_o) and np.array_equal(c.reshape(V, S1), want_c)
    free = packed(s0, V, 8, S1)[2].sum(0)
    assert np.array_equal(sim.counts()[1:], (free + np.bincount(res, minlength=S1))[1:])
    bad = s0.copy()
    bad[5] = S1
    with pytest.raises(CellsimError):
        sim.set_lattice(bad)
    assert np.array_equal(sim.get_lattice()[0], s)  # refused before anything changed
