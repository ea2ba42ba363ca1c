"""The autotuner's remembered choice belongs to a population: a handle of the same shapes with many times the
particles, or another precision, is timed by itself; one like the first takes the remembered choice.  A tune
that times the variants takes thousands of times as long as one that remembers."""
import time

import pytest

from cell_simulation_gb300 import PREC_FP64, RNG_PHILOX
from tests.test_new_forms_gpu import one_region

pytestmark = pytest.mark.gpu


def tuned(counts, precision=None, frames=0):
    """((variant, ms per frame), seconds that the tune took)"""
    sim = one_region((27, 26, 25), 16, counts, (30.0, 10.0, 500.0 if frames else 0.0))
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    if precision is not None:
        sim.set_precision(precision)
    if frames:
        sim.step_philox(frames, 3)
    sim.synchronize()
    t = time.perf_counter()
    choice = sim.autotune(frames_per_trial=2)
    return choice, time.perf_counter() - t


def test_remembered_choice_belongs_to_the_population():
    few, many = (1000, 1000, 40), (20000, 20000, 0)
    first, _ = tuned(few)
    again, remembered = tuned(few)
    assert again == first
    crowded, s = tuned(many)
    assert s > 10 * remembered
    assert tuned(many)[0] == crowded
    _, s = tuned(few, PREC_FP64)
    assert s > 10 * remembered


def test_population_that_the_host_has_not_read():
    """The particles count as they are, not as the host last saw them."""
    start = (900, 900, 40)
    tuned(start, frames=1)
    _, remembered = tuned(start, frames=1)
    _, s = tuned(start, frames=60)
    assert s > 10 * remembered
