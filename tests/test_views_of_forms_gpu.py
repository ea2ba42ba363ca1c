"""Region and reservoir views after frames of the forms that keep the lattice in a layout of their own: the same
volumes as from the column tiles, the species view and the slots as well afterwards, and no time spent on writing
slots that they do not read."""
import time

import numpy as np
import pytest
import torch

from cell_simulation_gb300 import RNG_PHILOX, configs, native, tiling_kinds, tiling_variants
from tests.helpers import multi_region_model
from tests.test_new_forms_gpu import in_place, lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [lists, in_place])
def test_views_of_forms(form):
    mk = lambda: multi_region_model(res=(9, 8, 40), K=16, counts=(60, 50, 40, 30), reservoir=form is in_place)
    out = []
    for tiling in (form(16), next(i for i, t in enumerate(tiling_variants()) if t[0] == 16 and tiling_kinds()[i][0] == 0)):
        sim = mk()
        sim.prepare_for_gpu(RNG_PHILOX, 0)
        sim.set_tiling(tiling)
        got = []
        for n in (1, 6):
            sim.step_philox(n, 9)
            got += [sim.render_view(1), sim.render_view(2), sim.render_view(1, 2, 5), sim.render_view(0, 1, 3), sim.render_view(0)]
            sim.step_philox(2, 9)
            got += [sim.render_view(2), sim.get_lattice()[0], sim.counts()]
        out.append(got)
    for i, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), i


def test_region_view_writes_no_slots():
    """Right after frames, and again with nothing changed."""
    sim = configs.c3_multi_region().sim
    sim.prepare_for_gpu(RNG_PHILOX, 0)
    sim.set_tiling(in_place(16))
    buf = torch.empty(256 ** 3, dtype=torch.float32, device="cuda")
    first, again = [], []
    for _ in range(20):
        sim.step_philox(1, 5)
        sim.synchronize()
        for times in (first, again):
            t = time.perf_counter()
            native.check(native.load().cs_render_view(sim._h, 1, 0, 0, None, buf.data_ptr()))
            times.append(time.perf_counter() - t)
    assert np.median(first) < 1.25 * np.median(again), (np.median(first), np.median(again))
