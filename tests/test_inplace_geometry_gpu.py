"""The in-place form where a block has more than a line: the benchmark's cells (256 cubed: lines of four words per
thread, 192 cubed: two, 128 cubed: one), lines between one and two words per thread, and crowded lattices whose units
list more voxels than fit in one list, on the simple and the general path and among the decisions.  Bit for bit
against the oracle (integer state: the tolerance is zero)."""
import numpy as np
import pytest

from cell_simulation_gb300 import configs
from tests.helpers import crowded_model
from tests.test_bench_geometry_gpu import _check, _gpu_frames, _oracle_frames
from tests.test_new_forms_gpu import check, in_place, one_region

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,frames,seed", [("c3", 4, 0xC0FFEE), ("c5", 4, 4242), ("c2", 6, 2024)])
def test_benchmark_cells(orc, cell, frames, seed):
    mk = {"c3": configs.c3_multi_region, "c5": configs.c5_stiff, "c2": configs.c2_single_cell}[cell]
    want = _oracle_frames(orc, mk().sim, frames, seed=seed)
    assert want[2][0] > 0
    _check(_gpu_frames(mk().sim, frames, seed, in_place(16)), want, cell)


@pytest.mark.parametrize("K", [8, 16])
@pytest.mark.parametrize("res", [(257, 3, 35), (300, 2, 33), (512, 2, 31), (513, 2, 31), (3, 257, 35), (2, 400, 33), (2, 512, 31)])
def test_line_lengths(orc, K, res):
    """Lines of just past one, of two and of just past two words per thread, along x and along y."""
    v = int(np.prod(res))
    mk = lambda: one_region(res, K, (v // 12, v // 12, v // 20), (300.0, 60.0, 0.0))
    check(orc, mk, 6, 91, in_place(K), chunks=(2,))


@pytest.mark.parametrize("K,res,per_voxel", [
    (8, (128, 128, 96), 0.3),    # units of some 100 to 200 words: about 1,000 movers a line, most of them simple
    (8, (128, 128, 96), 2.0),    # nearly every voxel on the general path, refused moves
    (16, (100, 130, 128), 5.0),  # ... with K = 16
    (16, (160, 40, 160), 0.8),
])
def test_units_of_many_voxels(orc, K, res, per_voxel):
    v = int(np.prod(res) * per_voxel)
    mk = lambda: crowded_model(res=res, K=K, counts=(v // 3, v // 3, v - 2 * (v // 3)))
    d = check(orc, mk, 2, 8, in_place(K), chunks=(1,))
    assert d[0] > 0
