"""Ensembles stepped batched and replicate by replicate in turn, in odd and even numbers of frames: every form, and the
rule's choice, computes the lattices of the in-place form bit for bit (after an odd number of frames of the other
sort, the frames of the forms with work counters found no work left)."""
import numpy as np
import pytest

from cell_simulation_gb300 import Ensemble, configs, tiling_kinds, tiling_variants
from tests.test_new_forms_gpu import in_place, lists

pytestmark = pytest.mark.gpu

CALLS = [(5, True), (5, False), (1, True), (3, False), (2, True), (1, False), (1, False), (1, True), (4, False), (3, True)]


def of_kind(K, kind, ty=None):
    return [i for i, (t, k) in enumerate(zip(tiling_variants(), tiling_kinds()))
            if t[0] == K and k[0] == kind and (ty is None or t[1] == ty)]


def stepped(K, tiling, particles, res):
    n = len(res)
    ens = Ensemble(configs.c4_ensemble_template(K=K), res, np.arange(1, n + 1, dtype=np.uint64),
                   np.linspace(0.5, 2.0, n).astype(np.float32),
                   np.array([0, particles // 2, particles - particles // 2, 0], np.uint32))
    if tiling is not None:
        ens.set_tiling(tiling)
    out = []
    for frames, batched in CALLS:
        ens.step(frames, batched=batched)
        out += [ens.slots(), ens.counts()]
    out.append(ens.diagnostics()[:4])
    ens.close()
    return out


@pytest.mark.parametrize("K", [8, 16])
@pytest.mark.parametrize("particles", [60, 3000])
def test_every_form(K, particles):
    res = np.array([[9, 8, 11], [6, 10, 35], [13, 7, 16], [10, 6, 40], [11, 11, 21]], np.uint32)
    want = stepped(K, in_place(K), particles, res)
    forms = [None, of_kind(K, 0)[0], of_kind(K, 1)[0], of_kind(K, 1)[-1], of_kind(K, 3)[0]]
    forms += [of_kind(K, 2, 0)[i] for i in (0, -1)] + of_kind(K, 2, 1)[:1]
    if particles < 100:
        forms.append(lists(K))
    for tiling in forms:
        for i, (a, b) in enumerate(zip(stepped(K, tiling, particles, res), want)):
            assert np.array_equal(a, b), (tiling, i)
