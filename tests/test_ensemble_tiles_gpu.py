"""Ideal steps of ensembles left untuned, at the sizes where the tile and the
chunk that creation chooses change (few and many replicas, sides that 32 x 8 or
16 x 16 tiles cover better, chunks that do not divide the side evenly, TMA
replicas alone and beside others), against single lattices: the same arithmetic
compiled into another kernel, 1e-13 per site as for every tuned ensemble."""
import numpy as np
import pytest

from lgvtest import rand_state, site_rel_err
from test_ensemble_gpu import IDEAL, make, singles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [[4, 6], [20] * 3, [48, 48], [24] * 32, [34, 18, 50], [32, 64, 90], [48] * 14, [32] * 40])
def test_untuned_ideal_step(lgv, sides):
    specs = [(N, 40 + i, 0.003) for i, N in enumerate(sides)]
    L, lib, e = make(lgv, specs)
    try:
        states = [rand_state(N, i) for i, N in enumerate(sides)]
        for r, u in enumerate(states):
            L.check(lib.lgv_ensemble_set_state(e, r, L.ptr(u)), "set_state")
        L.check(lib.lgv_ensemble_step(e, IDEAL, 1, 1, 0.04, 0.0, 2), "ensemble_step")
        pick = sorted({0, len(sides) // 2, len(sides) - 1})
        want = singles(lgv, [specs[r] for r in pick], [states[r] for r in pick], [(IDEAL, 0.04, 0.0, 2)])
        for r, w in zip(pick, want):
            got = np.empty_like(w)
            L.check(lib.lgv_ensemble_get_state(e, r, L.ptr(got)), "get_state")
            assert site_rel_err(got, w) <= 1e-13, f"replica {r} of {sides}"
    finally:
        lib.lgv_ensemble_destroy(e)
