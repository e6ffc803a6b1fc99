"""Euler-Maruyama steps of ensembles whose planes leave most of a block without a
site: replicas of 4^3 to 18^3, alone and beside one with full blocks, equal single
lattices to the last bit."""
import numpy as np
import pytest

from lgvtest import rand_state
from test_ensemble_gpu import EM, make, singles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [[4], [6, 4, 8], [10, 12], [14, 16, 18], [8, 34, 4]])
def test_planes_smaller_than_a_block(lgv, sides):
    specs = [(N, 90 + i, 0.006) for i, N in enumerate(sides)]
    L, lib, e = make(lgv, specs)
    try:
        states = [rand_state(N, 5 * N + i) for i, N in enumerate(sides)]
        for r, u in enumerate(states):
            L.check(lib.lgv_ensemble_set_state(e, r, L.ptr(u)), "set_state")
        L.check(lib.lgv_ensemble_step(e, EM, 1, 1, 0.01, 0.0, 5), "step")
        for r, w in enumerate(singles(lgv, specs, states, [(EM, 0.01, 0.0, 5)])):
            got = np.empty_like(w)
            L.check(lib.lgv_ensemble_get_state(e, r, L.ptr(got)), "get_state")
            assert np.array_equal(got, w), sides[r]
    finally:
        lib.lgv_ensemble_destroy(e)
