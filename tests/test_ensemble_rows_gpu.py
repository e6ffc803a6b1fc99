"""Charge steps of an ensemble against single lattices, bit for bit, at the
sides where the rows along x change their number per block: many rows, one row
per half block, rows of exactly a block's threads and of more."""
import numpy as np
import pytest

from lgvtest import rand_state
from test_ensemble_gpu import CHARGE, make, singles

pytestmark = pytest.mark.gpu


def test_charge_rows(lgv):
    specs = [(N, 20 + N, 0.003) for N in (4, 6, 18, 62, 64, 66, 126, 128, 130, 254, 256, 258)]
    L, lib, e = make(lgv, specs)
    try:
        states = [rand_state(N, N) for N, _, _ in specs]
        for r, u in enumerate(states):
            L.check(lib.lgv_ensemble_set_state(e, r, L.ptr(u)), "set_state")
        L.check(lib.lgv_ensemble_step(e, CHARGE, 2, 3, 0.1, 0.0, 3), "ensemble_step")
        for r, want in enumerate(singles(lgv, specs, states, [(CHARGE, 0.1, 0.0, 3)])):
            got = np.empty_like(want)
            L.check(lib.lgv_ensemble_get_state(e, r, L.ptr(got)), "get_state")
            assert np.array_equal(got, want), specs[r]
    finally:
        lib.lgv_ensemble_destroy(e)
