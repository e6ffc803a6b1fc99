"""The staging buffer that an ensemble keeps between set_state and get_state
calls gives way: with the device's memory filled so far that a differentiable run,
the autotuner's copy of the state or a new tuning fits only without it, those calls
succeed, and the state still reads back afterwards."""
import ctypes as C

import numpy as np
import pytest

from lgvtest import rand_state
from test_ensemble_gpu import IDEAL, make

pytestmark = pytest.mark.gpu

N = 128
STAGING = 80 * N ** 3  # 168 MB
MB = 1 << 20


def filled(torch, leave):
    """Memory taken so that about `leave` bytes are free."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


def diff_bytes(steps, every):
    nck = (steps - 1) // every + 1
    return (nck + every + 2) * 32 * N ** 3


@pytest.mark.parametrize("what", ["diff", "autotune"])
def test_calls_fit_without_the_staging(lgv, what):
    import torch

    def call(L, lib, e):
        if what == "diff":
            obs = np.zeros(2)
            return lib.lgv_ensemble_diff_forward(e, 0.01, 0.0, 2, 1, 1, L.ptr(obs))
        choice, ms = (C.c_int * 3)(), C.c_double()
        return lib.lgv_ensemble_autotune(e, IDEAL, 1, 1, 0.01, 2, choice, C.byref(ms))

    L, lib, e = make(lgv, [(32, 3, 0.003)])  # a first run, so that every kernel is loaded
    small = rand_state(32, 1)
    L.check(lib.lgv_ensemble_set_state(e, 0, L.ptr(small)), "set_state")
    L.check(call(L, lib, e), what)
    lib.lgv_ensemble_destroy(e)

    need = diff_bytes(2, 1) if what == "diff" else 80 * N ** 3
    L, lib, e = make(lgv, [(N, 4, 0.003)])
    hold = None
    try:
        u = rand_state(N, 2)
        L.check(lib.lgv_ensemble_set_state(e, 0, L.ptr(u)), "set_state")
        # 100 MB short with the staging there, 68 MB to spare without it
        hold = filled(torch, need - 100 * MB)
        assert call(L, lib, e) == L.LGV_OK, lib.lgv_last_error()
        del hold
        torch.cuda.empty_cache()
        got = np.empty_like(u)
        L.check(lib.lgv_ensemble_get_state(e, 0, L.ptr(got)), "get_state")
        if what == "autotune":
            assert np.array_equal(got, u)
        else:
            assert np.array_equal(got[..., 4:], u[..., 4:]) and not np.array_equal(got[..., :4], u[..., :4])
    finally:
        lib.lgv_ensemble_destroy(e)
