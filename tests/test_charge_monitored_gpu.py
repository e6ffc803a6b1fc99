"""The charge heat bath with accept statistics on, one face per launch: the same
state as without them, to the last bit, and a number of decisions that does not
depend on the sizes; at the sides where the pass's grid changes (planes flat over
the blocks, half rows of whole blocks)."""
import numpy as np
import pytest

from lgvtest import GpuLattice, rand_state

pytestmark = pytest.mark.gpu

CHARGE = 5
COEF = dict(mass0=-4.8, lam=4.0, H=0.003, chi=5.0, diffusion=1.0 / 3.0, seed=771)


@pytest.mark.parametrize("N", [4, 8, 34, 50, 90, 256])
def test_statistics_leave_the_state_alone(lgv, N):
    u = rand_state(N, N)
    states = []
    for on in (False, True):
        g = GpuLattice(lgv, N, **COEF)
        g.set_state(u)
        g.monitors(on)
        g.step(CHARGE, 0.2, nsteps=2)
        states.append(g.get_state())
        if on:
            m = g.monitors()[2]
            assert m["down_counts"] + m["up_counts"] == 2 * 18 * N ** 3 and m["up_yes"] + m["up_no"] == m["up_counts"]
        g.close()
    assert np.array_equal(states[0], states[1])


def test_statistics_cost_a_small_factor(lgv, monkeypatch):
    """48^3, one face per launch: 42 us a step, with statistics 107 while their kernel was held to 32 registers (424
    bytes of spill) and 37 since."""
    import ctypes as C

    import torch

    ms = {}
    for on in (False, True):
        monkeypatch.setenv("LGV_CHARGE_FUSED", "0")
        g = GpuLattice(lgv, 48, **COEF)
        monkeypatch.delenv("LGV_CHARGE_FUSED")
        st = torch.cuda.Stream()
        g.L.check(g.lib.lgv_set_stream(g.h, C.c_void_p(st.cuda_stream)), "set_stream")
        g.initialize(2)
        g.monitors(on)
        best = 1e300
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record(st)
            g.step(CHARGE, 0.04, nsteps=40)
            e[1].record(st)
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]) / 40)
        ms[on] = best
        g.close()
    assert ms[True] <= 1.5 * ms[False], ms
