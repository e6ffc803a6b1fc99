"""The two-face charge launches against one face per launch (LGV_CHARGE_FUSED=0
at creation) with counter noise, for both orders of the faces and all three
orders of the directions that the counter draws, at the sides where the runs
and rows change: the smallest, runs of 8, 16 and 32 sites whole and cut short,
rows that share a block and rows of several warps, three and six charges per
thread.  Both make the same links with the same words, so the charges agree to
the last bit and phi is untouched."""
import numpy as np
import pytest

from lgvtest import GpuLattice, rand_state

pytestmark = pytest.mark.gpu

CHARGE = 5
COEF = dict(mass0=-4.8, lam=4.0, H=0.003, chi=5.0, diffusion=1.0 / 3.0, seed=77)


@pytest.mark.parametrize("N", [4, 6, 8, 10, 18, 32, 34, 64, 66, 86, 90, 120, 130, 258])
def test_two_faces_equal_one(lgv, monkeypatch, N):
    u = rand_state(N, N)
    runs = []
    for fused in ("1", "0"):
        monkeypatch.setenv("LGV_CHARGE_FUSED", fused)
        g = GpuLattice(lgv, N, **COEF)
        g.set_state(u)
        g.step(CHARGE, 0.2, nsteps=9 if N < 100 else 3)
        runs.append(g.get_state())
        assert g.counter() == (63 if N < 100 else 21)
        g.close()
    assert np.array_equal(runs[0], runs[1])
    assert np.array_equal(runs[0][..., :4], u[..., :4])
    assert not np.array_equal(runs[0][..., 4:], u[..., 4:])


def test_decisions_that_single_precision_leaves_open(lgv, oracle_mod):
    """Where the proposal barely changes the action, e^{-dS} is 1 to single precision and the uniform close to 1
    decides: steps a thousand times smaller than usual put many links there, and a charge of 1e8 makes dS overflow
    single precision.  The oracle's decisions are reproduced."""
    N = 32
    for dt, scale in ((1e-9, 1.0), (0.04, 1e8), (0.04, 1e-8)):
        g = GpuLattice(lgv, N, **COEF)
        o = oracle_mod.Oracle(N, mode=oracle_mod.COUNTER, **COEF)
        u = rand_state(N, 5)
        u[..., 4:] *= scale
        for x in (g, o):
            x.set_state(u)
            x.step(CHARGE, dt, nsteps=2)
        a, b = g.get_state()[..., 4:], o.get_state()[..., 4:]
        assert np.abs(a - b).max() <= 1e-12 * max(1.0, scale), (dt, scale)
