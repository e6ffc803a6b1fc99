"""The two-launch ideal step (sides below 128, and up to 200 where 32 does not
divide them) against the oracle at its edges: the smallest side, rows shorter
than a block, a plane that is not a multiple of a block, the last side of each
rule and the first beyond it.  Per-site agreement to 1e-12, as every stepper."""
import pytest

from lgvtest import GpuLattice, assert_state_close, rand_state

pytestmark = pytest.mark.gpu

IDEAL = 3
COEF = dict(mass0=-4.8, lam=4.0, H=0.01, chi=5.0, seed=3)


@pytest.mark.parametrize("N", [4, 6, 18, 32, 34, 96, 98, 126, 128, 200, 202])
def test_ideal_step(lgv, oracle_mod, N):
    g = GpuLattice(lgv, N, **COEF)
    o = oracle_mod.Oracle(N, mode=oracle_mod.COUNTER, **COEF)
    u = rand_state(N, N)
    for x in (g, o):
        x.set_state(u)
        x.step(IDEAL, 0.04, nsteps=2 if N < 120 else 1)
    assert_state_close(g.get_state(), o.get_state(), what=f"ideal step at {N}")
