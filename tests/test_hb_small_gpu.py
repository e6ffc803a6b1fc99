"""The phi heat bath's two compilations of one pass, for small and for other
lattices, at their bounds (122 and 124; 52 and 54 with Gaussian proposals) and
within, against the oracle: the same decisions, per-site agreement to 1e-12 as
every stepper."""
import pytest

from lgvtest import GpuLattice, assert_state_close, rand_state

pytestmark = pytest.mark.gpu

HB = 4
COEF = dict(mass0=-4.8, lam=4.0, H=0.01, chi=5.0, seed=9)


@pytest.mark.parametrize("gauss,N", [(0, 4), (0, 18), (0, 90), (0, 122), (0, 124), (1, 4), (1, 52), (1, 54)])
def test_heat_bath_sweeps(lgv, oracle_mod, gauss, N):
    g = GpuLattice(lgv, N, **COEF)
    o = oracle_mod.Oracle(N, mode=oracle_mod.COUNTER, **COEF)
    if gauss:
        g.L.check(g.lib.lgv_set_hb_proposal(g.h, 1), "set_hb_proposal")
        o.set_hb_proposal(1)
    u = rand_state(N, N)
    for x in (g, o):
        x.set_state(u)
        x.step(HB, 0.04, nsteps=2)
    assert_state_close(g.get_state(), o.get_state(), what=f"heat bath at {N}")
    g.close()
