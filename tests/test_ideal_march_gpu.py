"""The marching ideal kernels on lattices of their own and on slabs, past the
sides that the flat launches take: the TMA-staged kernel from 128 on (sides that
32 divides) and the cp.async one above 200.

- one ideal step equals the oracle's to 1e-12 per site;
- slabs (ghost planes, fewer planes than the side) gathered equal the whole
  lattice bit for bit, for the ideal step and for PV2HBSplit23;
- every bounded wait of the TMA kernel cut to zero polls is reported as
  LGV_ERR_TIMEOUT by the next synchronising call, and the context stays usable."""
import os

import numpy as np
import pytest

from lgvtest import GpuLattice, assert_state_close, rand_state
from test_slab_gpu import run_slabs, run_whole

pytestmark = pytest.mark.gpu

PV2, IDEAL = 0, 3
COEF = dict(mass0=-4.813, lam=10.0, H=0.01, chi=5.0, gamma=1.0, diffusion=1.0 / 3.0, seed=991)


@pytest.mark.parametrize("N", [128, 202])
def test_one_step_matches_the_oracle(lgv, oracle_mod, N):
    u = rand_state(N, N, phi_scale=0.3)
    g = GpuLattice(lgv, N, **COEF)
    o = oracle_mod.Oracle(N, mode=oracle_mod.COUNTER, nranks=min(16, os.cpu_count() or 1), **COEF)
    for x in (g, o):
        x.set_state(u)
        x.step(IDEAL, 0.05)
    assert_state_close(g.get_state(), o.get_state(), what=f"ideal step at {N}")
    g.close()


@pytest.mark.parametrize("N,R", [(128, 2), (128, 3), (202, 2)])
def test_slabs_equal_whole_lattice(lgv, N, R):
    u = rand_state(N, 31 * N + R)
    plan = [(IDEAL, 0.05, 1, 1, 1), (PV2, 0.04, 1, 2, 3)]
    slabs, got = run_slabs(N, R, u, plan, COEF)
    g = run_whole(N, u, plan, COEF)
    assert np.array_equal(got, g.get_state())
    for s in slabs:
        s.close()
    g.close()


def test_tma_wait_gives_up_with_an_error(lgv, monkeypatch):
    from langevina_b200 import _lib as L

    N = 128
    u = rand_state(N, 5)
    monkeypatch.setenv("LGV_WAIT_LIMIT", "0")
    g = GpuLattice(lgv, N, **COEF)
    monkeypatch.delenv("LGV_WAIT_LIMIT")
    g.set_state(u)
    g.step(IDEAL, 0.05)
    with pytest.raises(L.LgvError) as ei:
        g.get_state()
    assert ei.value.status == L.LGV_ERR_TIMEOUT and "timed out" in str(ei.value)
    g.close()
    h = GpuLattice(lgv, N, **COEF)
    h.set_state(u)
    h.step(IDEAL, 0.05)
    assert np.isfinite(h.get_state()).all()
    h.close()
