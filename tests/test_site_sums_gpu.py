"""Site sums of the differentiable runs at the sides where the addition of the
block rows changes from one kernel to two (4096 blocks, between 100 and 102)
and beyond, and the gradient of a run with more steps than one kernel adds.

An average is a sum of V numbers through a tree: 16 levels at most within a
block, up to 64 block rows by one thread, 64 threads and 16 segments in turn,
so its error is at most 160 x 2^-53 of the mean magnitude."""
import numpy as np
import pytest

from lgvtest import rand_state
from test_adjoint_gpu import CFG4, SEED, EmLattice, assert_grad_close, kw_of, theta_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [100, 102, 104, 130])
def test_averages(lgv, N):
    lat = EmLattice(lgv, N, seed=SEED, **kw_of(theta_of(CFG4)))
    u = rand_state(N, N)
    lat.set_state(u)
    lat.forward(0.02, 1, 0, 1)
    avg = lat.averages(1)
    for got, x in zip(avg, (u, lat.get_state())):
        phi = x[..., :4].astype(np.longdouble)
        assert np.all(np.abs(got - phi.mean(axis=(0, 1, 2))) <= 160 * 2.0 ** -53 * np.abs(phi).mean(axis=(0, 1, 2)))
    lat.close()


def test_gradient_of_many_steps(lgv, oracle_mod):
    import diff_adjoint as da

    N, S, b, dt = 4, 4200, 4100, 0.02
    theta = theta_of(CFG4)
    theta[2] = 0.3
    lat = EmLattice(lgv, N, seed=SEED, **kw_of(theta))
    u = rand_state(N, 7)
    lat.set_state(u)
    lat.counter(0)
    lat.forward(dt, S, b, 64)
    run = da.Run("em", theta, dt, SEED, 0)
    us = run.forward(u, S)
    assert_grad_close(lat.backward(), run.gradient(us, b), 1e-9, "em adjoint of 4200 steps")
