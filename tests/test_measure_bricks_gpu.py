"""The one-pass measurement at the edges of its bricks (32 sites by 4 to 32
rows by 8 planes): sides that leave part of a brick empty in every direction,
one brick and many, each row count.  A wall is a mean over N^2 sites, summed in
pieces of at most 64 terms: its error is far below N^2 2^-53 max|obs|; the
bound used is (64 + 2 log2 N + 8) 2^-52 times the largest mean of |obs|."""
import math

import numpy as np
import pytest

from lgvtest import GpuLattice, rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [4, 6, 10, 30, 32, 34, 62, 66, 90, 98, 132])
def test_walls_of_ragged_sides(lgv, N):
    u = rand_state(N, 11 * N)
    u[..., 0] += 0.3
    g = GpuLattice(lgv, N, mass0=-4.8, lam=4.0, H=0.003)
    g.set_state(u)
    m = g.measure()
    again = g.measure()  # the brick shares and counters serve the next measurement
    phi, q = np.moveaxis(u[..., :4], -1, 0), np.moveaxis(u[..., 4:], -1, 0)
    p2 = (phi * phi).sum(0)
    n = phi / np.sqrt(p2)
    con = lambda r: np.stack([-(n[1] * r[0]) - n[2] * r[1] - n[3] * r[2], n[0] * r[0] + n[3] * r[4] - n[2] * r[5],
                              n[0] * r[1] - n[3] * r[3] + n[1] * r[5], n[0] * r[2] + n[2] * r[3] - n[1] * r[4]])
    obs = np.concatenate([phi, q, p2[None]])
    phase = np.concatenate([np.sqrt(p2)[None], n, con(q), con(q[[3, 4, 5, 0, 1, 2]]), p2[None]])
    mean = lambda f, dims: f.astype(np.longdouble).mean(axis=dims).astype(np.float64)  # numpy's own sums are longer chains
    rel = (64 + 2 * math.log2(N) + 8) * 2.0 ** -52
    for axis, dims in enumerate(((1, 2), (1, 3), (2, 3))):
        for got, f in ((m.wall[axis], obs), (m.wall_phase[axis], phase)):
            assert np.all(np.abs(got - mean(f, dims)) <= rel * max(1.0, np.abs(f).mean(axis=dims).max())), axis
    assert np.all(np.abs(m.OAverage - mean(obs, (1, 2, 3))) <= rel * np.abs(obs).mean())
    for k, v in m.arrays().items():
        assert np.array_equal(v, again.arrays()[k]), k
