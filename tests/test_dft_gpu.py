"""The two-factor DFT of lgv_x2k at the sizes where its factors and its
shared-memory layout change: one column (N = 2), primes (N1 a prime, N2 = 2),
odd N1, whole and broken row blocks, one row per block, and the rows read from
global memory (N > 4096).  A mode is a sum of N1 and then N2 terms with exact
twiddles to half an ulp, so its error is at most (N1 + N2 + 8) 2^-52 times the
mean of |w|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def factors(N):
    best = (N // 2, 2)
    for n2 in range(2, N + 1, 2):
        if N % n2 == 0 and N // n2 + n2 <= sum(best):
            best = (N // n2, n2)
    return best


@pytest.mark.parametrize("N,rows", [(2, 1), (4, 17), (6, 33), (16, 16), (26, 15), (90, 31), (166, 5), (256, 47),
                                    (250, 1), (640, 19), (1018, 3), (4096, 2), (4094, 3), (4098, 2), (8192, 3),
                                    (8186, 2)])
def test_x2k_sizes(lgv, N, rows):
    from langevina_b200 import postprocess as G

    w = np.random.default_rng(N + rows).normal(size=(rows, N)) + 0.3
    got = G.x2k(w)
    x = np.arange(N, dtype=np.longdouble)
    k = np.arange(N // 2 + 1)
    arg = (np.outer(k, np.arange(N)) % N).astype(np.longdouble) * (2 * np.arccos(np.longdouble(-1)) / N)
    want = np.stack([(w[:, None, :] * np.cos(arg)).sum(-1), -(w[:, None, :] * np.sin(arg)).sum(-1)], -1) \
        if N <= 700 else None
    if want is None:  # the long sums one row and a few modes at a time
        k = np.unique(np.r_[0:6, N // 4 - 1:N // 4 + 2, N // 2 - 4:N // 2 + 1])
        arg = arg[k]
        want = np.stack([np.stack([(np.cos(arg) * r).sum(-1), -(np.sin(arg) * r).sum(-1)], -1) for r in w])
        got = got[:, k]
    bound = (sum(factors(N)) + 8) * 2.0 ** -52 * np.abs(w).mean(1)
    err = np.abs(got - (want / N).astype(np.float64)).max(axis=(1, 2))
    assert np.all(err <= bound), (err / bound).max()
    assert x.size == N and not np.any(got[:, -1, 1])  # k = N/2 is real, exactly


def test_x2k_rows_of_a_block_do_not_mix(lgv):
    """A row that is not finite leaves the others of its block as they are, and is not finite itself."""
    from langevina_b200 import postprocess as G

    w = np.random.default_rng(3).normal(size=(20, 90))
    want = G.x2k(w)
    for bad in (np.inf, -np.inf, np.nan):
        v = w.copy()
        v[7, 13] = bad
        got = G.x2k(v)
        keep = np.arange(20) != 7
        assert np.array_equal(got[keep], want[keep])
        assert not np.isfinite(got[7, :, 0]).any()
