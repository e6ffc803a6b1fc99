"""lgv_time_correlator at the edges of its time chunks (16 steps), lag groups
(8 complex or 16 real lags, 4 groups per block) and series blocks (32): short
series, T around whole chunks, all lags up to T, pairs on 8-byte boundaries,
decimation.  A correlation is a sum of n products divided by n: its error is at
most (n + 4) 2^-52 times the mean of |a| |b| (twice that for a complex
product's part), with |a| the modulus."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def call(a, b, ntmax, decim, conn, cplx, shift):
    import torch
    from langevina_b200 import _lib as L

    T, ns, w = a.shape[0], a.shape[1], 2 if cplx else 1
    view = lambda x: np.ascontiguousarray(x).view(np.float64).reshape(T, ns * w)
    ld = ns * w + (1 if shift else 0)  # an odd row length: rows on 8-byte boundaries only
    dev = []
    for x in (a, b):
        buf = torch.zeros(1 + T * ld, dtype=torch.float64)
        buf[1 if shift else 0:][:T * ld].reshape(T, ld)[:, :ns * w] = torch.from_numpy(view(x))
        dev.append(buf.cuda())
    out = torch.full((ntmax, ns * w), float("nan"), dtype=torch.float64, device="cuda")
    off = 8 if shift else 0
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    L.check(L.load().lgv_time_correlator(C.c_void_p(dev[0].data_ptr() + off), C.c_void_p(dev[1].data_ptr() + off), T, ns,
                                         ld, int(cplx), ntmax, decim, int(conn), C.c_void_p(out.data_ptr()), st), "corr")
    r = out.cpu().numpy()
    return r.view(np.complex128) if cplx else r


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("T,ns,ntmax,decim,shift", [
    (1, 1, 1, 1, False), (15, 33, 15, 1, False), (16, 32, 16, 1, True), (17, 31, 17, 1, False), (47, 5, 9, 1, False),
    (48, 64, 48, 1, True), (49, 1, 33, 1, False), (80, 40, 65, 1, False), (129, 7, 129, 1, True),
    (200, 35, 64, 1, False), (33, 34, 33, 2, False), (100, 3, 70, 7, True), (64, 33, 20, 100, False)])
def test_edges(lgv, cplx, T, ns, ntmax, decim, shift):
    rng = np.random.default_rng(T * 131 + ns)
    a, b = rng.normal(size=(T, ns)) + 0.2, rng.normal(size=(T, ns)) - 0.1
    if cplx:
        a, b = a + 1j * rng.normal(size=(T, ns)), b + 1j * rng.normal(size=(T, ns))
    for conn in (False, True):
        got = call(a, b, ntmax, decim, conn, cplx, shift)
        off = a.mean(0) * b.mean(0) if conn else 0.0
        for t in range(ntmax):
            x, y = a[:T - t:decim], b[t::decim]
            y = y[:len(x)]
            want = (x * y).mean(0) - off
            scale = (np.abs(x) * np.abs(y)).mean(0) + (np.abs(a).mean(0) * np.abs(b).mean(0) if conn else 0.0)
            assert np.all(np.abs(got[t] - want) <= 2 * (T + 4) * 2.0 ** -52 * 2 * scale), t


def test_samples_past_the_end_do_not_enter(lgv):
    """A sample of a enters no lag that reaches past the end, one of b none that it precedes: a NaN stays where it belongs."""
    T, ns, nt = 70, 33, 40
    rng = np.random.default_rng(9)
    a, b = rng.normal(size=(T, ns)), rng.normal(size=(T, ns))
    a[T - 3] = np.nan  # enters lags 0, 1, 2
    got = call(a, b, nt, 1, False, False, False)
    assert np.isnan(got[:3]).all() and np.isfinite(got[3:]).all()
    a[T - 3], b[5] = 0.0, np.inf  # enters lags 0 .. 5
    got = call(a, b, nt, 1, False, False, False)
    assert (~np.isfinite(got[:6])).all() and np.isfinite(got[6:]).all()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("T,ns,ntmax,shift", [(128, 3, 100, False), (130, 1, 5, True), (511, 33, 40, False),
                                              (513, 2, 512, False), (1000, 70, 333, False), (2049, 5, 17, True)])
def test_time_shared_by_a_cluster(lgv, cplx, T, ns, ntmax, shift):
    """Few series: two to eight blocks share the time, with shares that end inside a chunk, hold only the tail
    that no full chunk covers, or are empty for the largest lags."""
    test_edges(lgv, cplx, T, ns, ntmax, 1, shift)
