"""lgv_time_correlator where a large part of the chunks holds products past the
end of the series: short series, every lag up to T, real and complex.  A product
past the end is not formed, whatever the samples are (a NaN or an infinity stays
in the lags that it enters), and such chunks cost about what the others do.  The
sums' bound is that of test_correlator_chunks_gpu."""
import ctypes as C

import numpy as np
import pytest

from test_correlator_chunks_gpu import call, test_edges as check_edges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("T,ns,ntmax", [(2, 33, 2), (7, 1, 7), (18, 40, 18), (31, 3, 31), (46, 33, 46), (63, 5, 40),
                                        (65, 2, 65), (95, 34, 95), (97, 1, 80), (112, 64, 66)])
def test_short_series(lgv, cplx, T, ns, ntmax):
    check_edges(lgv, cplx, T, ns, ntmax, 1, False)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("T", [9, 16, 33, 50, 79, 110])
def test_values_that_are_not_finite_stay_in_their_lags(lgv, cplx, T):
    ns = 34
    rng = np.random.default_rng(T)
    draw = lambda: rng.normal(size=(T, ns)) + (1j * rng.normal(size=(T, ns)) if cplx else 0.0)
    a, b = draw(), draw()
    want = call(a, b, T, 1, False, cplx, False)
    for q in sorted({0, 1, 3, T // 2, T - 1}):
        for bad in (np.inf, np.nan):
            x, y = a.copy(), b.copy()
            x[T - 1 - q] = bad  # enters the lags 0 .. q
            got = call(x, b, T, 1, False, cplx, False)
            assert not np.isfinite(got[:q + 1]).any() and np.array_equal(got[q + 1:], want[q + 1:]), (q, bad)
            y[q] = bad          # so does this one
            got = call(a, y, T, 1, False, cplx, False)
            assert not np.isfinite(got[:q + 1]).any() and np.array_equal(got[q + 1:], want[q + 1:]), (q, bad)


def test_real_series_cost_no_more_than_complex_ones(lgv):
    """300 samples of 4000 series, 15 lags: a complex series is four times the products and twice the data, yet
    the real one took 70 us against 41 when the products of the last chunks were taken one by one (now 18)."""
    import torch
    from langevina_b200 import _lib as L

    lib, T, ns, nt = L.load(), 300, 4000, 15
    us = {}
    for w in (1, 2):
        a = torch.randn(T, ns * w, dtype=torch.float64, device="cuda")
        out = torch.empty(nt, ns * w, dtype=torch.float64, device="cuda")
        stream = torch.cuda.current_stream()
        run = lambda: L.check(lib.lgv_time_correlator(C.c_void_p(a.data_ptr()), C.c_void_p(a.data_ptr()), T, ns, ns * w,
                                                      w - 1, nt, 1, 0, C.c_void_p(out.data_ptr()),
                                                      C.c_void_p(stream.cuda_stream)), "corr")
        best = 1e300
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(20):
                run()
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 50)
        us[w] = best
    assert us[1] <= us[2], us
