"""lgv_x2k of short rows, whose blocks take 16 to 256 rows by their number and
copy them as one run (N below 48): row counts around every block size, with
broken last blocks, on both sides of that bound.  A row's modes do not depend on
its place, so every row equals the same row transformed alone, to the last bit;
errors are bounded as in test_dft_gpu."""
import ctypes as C

import numpy as np
import pytest

from test_dft_gpu import factors

pytestmark = pytest.mark.gpu

ROUND = 148 * 3  # resident blocks


@pytest.mark.parametrize("N", [2, 4, 6, 14, 24, 46, 48, 62])
@pytest.mark.parametrize("rows", [15, ROUND * 16, ROUND * 16 + 1, ROUND * 32 + 31, ROUND * 64 + 65, ROUND * 128 + 3,
                                  ROUND * 256 + 257])
def test_rows_by_the_block(lgv, N, rows):
    from langevina_b200 import postprocess as G

    w = np.random.default_rng(N * 7 + rows).normal(size=(rows, N)) + 0.3
    got = G.x2k(w)
    want = np.fft.rfft(w, axis=-1) / N
    want = np.stack([want.real, want.imag], -1)
    # numpy's own transform is within log2(N) rounding steps of the exact one
    bound = (sum(factors(N)) + 8 + 4 * np.log2(N)) * 2.0 ** -52 * np.abs(w).mean(1)
    assert np.all(np.abs(got - want).max(axis=(1, 2)) <= bound)
    for r in sorted({0, 1, 14, rows // 2, rows - 2, rows - 1}):
        assert np.array_equal(got[r:r + 1], G.x2k(w[r:r + 1])), r


def test_rows_of_6_cost_less_than_rows_of_16(lgv):
    """300 000 rows: 121 us for rows of 6 and 113 for rows of 16 with a warp per row, now 23 and 39."""
    import torch
    from langevina_b200 import _lib as L

    us = {}
    for N in (6, 16):
        w = torch.randn(300000, N, dtype=torch.float64, device="cuda")
        out = torch.empty(300000, N // 2 + 1, 2, dtype=torch.float64, device="cuda")
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        best = 1e300
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(10):
                L.check(L.load().lgv_x2k(C.c_void_p(w.data_ptr()), 300000, N, C.c_void_p(out.data_ptr()), st), "x2k")
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 100)
        us[N] = best
    assert us[6] <= 0.85 * us[16], us
