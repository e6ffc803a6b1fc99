// lgv_dft.cuh -- the real-to-complex DFT of a wall row, W(k) = (1/N) sum_x
// w(x) e^{-2 pi i k x / N}, k = 0..N/2 (FFTW's r2c sign), shared by the
// measurer (lgv_kernels.cu) and lgv_x2k (lgv_post.cu).
//
// Two-factor Cooley-Tukey, N = N1 N2 with N2 even.  With x = N2 n1 + n2 and
// k = k1 + N1 k2,
//   Z(k1, n2) = e^{-2 pi i n2 k1 / N} sum_n1 w(N2 n1 + n2) e^{-2 pi i n1 k1 / N1}
//   W(k1 + N1 k2) = (1/N) sum_n2 Z(k1, n2) e^{-2 pi i n2 k2 / N2}.
// Since w is real only k1 = 0..N1/2 are formed: a mode whose k mod N1 is above
// N1/2 is the conjugate of mode N - k.  The terms n and -n of either sum share
// a cosine and a sine up to sign, so they are added and subtracted first, and
// the outputs k2 and -k2 share their four partial sums.  A row costs about N
// (N1 + N2) / 2 multiply-adds instead of the direct sum's N (N + 2): 20 N
// against 258 N at N = 256.  N2 is even so that k = N/2 falls on k1 = 0, whose
// sums are real: its imaginary part is an exact zero, as in the direct sum.
//
// Every output is one fixed chain of operations (explicit fma, increasing n1,
// then increasing n2), whatever the thread layout around it, so a measured
// wall transforms to the measurer's k wall bit for bit.  A value that is not
// finite makes every mode of its row not finite, as the direct sum does.
#pragma once

#include <cuda_runtime.h>

namespace lgv {
namespace dft {

struct Plan {
  int N, N1, N2;
  int K1;      // N1 / 2 + 1 columns k1
  double inv;  // 1 / N when N is a power of two (then x inv = x / N exactly), else 0
};

// the factors with the fewest multiply-adds (N even)
inline Plan make_plan(int N) {
  const double inv = (N & (N - 1)) == 0 ? 1.0 / N : 0.0;
  Plan p{N, N / 2, 2, N / 4 + 1, inv};
  for (int n2 = 2; n2 <= N; n2 += 2)
    if (N % n2 == 0 && N / n2 + n2 <= p.N1 + p.N2) p = Plan{N, N / n2, n2, N / n2 / 2 + 1, inv};
  return p;
}

// tw[m] = (cos, sin)(2 pi m / N)
__device__ __forceinline__ void fill_twiddles(double2 *tw, int N) {
  for (int m = threadIdx.x; m < N; m += blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)m / (double)N, &s, &c);
    tw[m] = make_double2(c, s);
  }
}

// A walk through the table in steps of `step` elements modulo N (byte offsets).
struct Walk {
  unsigned off, step;
  __device__ __forceinline__ Walk() {}
  __device__ __forceinline__ Walk(int st) : off(16u * st), step(16u * st) {}
  __device__ __forceinline__ double2 next(const double2 *tw, unsigned lim) {
    const double2 t = *(const double2 *)((const char *)tw + off);
    off += step;
    off = min(off, off - lim);  // off - lim wraps to a large value while off < lim
    return t;
  }
};

// Z(k1[b], n2) for B columns: w points at element n2 of the row.
template <int B>
__device__ __forceinline__ void inner(const double *w, const Plan &p, const double2 *tw, int n2, const int (&k1)[B],
                                      double2 (&z)[B]) {
  const unsigned lim = 16u * p.N;
  const int N2 = p.N2;
  double yr[B], yi[B];
  Walk wk[B];
  const double v0 = w[0];
  const bool even = !(p.N1 & 1);
  const double vh = even ? w[(p.N1 >> 1) * N2] : 0.0;
#pragma unroll
  for (int b = 0; b < B; ++b) {
    yr[b] = even ? v0 + ((k1[b] & 1) ? -vh : vh) : v0;
    yi[b] = 0.0;
    wk[b] = Walk(k1[b] * N2);
  }
  const double *wa = w + N2, *wb = w + (p.N1 - 1) * N2;
  for (int n1 = 1; n1 <= (p.N1 - 1) / 2; ++n1, wa += N2, wb -= N2) {
    const double a = *wa, c = *wb, sum = a + c, dif = a - c;
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const double2 t = wk[b].next(tw, lim);
      yr[b] = fma(sum, t.x, yr[b]);
      yi[b] = fma(-dif, t.y, yi[b]);
    }
  }
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const double2 t = tw[n2 * k1[b]];
    z[b].x = fma(yr[b], t.x, __dmul_rn(yi[b], t.y));
    z[b].y = fma(yi[b], t.x, -__dmul_rn(yr[b], t.y));
  }
}

// N W(k1 + N1 k2[b]) -> W and N W(k1 + N1 (N2 - k2[b])) -> M for B values of
// k2 = 0..N2/2: z points at Z(k1, 0).
template <int B>
__device__ __forceinline__ void outer(const double2 *z, const Plan &p, const double2 *tw, const int (&k2)[B],
                                      double2 (&W)[B], double2 (&M)[B]) {
  const unsigned lim = 16u * p.N;
  double rc[B], rs[B], ic[B], is[B];  // sums of re cos, re sin, im cos, im sin
  Walk wk[B];
  const double2 z0 = z[0], zh = z[p.N2 >> 1];
#pragma unroll
  for (int b = 0; b < B; ++b) {
    rc[b] = z0.x + ((k2[b] & 1) ? -zh.x : zh.x);
    ic[b] = z0.y + ((k2[b] & 1) ? -zh.y : zh.y);
    rs[b] = is[b] = 0.0;
    wk[b] = Walk(k2[b] * p.N1);
  }
  for (int n2 = 1; n2 < p.N2 >> 1; ++n2) {
    const double2 a = z[n2], c = z[p.N2 - n2];
    const double xs = a.x + c.x, xd = a.x - c.x, ys = a.y + c.y, yd = a.y - c.y;
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const double2 t = wk[b].next(tw, lim);
      rc[b] = fma(xs, t.x, rc[b]);
      ic[b] = fma(ys, t.x, ic[b]);
      rs[b] = fma(xd, t.y, rs[b]);
      is[b] = fma(yd, t.y, is[b]);
    }
  }
#pragma unroll
  for (int b = 0; b < B; ++b) {
    W[b] = make_double2(rc[b] + is[b], ic[b] - rs[b]);
    M[b] = make_double2(rc[b] - is[b], ic[b] + rs[b]);
  }
}

// v / N
__device__ __forceinline__ double scaled(const Plan &p, double v) { return p.inv != 0.0 ? v * p.inv : v / (double)p.N; }

// Stores W = N W(k1 + N1 k2), divided by N if SCALE, into o[2 kk], o[2 kk + 1]
// where it gives an output kk = 0..N/2 that no other (k1, k2) gives.
template <bool SCALE = true>
__device__ __forceinline__ void store(const Plan &p, int k1, int k2, const double2 &W, double *o) {
  const int k = k1 + p.N1 * k2;
  const bool conj = 2 * k > p.N;
  if (conj && (k1 == 0 || 2 * k1 == p.N1)) return;
  const int kk = conj ? p.N - k : k;
  const double y = conj ? -W.y : W.y;
  if (!SCALE) {
    o[2 * kk] = W.x;
    o[2 * kk + 1] = y;
  } else if (p.inv != 0.0) {
    o[2 * kk] = W.x * p.inv;
    o[2 * kk + 1] = y * p.inv;
  } else {
    o[2 * kk] = W.x / (double)p.N;
    o[2 * kk + 1] = y / (double)p.N;
  }
}

}  // namespace dft
}  // namespace lgv
