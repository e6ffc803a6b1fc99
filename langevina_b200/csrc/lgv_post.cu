// lgv_post.cu -- post-processing of measurement histories on the device: the
// reference's x2k.exe and x2k_rotated.exe transforms and the time correlators
// of its analysis library, for data that already sits in device memory.
//
//   lgv_x2k              x2k.cxx:94-113         r2c DFT / N of every wall row
//   lgv_x2k_rotated      x2k_rotated.cxx:92-143 k walls into the vev frame
//   lgv_time_correlator  python/Loader.py:229-254 computeOtOtp (mean statistic)
//
// All three are stateless, take device pointers and run asynchronously on the
// caller's stream.  Results are deterministic: every sum runs in a fixed order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "../../include/lgv.h"
#include "lgv_dft.cuh"

namespace dft = lgv::dft;

void lgv_internal_set_error(const char *msg);

namespace {

int fail(int code, const char *msg) {
  lgv_internal_set_error(msg);
  return code;
}

int launched(const char *where) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    lgv_internal_set_error(where);
    return LGV_ERR_CUDA;
  }
  return LGV_OK;
}

// ----------------------------------------------------------------------------
// x2k: W(k) = (1/N) sum_x W(x) e^{-2 pi i k x / N}, k = 0..N/2 (FFTW's r2c sign
// and the 1/N of x2k.cxx:107-108), by the two-factor transform of lgv_dft.cuh,
// whose chains the measurer's DFT shares, so the transform of a measured wall
// reproduces the measurer's k wall bit for bit.
//
// A block takes R rows (a power of two; lanes are rows, so a twiddle is read
// once for the whole warp and the row strides, odd, keep the lanes on distinct
// banks).  Rows come in and modes leave through shared memory in whole lines;
// kX2kB1 columns, then kX2kB2 k2's, per thread share each row value: more read
// fewer values, fewer leave less of the last threads' work to waste.  STAGE =
// false (N above kX2kStageMaxN, one row per block): the table of N twiddles takes
// the room of the row, which is read and written in global memory.  33 792 rows
// of 256: 70 us (139 MB in and out take 21), against 653 us for the direct sums,
// which shared-memory bandwidth bound; now the phases between barriers do.  The
// choice: 3 columns and 2 k2's 70 us, 3 and 3 72, 2 and 2 78, 5 and 5 84, 4 and 4
// 92 (rows of 90, 500, 24 and 166: the first is the fastest too); at 5 and 5, 8
// rows and four blocks per SM 138 us, 16 rows and two blocks 90.
constexpr int kX2kThreads = 256, kX2kB1 = 3, kX2kB2 = 2, kX2kStageMaxN = 4096;
// 16 rows per block where they fit; of rows below kX2kRunN up to 256, so that the
// blocks stay one round
constexpr int kX2kLogRows = 4, kX2kMaxLogRows = 8;
constexpr int kX2kBlocks = 3;   // blocks per SM

constexpr size_t kX2kSmem = 226 * 1024 / kX2kBlocks - 1024;

struct X2kShape {
  dft::Plan p;
  int R, logR;  // rows per block
  int SA, SZ;   // strides of a row of walls / modes (doubles) and of Z (double2), odd
};

// A warp per row leaves lanes idle where rows are short, and so do 16 rows where a
// row has few columns: below this the block copies its rows as one run, takes more
// of them, and divides by N as they leave (10 000 rows of 6: 9.8 -> 6.9 us, 60 000:
// 27 -> 10, where direct sums take 6.0 and 12; 60 000 of 20 and 46: 30 -> 21 and 38
// -> 34, but of 62 45 -> 47).
constexpr int kX2kRunN = 48;

// This thread's elements of the nr rows of M doubles that are one run at g, and
// that lie `stride` apart in shared memory; f(element of g, element of shared memory).
template <typename F>
__device__ __forceinline__ void run_elements(int nr, int M, int stride, F f) {
  int r = threadIdx.x / M, x = threadIdx.x - r * M;
  const int dr = kX2kThreads / M, dx = kX2kThreads - dr * M;
#pragma unroll 4
  for (int e = threadIdx.x; e < nr * M; e += kX2kThreads) {
    f(e, r * stride + x);
    r += dr;
    x += dx;
    if (x >= M) {
      x -= M;
      ++r;
    }
  }
}

// RUNS: rows copied as one run, and divided by N as they leave.
template <bool STAGE, bool RUNS>
__global__ void __launch_bounds__(kX2kThreads, kX2kBlocks) x2k_kernel(const double *__restrict__ w, long long rows, X2kShape s,
                                                          double *__restrict__ out) {
  extern __shared__ __align__(16) double2 sm2[];
  const dft::Plan p = s.p;
  const int N = p.N, NK = N / 2 + 1, R = s.R;
  double2 *tw = sm2, *Z = sm2 + N;
  double *A = (double *)(Z + (size_t)R * s.SZ);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  dft::fill_twiddles(tw, N);
  for (long long r0 = (long long)blockIdx.x * R; r0 < rows; r0 += (long long)gridDim.x * R) {
  const int nr = (int)min((long long)R, rows - r0);
  if (STAGE) {
    if (RUNS) {
      const double *src = w + r0 * N;
      run_elements(nr, N, s.SA, [&](int e, int a) { A[a] = src[e]; });
    } else {
      for (int rr = warp; rr < nr; rr += kX2kThreads / 32)
        for (int x = lane; x < N; x += 32) A[rr * s.SA + x] = w[(r0 + rr) * N + x];
    }
  }
  __syncthreads();
  const int rr = threadIdx.x & (R - 1), u0 = threadIdx.x >> s.logR, nu = kX2kThreads >> s.logR;
  const bool live = rr < nr;
  const double *row = STAGE ? A + rr * s.SA : w + r0 * N;
  double2 *Zr = Z + (size_t)rr * s.SZ;
  const int nb1 = (p.K1 + kX2kB1 - 1) / kX2kB1;
  for (int u = u0; u < p.N2 * nb1; u += nu) {
    const int n2 = u / nb1, c0 = (u - n2 * nb1) * kX2kB1;
    int k1[kX2kB1];
    double2 z[kX2kB1];
#pragma unroll
    for (int b = 0; b < kX2kB1; ++b) k1[b] = min(c0 + b, p.K1 - 1);
    if (live) {
      dft::inner<kX2kB1>(row + n2, p, tw, n2, k1, z);
#pragma unroll
      for (int b = 0; b < kX2kB1; ++b)
        if (c0 + b < p.K1) Zr[(c0 + b) * p.N2 + n2] = z[b];
    }
  }
  __syncthreads();
  double *o = STAGE ? A + rr * s.SA : out + r0 * NK * 2;
  const int n2h = p.N2 / 2 + 1, nb2 = (n2h + kX2kB2 - 1) / kX2kB2;
  for (int u = u0; u < p.K1 * nb2; u += nu) {
    const int k1 = u / nb2, c0 = (u - k1 * nb2) * kX2kB2;
    int k2[kX2kB2];
    double2 W[kX2kB2], M[kX2kB2];
#pragma unroll
    for (int b = 0; b < kX2kB2; ++b) k2[b] = min(c0 + b, n2h - 1);
    if (live) {
      dft::outer<kX2kB2>(Zr + k1 * p.N2, p, tw, k2, W, M);
#pragma unroll
      for (int b = 0; b < kX2kB2; ++b) {
        if (c0 + b >= n2h) continue;
        dft::store<!RUNS>(p, k1, k2[b], W[b], o);
        if (k2[b] > 0 && 2 * k2[b] < p.N2) dft::store<!RUNS>(p, k1, p.N2 - k2[b], M[b], o);
      }
    }
  }
  __syncthreads();
  if (STAGE) {
    if (RUNS) {
      double *dst = out + r0 * NK * 2;
      run_elements(nr, 2 * NK, s.SA, [&](int e, int a) { dst[e] = dft::scaled(p, A[a]); });
    } else {
      for (int r = warp; r < nr; r += kX2kThreads / 32)
        for (int x = lane; x < 2 * NK; x += 32) out[(r0 + r) * NK * 2 + x] = A[r * s.SA + x];
    }
    __syncthreads();
  }
  }
}

// ----------------------------------------------------------------------------
// x2k_rotated (x2k_rotated.cxx:92-143).  Per row, n = (Re W_a(k=0)) / |.| for
// the four phi rows a = 0..3 (the identity direction (1,0,0,0) when the norm is
// below DBL_MIN); per k: phis = n.phi(k), phir_a = phi_a - n_a phis,
// A = contract_rho(n, rho(k)), V = contract_rho(n, dual(rho(k))) with rho the
// six charge rows 4..9 and dual(rho) = (rho3..5, rho0..2).  Output rows:
// 0 phis, 1-4 phir, 5-8 A, 9-12 V.
__global__ void __launch_bounds__(128) x2k_rotated_kernel(const double *__restrict__ in, long long rows, int nf,
                                                          int NK, double *__restrict__ out) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= rows * NK) return;
  const long long r = t / NK;
  const int k = (int)(t - r * NK);
  const double *w = in + r * nf * NK * 2;
  auto re = [&](int a, int kk) { return w[((long long)a * NK + kk) * 2]; };
  auto im = [&](int a, int kk) { return w[((long long)a * NK + kk) * 2 + 1]; };
  double n[4], nrm = 0;
  for (int a = 0; a < 4; ++a) {
    n[a] = re(a, 0);
    nrm += n[a] * n[a];
  }
  nrm = sqrt(nrm);
  if (nrm < 2.2250738585072014e-308) {
    n[0] = 1;
    n[1] = n[2] = n[3] = 0;
  } else {
    for (int a = 0; a < 4; ++a) n[a] /= nrm;
  }
  double pr[4], pi[4], rr[6], ri[6];
  for (int a = 0; a < 4; ++a) {
    pr[a] = re(a, k);
    pi[a] = im(a, k);
  }
  for (int b = 0; b < 6; ++b) {
    rr[b] = re(4 + b, k);
    ri[b] = im(4 + b, k);
  }
  double sr = 0, si = 0;
  for (int a = 0; a < 4; ++a) {
    sr += n[a] * pr[a];
    si += n[a] * pi[a];
  }
  double *o = out + r * 13 * NK * 2;
  auto put = [&](int a, double x, double y) {
    o[((long long)a * NK + k) * 2] = x;
    o[((long long)a * NK + k) * 2 + 1] = y;
  };
  put(0, sr, si);
  for (int a = 0; a < 4; ++a) put(1 + a, pr[a] - n[a] * sr, pi[a] - n[a] * si);
  // contract_rho(n, rho) (x2k_rotated.cxx:16-26) on real and imaginary parts
  auto contract = [&](const double *q, double *c) {
    c[0] = -(n[1] * q[0]) - n[2] * q[1] - n[3] * q[2];
    c[1] = n[0] * q[0] + n[3] * q[4] - n[2] * q[5];
    c[2] = n[0] * q[1] - n[3] * q[3] + n[1] * q[5];
    c[3] = n[0] * q[2] + n[2] * q[3] - n[1] * q[4];
  };
  double cr[4], ci[4];
  contract(rr, cr);
  contract(ri, ci);
  for (int a = 0; a < 4; ++a) put(5 + a, cr[a], ci[a]);
  const double dr[6] = {rr[3], rr[4], rr[5], rr[0], rr[1], rr[2]};
  const double di[6] = {ri[3], ri[4], ri[5], ri[0], ri[1], ri[2]};
  contract(dr, cr);
  contract(di, ci);
  for (int a = 0; a < 4; ++a) put(9 + a, cr[a], ci[a]);
}

// ----------------------------------------------------------------------------
// Time correlator (computeOtOtp, Loader.py:229-254): for every series s and
// lag tau < ntmax,
//   C_s(tau) = mean over t = 0, decim, 2 decim, ... < T - tau of a_s(t) b_s(t + tau)
// (complex product, no conjugation: the caller conjugates b, as the reference's
// computeOtOtp(d, np.conj(d))), minus mean(a_s) mean(b_s) over all T when
// `conn`.  Series are columns of time-major arrays: element t of series s at
// a[t * ld + s] (real) or a[t * ld + 2 s], +1 (complex).  Output time-major too:
// out[tau * ns + s] (complex: pairs).
//
// Block: 32 series (lanes) x kCorrLagWarps lag groups (warps); a thread owns G
// consecutive lags and keeps their sums in registers.  Every sum has a fixed
// order: with decim = 1 the products of G steps, then those sums over t, then the
// shares of the blocks that divide the time, whose number follows from T, ntmax
// and the number of series (and with it the last bits); with decim > 1 the
// products in increasing t.  The means of `conn` are sums of four quarters of the
// time with decim = 1, of all samples in increasing t otherwise.
template <bool CPLX>
struct Val {
  double re, im;
};

// VEC: complex pairs are 16-byte aligned (both arrays and ld even), so one
// 16-byte load brings a pair.
template <bool CPLX, bool VEC>
__device__ __forceinline__ Val<CPLX> ld_val(const double *p) {
  Val<CPLX> v;
  if (CPLX && VEC) {
    const double2 q = *reinterpret_cast<const double2 *>(p);
    v.re = q.x;
    v.im = q.y;
  } else {
    v.re = p[0];
    v.im = CPLX ? p[1] : 0.0;
  }
  return v;
}

template <bool CPLX>
__device__ __forceinline__ void mac(Val<CPLX> &acc, const Val<CPLX> &x, const Val<CPLX> &y) {
  if (CPLX) {
    acc.re = fma(x.re, y.re, acc.re);
    acc.re = fma(-x.im, y.im, acc.re);
    acc.im = fma(x.re, y.im, acc.im);
    acc.im = fma(x.im, y.re, acc.im);
  } else {
    acc.re = fma(x.re, y.re, acc.re);
  }
}

constexpr int kCorrLagWarps = 4;

// The sums of n samples of both series, each in increasing t: U samples of both are
// asked for before the first is added.
template <bool CPLX, bool VEC>
__device__ __forceinline__ void sample_sums(const double *pa, const double *pb, long long n, long long ld,
                                            Val<CPLX> &sa, Val<CPLX> &sb) {
  constexpr int U = CPLX ? 8 : 16;
  sa.re = sa.im = sb.re = sb.im = 0.0;
  auto add = [](Val<CPLX> &s, const Val<CPLX> &x) {
    s.re += x.re;
    s.im += x.im;
  };
  long long t = 0;
#pragma unroll 1
  for (; t + U <= n; t += U) {
    Val<CPLX> x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      x[u] = ld_val<CPLX, VEC>(pa + u * ld);
      y[u] = ld_val<CPLX, VEC>(pb + u * ld);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      add(sa, x[u]);
      add(sb, y[u]);
    }
    pa += U * ld;
    pb += U * ld;
  }
#pragma unroll 1
  for (; t < n; ++t, pa += ld, pb += ld) {
    add(sa, ld_val<CPLX, VEC>(pa));
    add(sb, ld_val<CPLX, VEC>(pb));
  }
}

// mean(a_s) mean(b_s) from the sums over all T samples
template <bool CPLX>
__device__ __forceinline__ Val<CPLX> mean_product(Val<CPLX> sa, Val<CPLX> sb, long long T) {
  Val<CPLX> cc;
  cc.re = cc.im = 0.0;
  sa.re /= (double)T;
  sa.im /= (double)T;
  sb.re /= (double)T;
  sb.im /= (double)T;
  mac<CPLX>(cc, sa, sb);
  return cc;
}

template <bool CPLX, int G>
__device__ __forceinline__ void store_lags(const Val<CPLX> (&acc)[G], const Val<CPLX> &cc, long long tau0, long long T,
                                           int ntmax, int decim, double *o, long long row) {
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const long long tau = tau0 + g;
    if (tau >= ntmax) break;
    const double cnt = (double)((T - tau + decim - 1) / decim);
    o[tau * row] = acc[g].re / cnt - cc.re;
    if (CPLX) o[tau * row + 1] = acc[g].im / cnt - cc.im;
  }
}

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}
// the double at this block's address p in the shared memory of block `rank` of the cluster
__device__ __forceinline__ double cluster_ld(const double *p, unsigned rank) {
  unsigned addr;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(addr) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];\n" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
// one value (pair) of a row into shared memory, asynchronously
template <bool CPLX, bool VEC>
__device__ __forceinline__ void copy_val(double *dst, const double *src) {
  if (CPLX && VEC) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    if (CPLX) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(dst + 1)), "l"(src + 1) : "memory");
  }
}

// The products of G steps (values of a from xa on) with G lags each, added to
// acc: step u and lag g take row u + g of the window of b, whose first G rows are
// at w0 and the others at w1 (rows are 32 values apart).  FULL: all products are
// wanted; otherwise those with u + g < left, and no other is formed.  The G steps'
// products are added by themselves first; the two that a complex multiply-add
// gives one sum are G chains apart.
template <bool CPLX, int G, bool FULL>
__device__ __forceinline__ void add_group(Val<CPLX> (&acc)[G], const double *xa, const double *w0, const double *w1,
                                          int left) {
  constexpr int W = CPLX ? 2 : 1;
  Val<CPLX> wb[2 * G - 1], sum[G];
#pragma unroll
  for (int i = 0; i < 2 * G - 1; ++i) wb[i] = ld_val<CPLX, true>((i < G ? w0 : w1) + (i < G ? i : i - G) * 32 * W);
#pragma unroll
  for (int g = 0; g < G; ++g) sum[g].re = sum[g].im = 0.0;
#pragma unroll
  for (int u = 0; u < G; ++u) {
    const Val<CPLX> x = ld_val<CPLX, true>(xa + u * 32 * W);
    auto in = [&](int g) { return FULL || u + g < left; };
#pragma unroll
    for (int g = 0; g < G; ++g)
      if (in(g)) sum[g].re = u == 0 ? x.re * wb[g].re : fma(x.re, wb[u + g].re, sum[g].re);
    if (CPLX) {
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (in(g)) sum[g].im = u == 0 ? x.re * wb[g].im : fma(x.re, wb[u + g].im, sum[g].im);
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (in(g)) sum[g].re = fma(-x.im, wb[u + g].im, sum[g].re);
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (in(g)) sum[g].im = fma(x.im, wb[u + g].re, sum[g].im);
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    acc[g].re += sum[g].re;
    if (CPLX) acc[g].im += sum[g].im;
  }
}

// Every sample (decim 1).  Time runs in chunks of kCorrChunk steps: the block
// keeps the chunk's rows of a (two chunks, one arriving by cp.async while the
// other is used) and a ring of the rows of b its lags reach, each row loaded
// once per block.  Within a chunk a thread reads G values of a and 2G - 1 of b
// from shared memory per G steps for G^2 multiply-adds.  What it replaces read
// the same values from global memory and waited for them: 14.8 of 16.2 cycles
// per issue on the load, FP64 pipe a fifth busy.  2000 samples of 1419 complex
// series, 250 lags: 600 -> 276 us (a complex multiply-add is four fma's, 155 us
// of FP64 pipe; 320 us without the time shared by two blocks, when 360 blocks
// left half the SMs with two and half with three).  Two warps per block copy more
// per product (424 us), six and eight leave the last wave emptier (374, 437 us).
// The groups of the last chunks, where some products lie past the end, are
// unrolled like the others with each product under its test: taken one by one
// (ring row by ring row) they cost a block of real series some 40 us (100 samples
// of 20 000, 20 lags 111 -> 32 us; 300 of 4257, 15 lags 70 -> 20; 1000 of 4257,
// 200 lags 166 -> 123; 2000 of 1419, 250 lags 134 -> 104).
// Complex blocks are held to 128 registers, which four per SM need.
constexpr int kCorrChunk = 16;

template <bool CPLX, bool VEC, int G>
__global__ void __launch_bounds__(32 * kCorrLagWarps, CPLX ? 4 : 3) otot_kernel(const double *__restrict__ a,
                                                                 const double *__restrict__ b, long long T,
                                                                 long long Tz, long long ns, long long ld, int ntmax,
                                                                 int conn, double *__restrict__ out) {
  constexpr int W = CPLX ? 2 : 1, C = kCorrChunk, NW = kCorrLagWarps, L = NW * G;
  constexpr int RB = L + 2 * C;  // ring rows of b: the chunk's C + L - 1, and the C arriving
  static_assert(RB % C == 0 && C % G == 0 && L % G == 0, "otot_kernel: ring");
  extern __shared__ __align__(16) double sm[];
  double *sa = sm, *sb = sm + 2 * C * 32 * W;
  const int lane = threadIdx.x, wp = threadIdx.y;
  const long long s = (long long)blockIdx.x * 32 + lane, tb = (long long)blockIdx.y * L, tau0 = tb + wp * G;
  const bool live = s < ns;
  const double *pa = a + (live ? s : 0) * W, *pb = b + (live ? s : 0) * W;
  const long long Ta = T - tb;  // samples of a that any lag of the block uses (tb < ntmax <= T)
  // this block's share of the time: blockIdx.z of the cluster's blocks takes Tz steps (a multiple of C)
  const long long tz = blockIdx.z * Tz, te = min(Ta, tz + Tz);
  // This thread copies rows wp, wp + NW, ... of every C rows; `left` rows are
  // left of the n asked for.  Ring rows start at multiples of C and the rings
  // are multiples of C long, so C rows never wrap.
  static_assert(C % NW == 0 && L % C == 0, "otot_kernel: copies");
  const double *ga = pa + (tz + wp) * ld, *gb = pb + (tb + tz + wp) * ld;
  const long long ldw = NW * ld;
  auto load_rows = [&](const double *&src, double *ring, long long left) {
    double *dst = ring + (wp * 32 + lane) * W;
    if (live) {
      if (left >= C) {
#pragma unroll
        for (int q = 0; q < C / NW; ++q) copy_val<CPLX, VEC>(dst + q * NW * 32 * W, src + q * ldw);
      } else {
        for (int q = 0; q < C / NW; ++q)
          if (wp + q * NW < left) copy_val<CPLX, VEC>(dst + q * NW * 32 * W, src + q * ldw);
      }
    }
    src += C * ld;
  };
  load_rows(ga, sa, Ta - tz);
#pragma unroll
  for (int q = 0; q < C + L; q += C) load_rows(gb, sb + q * 32 * W, Ta - tz - q);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  Val<CPLX> acc[G];
#pragma unroll
  for (int g = 0; g < G; ++g) acc[g].re = acc[g].im = 0.0;
  int ra = 0, rb = 0;  // ring rows of the chunk's first a and b
  for (long long t0 = tz; t0 < te; t0 += C) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    load_rows(ga, sa + (C - ra) * 32 * W, Ta - t0 - C);
    load_rows(gb, sb + (rb >= C ? rb - C : rb + RB - C) * 32 * W, Ta - t0 - C - L);  // onto the rows before rb
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    // The G steps' window of b: rows r .. r + 2G - 2, where the ring can end only at r + G (RB, rb, h, wp G are
    // multiples of G).  Step u and lag g of a group meet at window row u + g: a sample while h + u + g < left.
    const long long left = Ta - t0 - (tau0 - tb);
    auto groups = [&](auto full) {
#pragma unroll 1
      for (int h = 0; h < C; h += G) {
        int r = rb + h + wp * G;
        if (r >= RB) r -= RB;
        const double *w0 = sb + (r * 32 + lane) * W, *w1 = sb + ((r + G < RB ? r + G : 0) * 32 + lane) * W;
        add_group<CPLX, G, decltype(full)::value>(acc, sa + ((ra + h) * 32 + lane) * W, w0, w1, (int)left - h);
      }
    };
    if (left > 0 && tau0 < ntmax) {
      if (left >= C + G - 1) groups(std::true_type{});
      else groups(std::false_type{});
    }
    ra = C - ra;
    rb += C;
    if (rb >= RB) rb -= RB;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if (gridDim.z > 1) {  // the shares of the cluster's blocks, added by its first in their order
    __syncthreads();
    const int tid = wp * 32 + lane;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      sm[(g * W) * 32 * NW + tid] = acc[g].re;
      if (CPLX) sm[(g * W + 1) * 32 * NW + tid] = acc[g].im;
    }
    cluster_sync();
    if (blockIdx.z == 0) {
      for (unsigned z = 1; z < gridDim.z; ++z) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          acc[g].re += cluster_ld(sm + (g * W) * 32 * NW + tid, z);
          if (CPLX) acc[g].im += cluster_ld(sm + (g * W + 1) * 32 * NW + tid, z);
        }
      }
    }
    cluster_sync();  // the other blocks' shared memory stays until it is read
    if (blockIdx.z > 0) return;
  }
  Val<CPLX> cc;
  cc.re = cc.im = 0.0;
  // Each warp sums its share of the time, all add the shares in order (2000 samples
  // of 1419 series, 250 lags: 209 us real and 602 complex with all samples summed by
  // every thread, now 127 and 353).
  if (conn) {
    const long long share = (T + NW - 1) / NW, t0 = min(T, wp * share);
    Val<CPLX> sums[2];
    sample_sums<CPLX, VEC>(pa + t0 * ld, pb + t0 * ld, min(T, t0 + share) - t0, ld, sums[0], sums[1]);
    __syncthreads();  // the last reads of the ring are over
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      sm[((wp * 2 + i) * 2) * 32 + lane] = sums[i].re;
      if (CPLX) sm[((wp * 2 + i) * 2 + 1) * 32 + lane] = sums[i].im;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      sums[i].re = sums[i].im = 0.0;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        sums[i].re += sm[((w * 2 + i) * 2) * 32 + lane];
        if (CPLX) sums[i].im += sm[((w * 2 + i) * 2 + 1) * 32 + lane];
      }
    }
    cc = mean_product<CPLX>(sums[0], sums[1], T);
  }
  if (!live || tau0 >= ntmax) return;
  store_lags<CPLX, G>(acc, cc, tau0, T, ntmax, 1, out + s * W, ns * W);
}

template <bool CPLX, int G>
constexpr size_t otot_smem() {
  return (size_t)(4 * kCorrChunk + kCorrLagWarps * G) * 32 * (CPLX ? 2 : 1) * sizeof(double);
}

// Every decim-th sample (decim > 1): the rows of a chunk share little, so the
// values come from global memory, those of all G lags of one t at a time.
template <bool CPLX, bool VEC, int G>
__global__ void __launch_bounds__(32 * kCorrLagWarps) otot_decim_kernel(const double *__restrict__ a,
                                                                       const double *__restrict__ b, long long T,
                                                                       long long ns, long long ld, int ntmax,
                                                                       int decim, int conn, double *__restrict__ out) {
  constexpr int W = CPLX ? 2 : 1;
  const long long s = (long long)blockIdx.x * 32 + threadIdx.x;
  const long long tau0 = ((long long)blockIdx.y * kCorrLagWarps + threadIdx.y) * G;
  if (s >= ns || tau0 >= ntmax) return;
  const double *pa = a + s * W;
  const double *pb = b + s * W;
  Val<CPLX> acc[G];
#pragma unroll
  for (int g = 0; g < G; ++g) acc[g].re = acc[g].im = 0.0;
  long long t = 0;
#pragma unroll 2
  for (; t + tau0 + G - 1 < T; t += decim) {
    Val<CPLX> y[G];
    const Val<CPLX> x = ld_val<CPLX, VEC>(pa + t * ld);
#pragma unroll
    for (int g = 0; g < G; ++g) y[g] = ld_val<CPLX, VEC>(pb + (t + tau0 + g) * ld);
#pragma unroll
    for (int g = 0; g < G; ++g) mac<CPLX>(acc[g], x, y[g]);
  }
  for (; t + tau0 < T; t += decim) {
    const Val<CPLX> x = ld_val<CPLX, VEC>(pa + t * ld);
#pragma unroll
    for (int g = 0; g < G; ++g)
      if (t + tau0 + g < T) mac<CPLX>(acc[g], x, ld_val<CPLX, VEC>(pb + (t + tau0 + g) * ld));
  }
  Val<CPLX> cc;
  cc.re = cc.im = 0.0;
  if (conn) {
    Val<CPLX> sa, sb;
    sample_sums<CPLX, VEC>(pa, pb, T, ld, sa, sb);
    cc = mean_product<CPLX>(sa, sb, T);
  }
  store_lags<CPLX, G>(acc, cc, tau0, T, ntmax, decim, out + s * W, ns * W);
}

constexpr int kGReal = 16, kGCplx = 8;

}  // namespace

extern "C" {

int lgv_x2k(const double *walls, int64_t rows, int N, double *out, void *stream) {
  if (!walls || !out) return fail(LGV_ERR_INVALID, "lgv_x2k: NULL device pointer");
  if (rows < 0 || N < 2 || (N & 1) || N > 8192)
    return fail(LGV_ERR_INVALID, "lgv_x2k: rows >= 0, N even in [2, 8192]");
  if (rows == 0) return LGV_OK;
  X2kShape s;
  s.p = dft::make_plan(N);
  s.SA = N + 3;
  s.SZ = (s.p.K1 * s.p.N2) | 1;
  const bool stage = N <= kX2kStageMaxN;
  const size_t per_row = s.SZ * sizeof(double2) + (stage ? s.SA * sizeof(double) : 0);
  const size_t table = (size_t)N * sizeof(double2);
  s.logR = stage ? kX2kLogRows : 0;
  // more rows per block where that leaves fewer rounds of blocks
  while (N < kX2kRunN && s.logR < kX2kMaxLogRows && (rows >> s.logR) > 148LL * kX2kBlocks) ++s.logR;
  while (s.logR > 0 && table + (per_row << s.logR) > kX2kSmem) --s.logR;
  s.R = 1 << s.logR;
  const size_t smem = table + (per_row << s.logR);
  const long long blocks = std::min<long long>((rows + s.R - 1) / s.R, 148LL * kX2kBlocks);
  const auto kern = !stage ? x2k_kernel<false, false> : N < kX2kRunN ? x2k_kernel<true, true> : x2k_kernel<true, false>;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return fail(LGV_ERR_CUDA, "lgv_x2k: shared memory for the rows");
  kern<<<(unsigned)blocks, kX2kThreads, smem, (cudaStream_t)stream>>>(walls, rows, s, out);
  return launched("lgv_x2k: launch failed");
}

int lgv_x2k_rotated(const double *walls_k, int64_t rows, int nfields, int NK, double *out, void *stream) {
  if (!walls_k || !out) return fail(LGV_ERR_INVALID, "lgv_x2k_rotated: NULL device pointer");
  if (rows < 0 || nfields < 10 || NK < 1)
    return fail(LGV_ERR_INVALID, "lgv_x2k_rotated: rows >= 0, nfields >= 10, NK >= 1");
  if (rows == 0) return LGV_OK;
  const long long total = rows * (long long)NK;
  const long long blocks = (total + 127) / 128;
  if (blocks > 0x7fffffffLL) return fail(LGV_ERR_INVALID, "lgv_x2k_rotated: too many rows for one launch");
  x2k_rotated_kernel<<<(unsigned)blocks, 128, 0, (cudaStream_t)stream>>>(walls_k, rows, nfields, NK, out);
  return launched("lgv_x2k_rotated: launch failed");
}

int lgv_time_correlator(const double *a, const double *b, int64_t T, int64_t nseries, int64_t ld, int is_complex,
                        int ntmax, int decim, int conn, double *out, void *stream) {
  if (!a || !b || !out) return fail(LGV_ERR_INVALID, "lgv_time_correlator: NULL device pointer");
  if (T < 1 || nseries < 1 || decim < 1) return fail(LGV_ERR_INVALID, "lgv_time_correlator: T, nseries, decim >= 1");
  if (ntmax < 1 || ntmax > T) return fail(LGV_ERR_INVALID, "lgv_time_correlator: 1 <= ntmax <= T");
  if (ld < nseries * (is_complex ? 2 : 1)) return fail(LGV_ERR_INVALID, "lgv_time_correlator: ld below the row width");
  const int G = is_complex ? kGCplx : kGReal;
  const long long gs = (nseries + 31) / 32;
  const long long gl = ((long long)ntmax + G * kCorrLagWarps - 1) / (G * kCorrLagWarps);
  if (gs > 0x7fffffffLL || gl > 65535) return fail(LGV_ERR_INVALID, "lgv_time_correlator: grid too large");
  const dim3 grid((unsigned)gs, (unsigned)gl), block(32, kCorrLagWarps);
  const bool vec = ((uintptr_t)a % 16 == 0) && ((uintptr_t)b % 16 == 0) && ld % 2 == 0;
  cudaStream_t st = (cudaStream_t)stream;
  // Blocks that share the time of a set of series and lags, a cluster: as many
  // as make the busiest SM's share smallest, each at the cost of its own first
  // rows; one or two blocks leave an SM at about 0.55 and 0.8 of its rate
  // (2000 x 1419 complex, 250 lags: 330 / 276 / 296 us at 1 / 2 / 4 blocks; 4000 x
  // 363, 300 lags: 307 / 245 / 227 / 222 at 1 / 2 / 4 / 8; 300 x 4000, 60 lags: 56 /
  // 51 / 62).
  int Z = 1;
  if (decim == 1) {
    const long long n = gs * gl, over = G * kCorrLagWarps + 4 * kCorrChunk;
    double best = 0;
    for (int z = 1; z <= 8; z *= 2) {
      if (z > 1 && T / z < 4 * kCorrChunk) break;
      const long long k = (n * z + 147) / 148;
      const double cost = (double)(k * (T / z + over)) / (k == 1 ? 0.55 : k == 2 ? 0.8 : 1.0);
      if (z == 1 || cost < best) {
        best = cost;
        Z = z;
      }
    }
  }
#define LGV_OTOT(CP, VE, GG)                                                                                          \
  if (decim == 1) {                                                                                                  \
    constexpr size_t smem = otot_smem<CP, GG>();                                                                     \
    if (smem > 48 * 1024 && cudaFuncSetAttribute(otot_kernel<CP, VE, GG>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                 (int)smem) != cudaSuccess)                                          \
      return fail(LGV_ERR_CUDA, "lgv_time_correlator: shared memory");                                               \
    cudaLaunchConfig_t lc{};                                                                                         \
    lc.gridDim = dim3(grid.x, grid.y, (unsigned)Z);                                                                  \
    lc.blockDim = block;                                                                                             \
    lc.dynamicSmemBytes = smem;                                                                                      \
    lc.stream = st;                                                                                                  \
    cudaLaunchAttribute at{};                                                                                        \
    at.id = cudaLaunchAttributeClusterDimension;                                                                     \
    at.val.clusterDim.x = at.val.clusterDim.y = 1;                                                                   \
    at.val.clusterDim.z = (unsigned)Z;                                                                               \
    lc.attrs = &at;                                                                                                  \
    lc.numAttrs = 1;                                                                                                 \
    const long long Tz = ((T + Z - 1) / Z + kCorrChunk - 1) / kCorrChunk * kCorrChunk;                               \
    if (cudaLaunchKernelEx(&lc, otot_kernel<CP, VE, GG>, a, b, (long long)T, Tz, (long long)nseries, (long long)ld,   \
                           ntmax, conn, out) != cudaSuccess)                                                         \
      return launched("lgv_time_correlator: launch failed");                                                         \
  } else {                                                                                                           \
    otot_decim_kernel<CP, VE, GG><<<grid, block, 0, st>>>(a, b, T, nseries, ld, ntmax, decim, conn, out);            \
  }
  if (is_complex && vec) {
    LGV_OTOT(true, true, kGCplx)
  } else if (is_complex) {
    LGV_OTOT(true, false, kGCplx)
  } else {
    LGV_OTOT(false, false, kGReal)
  }
#undef LGV_OTOT
  return launched("lgv_time_correlator: launch failed");
}

}  // extern "C"
