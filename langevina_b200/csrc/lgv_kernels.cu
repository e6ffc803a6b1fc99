// lgv_kernels.cu -- sm_100a kernels of the Model A / Model G stepper and
// measurer.  FP64 throughout; HBM-bound stencils, no tensor-core work.
//
// Kernel map (reference loop each one replaces):
//   hb_pass_kernel      EulerLangevinHB::step, one checkerboard parity per
//                       launch (Stepper.cxx:287-389)
//   hb_pass_small_kernel  the same compiled for small lattices
//   hb_sweep_kernel     the same, both parities in one z-marching launch (opt-in)
//   charge_row_kernel,  ModelGChargeHB::step, both faces of one direction per
//   charge_run_kernel   launch (Stepper.cxx:471-518, modelg_update_charge_pair
//                       :419-441): x rows per block; y and z runs of sites per
//                       thread
//   charge_pass_kernel  the same, one face per launch (slabs, decision flags,
//                       injected noise, LGV_CHARGE_FUSED=0)
//   ideal_kernel        IdealPV2::step_no_reject fused: half rotation, charge
//                       advection stencil, half rotation (Stepper.cxx:68-202);
//                       the TMA-staged ideal_tma_kernel (lgv_ideal_tma.cu)
//                       replaces it for N divisible by 32, and rot_phi_kernel
//                       and ideal_flat_kernel, one thread per site, on small
//                       lattices (ideal_flat)
//   em_kernel           Euler-Maruyama Model A step (action of Stepper.cxx:354-355)
//   energy_*            IdealPV2::computeEnergy (Stepper.cxx:204-268)
//   meas_*              Measurer::computeSliceAverage / ...Phase /
//                       computeDerivedObs (measurer.cxx:10-317): one pass over
//                       the state and one kernel for the rest up to
//                       kMeasTileMaxN, five kernels beyond
//   sum_rows_kernel     adds the block rows of site sums in a fixed order
//   batch_*             the same steps for every replica of an ensemble in one
//                       launch (no counterpart: the reference runs one lattice)
//   em_adjoint_kernel, rot_phi_kernel, ideal_adj_a/b_kernel, batch_em_*
//                       adjoints of the Euler-Maruyama and ideal steps for the
//                       differentiable runs (no counterpart)
#include "lgv_dft.cuh"
#include "lgv_ideal_tma_cta.cuh"
#include "lgv_internal.h"
#include "lgv_pdl.cuh"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <vector>

namespace lgv {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ void warp_sum(double &v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ void warp_sum(unsigned long long &v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
}

// Sums v[0..3] over the CTA into out[0..3], a row of its own for every CTA:
// sum_rows_kernel adds the rows in a fixed order.  (Adding them in the launch
// itself, by the CTA that ends last, left the chip idle for 4 us of a 10 us
// step at 48^3.)
template <int NT>
__device__ __forceinline__ void block_sum4(double (&v)[4], double *out) {
  constexpr int NW = NT / 32;
  __shared__ double sm[4][NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    warp_sum(v[q]);
    if (lane == 0) sm[q][warp] = v[q];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) t += sm[threadIdx.x][w];
    out[threadIdx.x] = t;
  }
}

// Block (slot, seg): rows n of src[slot][nb][4] with n in segment seg of
// gridDim.y, summed in a fixed order, scaled, into out[slot][gridDim.y][4].
constexpr int kSumThreads = 256;

__device__ __forceinline__ void sum_rows(const double *src, int n0, int n1, double scale, double *out) {
  __shared__ double sm[kSumThreads];
  double t = 0;
#pragma unroll 8
  for (int n = n0 + (threadIdx.x >> 2); n < n1; n += kSumThreads / 4) t += src[(size_t)n * 4 + (threadIdx.x & 3)];
  sm[threadIdx.x] = t;
  __syncthreads();
  if (threadIdx.x < 4) {
    double u = 0;
#pragma unroll 16
    for (int w = 0; w < kSumThreads / 4; ++w) u += sm[w * 4 + threadIdx.x];
    out[threadIdx.x] = u * scale;
  }
}

__global__ void __launch_bounds__(kSumThreads) sum_rows_kernel(const double *src, int nb, double scale, double *out) {
  const int slot = blockIdx.x, seg = blockIdx.y, ns = gridDim.y, per = (nb + ns - 1) / ns;
  sum_rows(src + (size_t)slot * nb * 4, seg * per, min(nb, (seg + 1) * per), scale, out + ((size_t)slot * ns + seg) * 4);
}

// Per-thread monitor tally, reduced per block and added once per block.
struct MonLocal {
  unsigned long long dc = 0, uc = 0, uy = 0, un = 0;
  double dd = 0, ud = 0;
  __device__ __forceinline__ void down(double dS) { dc++; dd += dS; }
  __device__ __forceinline__ void up_yes(double dS) { uc++; uy++; ud += dS; }
  __device__ __forceinline__ void up_no() { uc++; un++; }
};

__device__ void mon_flush(MonLocal &m, MonAcc *acc) {
  __shared__ unsigned long long s_c[4][kThreads / 32];
  __shared__ double s_d[2][kThreads / 32];
  warp_sum(m.dc);
  warp_sum(m.uc);
  warp_sum(m.uy);
  warp_sum(m.un);
  warp_sum(m.dd);
  warp_sum(m.ud);
  // linear thread index: CTAs may be two-dimensional (hb_zpass_kernel)
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  const int nwarps = (blockDim.x * blockDim.y + 31) >> 5;
  const int w = tid >> 5, l = tid & 31;
  if (l == 0) {
    s_c[0][w] = m.dc;
    s_c[1][w] = m.uc;
    s_c[2][w] = m.uy;
    s_c[3][w] = m.un;
    s_d[0][w] = m.dd;
    s_d[1][w] = m.ud;
  }
  __syncthreads();
  if (tid == 0) {
    MonLocal t;
    for (int i = 0; i < nwarps; ++i) {
      t.dc += s_c[0][i];
      t.uc += s_c[1][i];
      t.uy += s_c[2][i];
      t.un += s_c[3][i];
      t.dd += s_d[0][i];
      t.ud += s_d[1][i];
    }
    atomicAdd(&acc->down_counts, t.dc);
    atomicAdd(&acc->up_counts, t.uc);
    atomicAdd(&acc->up_yes, t.uy);
    atomicAdd(&acc->up_no, t.un);
    atomicAdd(&acc->down_dS, t.dd);
    atomicAdd(&acc->up_dS, t.ud);
  }
}

// ----------------------------------------------------------------------------
// Layout conversion: host-order AoS u[k][j][i][10] <-> red-black SoA.
__global__ void aos_to_rb_kernel(const double *__restrict__ aos, Fields f, Geo g) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long V = 2 * g.V2;
  if (n >= V) return;
  const int i = (int)(n % g.N);
  const long long r = n / g.N;
  const int j = (int)(r % g.N), k = (int)(r / g.N);
  const long long o = rb_off(g, i, j, k);
#pragma unroll
  for (int L = 0; L < 10; ++L) f.c[L][o] = aos[n * 10 + L];
}

// 128 sites per block, staged through shared memory so that the AoS side is
// written in whole lines: written straight from the threads, each 8-byte store
// of a warp touched 32 sectors (256^3: 748 us, now 396 us = 6.8 TB/s of its
// 160 bytes per site; 160^3: 187, now 102 us).
constexpr int kAosSites = 128;

__global__ void __launch_bounds__(kAosSites) rb_to_aos_kernel(Fields f, double *__restrict__ aos, Geo g) {
  __shared__ double s[kAosSites * 10];
  const long long V = 2 * g.V2, n0 = (long long)blockIdx.x * kAosSites, n = n0 + threadIdx.x;
  if (n < V) {
    const long long r = n / g.N;
    const int i = (int)(n - r * g.N), k = (int)(r / g.N), j = (int)(r - (long long)k * g.N);
    const long long o = rb_off(g, i, j, k);
    double v[10];
#pragma unroll
    for (int L = 0; L < 10; ++L) v[L] = f.c[L][o];
#pragma unroll
    for (int L = 0; L < 10; ++L) s[threadIdx.x * 10 + L] = v[L];
  }
  __syncthreads();
  const int cnt = (int)min((long long)kAosSites, V - n0) * 10;
#pragma unroll
  for (int q = 0; q < 10; ++q) {
    const int e = q * kAosSites + threadIdx.x;
    if (e < cnt) aos[n0 * 10 + e] = s[e];
  }
}

// ----------------------------------------------------------------------------
// Initial conditions from the counter streams (stream index = natural index).
__global__ void init_phi_kernel(Fields f, Geo g, uint64_t sk, double scale) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= 2 * g.V2) return;
  const int i = (int)(n % g.N);
  const long long r = n / g.N;
  const int j = (int)(r % g.N), k = (int)(r / g.N);
  Xoro x = stream_at(sk, (uint64_t)n);
  double z[4];
  const uint64_t r1 = x.next(), r2 = x.next(), r3 = x.next(), r4 = x.next();
  box_muller(r1, r2, z[0], z[1]);
  box_muller(r3, r4, z[2], z[3]);
  const long long o = rb_off(g, i, j, k);
#pragma unroll
  for (int l = 0; l < 4; ++l) f.c[l][o] = scale * z[l];
}

// ModelA::initialize_gaussian_charges (ModelA.h:463-525): n = sqrt(chi) N(0,1)
// then the zero mode is removed.  Pass 1 draws and writes per-block partial
// sums; pass 2 sums the partials in a fixed order and subtracts the mean.
__global__ void init_charge_kernel(Fields f, Geo g, uint64_t sk, double sqrtchi, double *partial) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double z[6] = {0, 0, 0, 0, 0, 0};
  if (n < 2 * g.V2) {
    const int i = (int)(n % g.N);
    const long long r = n / g.N;
    const int j = (int)(r % g.N), k = (int)(r / g.N);
    Xoro x = stream_at(sk, (uint64_t)n);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint64_t ra = x.next(), rb = x.next();
      box_muller(ra, rb, z[2 * p], z[2 * p + 1]);
    }
    const long long o = rb_off(g, i, j, k);
#pragma unroll
    for (int L = 0; L < 6; ++L) {
      z[L] *= sqrtchi;
      f.c[4 + L][o] = z[L];
    }
  }
  __shared__ double s[6][kThreads / 32];
#pragma unroll
  for (int L = 0; L < 6; ++L) {
    warp_sum(z[L]);
    if ((threadIdx.x & 31) == 0) s[L][threadIdx.x >> 5] = z[L];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double t = 0;
    for (int w = 0; w < kThreads / 32; ++w) t += s[threadIdx.x][w];
    partial[(long long)blockIdx.x * 6 + threadIdx.x] = t;
  }
}

__global__ void charge_mean_kernel(const double *partial, int nblk, double invV, double *mean) {
  // one warp per component, fixed-order strided sums then a fixed shuffle tree
  const int L = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (L >= 6) return;
  double t = 0;
  for (int b = l; b < nblk; b += 32) t += partial[(long long)b * 6 + L];
  warp_sum(t);
  if (l == 0) mean[L] = t * invV;
}

__global__ void charge_sub_kernel(Fields f, long long V, const double *mean) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= V) return;
#pragma unroll
  for (int L = 0; L < 6; ++L) f.c[4 + L][n] -= mean[L];
}

// ----------------------------------------------------------------------------
// Asynchronous global -> shared copies (cp.async, one double per copy).
__device__ __forceinline__ void cp_async8(double *smem, const double *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

__device__ __forceinline__ int wrapn(int a, int n) {
  a %= n;
  return a < 0 ? a + n : a;
}

// One heat-bath decision (Stepper.cxx:332-378): proposal phi_n = phi_o +
// sqrt(2 dt Gamma) * variance1, action change dS, Metropolis accept.
struct HbDecision {
  double pn[4];
  double dS;
  bool accept;
  uint8_t flag;
};

// The counter noise of one heat-bath site: four proposals of variance one and
// the stream, whose next draw is the accept uniform.  GAUSS: the proposals are
// the four normals of two Box-Muller pairs from the site's first four draws (as
// Euler-Maruyama's noise) instead of the reference's U(-sqrt3, sqrt3),
// Stepper.cxx:343; both are symmetric with variance one, so detailed balance
// and the proposal scale are the same.
struct HbNoise {
  double v[4];
  Xoro rng;
};

template <bool GAUSS>
__device__ __forceinline__ void hb_noise(uint64_t sk, long long nat, HbNoise &r) {
  r.rng = stream_at(sk, (uint64_t)nat);
  if (GAUSS) {
    const uint64_t r1 = r.rng.next(), r2 = r.rng.next(), r3 = r.rng.next(), r4 = r.rng.next();
    box_muller(r1, r2, r.v[0], r.v[1]);
    box_muller(r3, r4, r.v[2], r.v[3]);
  } else {
#pragma unroll
    for (int l = 0; l < 4; ++l) r.v[l] = var1(r.rng.next());
  }
}

template <bool INJECTED>
__device__ __forceinline__ void hb_decide(const double po[4], const double heff[4], const HbArgs &a, long long nat,
                                          long long V, HbNoise &z, HbDecision &r) {
  double hphi_o = 0., hphi_n = 0., s_o = 0., s_n = 0.;
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const double v = INJECTED ? a.prop[(long long)l * V + nat] : z.v[l];
    r.pn[l] = po[l] + a.rdtg * v;
    s_o += po[l] * po[l];
    s_n += r.pn[l] * r.pn[l];
    hphi_o += heff[l] * po[l];
    hphi_n += heff[l] * r.pn[l];
  }
  hphi_o += a.H * po[0];
  hphi_n += a.H * r.pn[0];
  r.dS = -(hphi_n - hphi_o) + a.Lambda2 * (s_n - s_o) + a.lam4 * (s_n * s_n - s_o * s_o);
  if (r.dS < 0) {
    r.accept = true;
    r.flag = 1;
  } else {
    if (INJECTED) {
      r.accept = a.acc[nat] < exp(-r.dS);
    } else {
      const uint64_t w = z.rng.next();
      r.accept = metropolis((uint32_t)(w >> 32), r.dS, [&] { return u53(w) < exp(-r.dS); });
    }
    r.flag = r.accept ? 2 : 0;
  }
}

__device__ __forceinline__ void mon_count(MonLocal &m, const HbDecision &d) {
  if (d.flag == 1) m.down(d.dS);
  else if (d.flag == 2) m.up_yes(d.dS);
  else m.up_no();
}

// ----------------------------------------------------------------------------
// Phi heat bath, one checkerboard parity (EulerLangevinHB::step,
// Stepper.cxx:325-381).  One thread per site of `parity`: element m of the
// parity half-row (j, k); its six neighbours are elements of the other
// parity's half-rows.
// CG: phi is read at L2 (ld.global.cg), never from a possibly stale L1 line;
// the ordered sweep (hb_ordered_kernel) reads sites other CTAs of the same
// launch have just written.
template <bool CG>
__device__ __forceinline__ double ld_phi(const double *p) {
  if (CG) return __ldcg(p);
  return *p;
}

// I: the type of the offsets in a component plane -- unsigned, in bytes, when a
// plane is below 4 GB (idx32: N <= 812), so that an address is one 64-bit base of
// the component and one 32-bit offset; int, in elements, while those fit (idx_el);
// long long, in elements, otherwise (a sweep of 814^3 in eight blocks per SM: 11.8
// ms with long long, 10.8 with int; an Euler-Maruyama step 17.0 and 16.3).
__host__ __forceinline__ bool idx32(const Geo &g) {
  return 16 * g.V2 <= 0xffffffffLL && (long long)g.N * g.N * g.Ng <= 0x7fffffffLL;
}
__host__ __forceinline__ bool idx_el(const Geo &g) {
  return 2 * g.V2 <= 0x7fffffffLL && (long long)g.N * g.N * g.Ng <= 0x7fffffffLL;
}
template <typename I>
struct Unit {
  static constexpr I of = 1;
};
template <>
struct Unit<unsigned> {
  static constexpr unsigned of = 8;
};
__device__ __forceinline__ const double *at(const double *P, unsigned off) {
  return (const double *)((const char *)P + off);
}
__device__ __forceinline__ double *at(double *P, unsigned off) { return (double *)((char *)P + off); }
__device__ __forceinline__ const double *at(const double *P, int off) { return P + off; }
__device__ __forceinline__ double *at(double *P, int off) { return P + off; }
__device__ __forceinline__ const double *at(const double *P, long long off) { return P + off; }
__device__ __forceinline__ double *at(double *P, long long off) { return P + off; }

// A site and its six neighbours as offsets in a component plane.
template <typename I>
struct Nbrs {
  I own, xp, xm, jp, jm, kp, km;
};
template <typename I>
__device__ __forceinline__ Nbrs<I> nbrs_of(const Geo &g, int parity, int m, int j, int k) {
  const int N = g.N, s = (parity + j + k) & 1;
  const I u = Unit<I>::of, H = u * (I)g.H, P = H * (I)N;  // a row, a plane
  const I half = u * (I)g.V2, row = (I)k * P + (I)j * H, c = (parity ? (I)0 : half) + row + u * (I)m;
  int xm = m - 1 + s, xp = m + s;
  if (xm < 0) xm += g.H;
  if (xp == g.H) xp = 0;
  Nbrs<I> r;
  r.own = (parity ? half : (I)0) + row + u * (I)m;
  r.xp = c + u * (I)(xp - m);
  r.xm = c + u * (I)(xm - m);
  r.jp = c + (j + 1 == N ? H - P : H);
  r.jm = c - (j == 0 ? H - P : H);
  r.kp = c + (k + 1 == g.Nz ? P - P * (I)g.Nz : P);
  r.km = c - (k == 0 ? P - P * (I)g.Nz : P);
  return r;
}
template <bool CG = false, typename I = long long>
__device__ __forceinline__ double nbr_sum(const double *P, const Nbrs<I> &o) {
  return (ld_phi<CG>(at(P, o.xp)) + ld_phi<CG>(at(P, o.xm))) + (ld_phi<CG>(at(P, o.jp)) + ld_phi<CG>(at(P, o.jm))) +
         (ld_phi<CG>(at(P, o.kp)) + ld_phi<CG>(at(P, o.km)));
}

template <typename I>
__device__ __forceinline__ I nat_index_t(const Geo &g, int i, int j, int k) {
  int kk = k + g.kg;
  if (kk < 0) kk += g.Ng;
  else if (kk >= g.Ng) kk -= g.Ng;
  return ((I)kk * g.N + j) * g.N + i;
}

// EARLY: the noise is drawn before the wait for the previous kernel.
template <bool INJECTED, bool MON, bool CG = false, typename I = long long, bool GAUSS = false, bool EARLY = false>
__device__ __forceinline__ void hb_site(const Fields &f, const Geo &g, int parity, const HbArgs &a, int m, int j,
                                        int k, MonLocal &mon) {
  const Nbrs<I> o = nbrs_of<I>(g, parity, m, j, k);
  const long long nat = (long long)nat_index_t<I>(g, 2 * m + ((parity + j + k) & 1), j, k);
  HbNoise z;
  if (!INJECTED && EARLY) {
    hb_noise<GAUSS>(a.sk, nat, z);
    pdl_wait();
  }
  double po[4], heff[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    heff[l] = nbr_sum<CG>(f.c[l], o);
    po[l] = ld_phi<CG>(at(f.c[l], o.own));
  }
  if (!INJECTED && !EARLY) hb_noise<GAUSS>(a.sk, nat, z);
  HbDecision d;
  hb_decide<INJECTED>(po, heff, a, nat, global_sites(g), z, d);
  if (d.accept) {
#pragma unroll
    for (int l = 0; l < 4; ++l) *at(f.c[l], o.own) = d.pn[l];
  }
  if (MON) mon_count(mon, d);
  if (a.flags) a.flags[nat] = d.flag;
}

// Site of this thread in a one-parity pass.  ROWS (half rows a multiple of
// 128 long): grid (H/128, N, N), no index arithmetic.  Otherwise grid
// (N*H/128 rounded up, N): the sites of plane k are flat over the x blocks,
// so no lanes idle when a half row is shorter than the block (N < 256).
template <bool ROWS>
__device__ __forceinline__ bool pass_site(const Geo &g, int &m, int &j, int &k) {
  if (ROWS) {
    m = blockIdx.x * 128 + threadIdx.x;
    j = blockIdx.y;
    k = g.zrev ? (int)(gridDim.z - 1 - blockIdx.z) : (int)blockIdx.z;
    return true;
  }
  const unsigned t = blockIdx.x * 128 + threadIdx.x, H = (unsigned)g.H;
  if (t >= (unsigned)g.N * H) return false;
  const unsigned jj = t / H;
  m = (int)(t - jj * H);
  j = (int)jj;
  k = g.zrev ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y;
  return true;
}

__host__ __forceinline__ dim3 pass_grid(const Geo &g, bool rows) {
  return rows ? dim3(g.H / 128, g.N, g.Nz) : dim3((unsigned)(((long long)g.N * g.H + 127) / 128), g.Nz);
}

// The noise is drawn before the wait for the previous kernel, at every size (a
// sweep of two passes: 64^3 12.3 us launched plainly, 10.0 with the wait first,
// 9.1 with the noise first; 256^3 342 with the wait first, 329).
template <bool INJECTED, bool MON, bool ROWS, typename I, bool GAUSS>
__device__ __forceinline__ void hb_pass(const Fields &f, const Geo &g, int parity, const HbArgs &a) {
  pdl_launch();
  if (INJECTED) pdl_wait();
  int m, j, k;
  MonLocal mon;
  if (pass_site<ROWS>(g, m, j, k))
    hb_site<INJECTED, MON, false, I, GAUSS, true>(f, g, parity, a, m, j, k, mon);
  if (MON) mon_flush(mon, a.mon);
}

// Eight blocks per SM: 60 to 64 registers let more of a site's loads be in flight
// than the 40 that the compiler takes by itself with 32-bit offsets (Gaussian
// proposals 44): a sweep of 256^3 311 -> 285 us, 512^3 2589 -> 2470; Gaussian 64^3
// 9.2 -> 7.9, 128^3 55 -> 52, 196^3 232 -> 204, 256^3 543 -> 480, 512^3 4390 -> 3800
// (219, 513 and 3990 before the 32-bit byte offsets). Ten, seven: within 5 %.
template <bool INJECTED, bool MON, bool ROWS, typename I, bool GAUSS>
__global__ void __launch_bounds__(128, 8) hb_pass_kernel(Fields f, Geo g, int parity, HbArgs a) {
  hb_pass<INJECTED, MON, ROWS, I, GAUSS>(f, g, parity, a);
}
// The same compiled for few resident blocks: on a lattice that is over in a few
// waves a pass is one chain of latencies, and the registers (76, with Gaussian
// proposals 84) let a site's 28 loads be in flight together.
// A sweep of 32^3 6.2 -> 4.8 us, 48^3 9.2 -> 5.7, 64^3 10.0 -> 7.6, 80^3 12.4 ->
// 11.2, 96^3 16.6 -> 16.0, 110^3 23.7 -> 22.9; 128^3 33 either way, and beyond
// that eight blocks are faster (256^3 285 against 334-342).  Gaussian: 32^3 7.0 ->
// 4.7, 48^3 7.7 -> 4.9, but 64^3 7.9 -> 9.3.
template <bool GAUSS>
__global__ void __launch_bounds__(128, 1) hb_pass_small_kernel(Fields f, Geo g, int parity, HbArgs a) {
  hb_pass<false, false, false, unsigned, GAUSS>(f, g, parity, a);
}
__host__ __forceinline__ bool hb_small(const Geo &g, bool gauss) {
  return g.V2 <= 148LL * (gauss ? 512 : 3 * 2048);  // N up to 52, 122
}

// ----------------------------------------------------------------------------
// Phi heat bath, one checkerboard parity per launch, z-marching
// (EulerLangevinHB::step, Stepper.cxx:325-381).  A CTA of 32 x ZP_TY threads
// owns elements m0 .. m0+31 of half rows j0 .. j0+ZP_TY-1 and marches up a
// z-chunk.  The other parity's values of each plane are loaded once: the
// thread's own element stays in registers for three planes (its z-1, z and
// z+1 neighbours), and the plane's tile with a one-element ring goes to
// shared memory for the x and y neighbours.  A site therefore costs 8 global
// loads (its own 4 components and the other parity's 4 of the plane above)
// plus the ring's share, against 28 for hb_pass_kernel, and every value of
// the other parity crosses L2 about once.  Decisions, streams and results are
// those of hb_site.
constexpr int ZP_TM = 32, ZP_TY = 8, ZP_NT = ZP_TM * ZP_TY;
constexpr int ZP_W = ZP_TM + 2, ZP_R = ZP_TY + 2, ZP_PL = ZP_W * ZP_R;  // padded tile of one component
constexpr int ZP_RING = 2 * ZP_TM + 2 * ZP_TY;

template <bool INJECTED, bool MON>
__global__ void __launch_bounds__(ZP_NT) hb_zpass_kernel(Fields f, Geo g, int parity, int zchunk, HbArgs a) {
  __shared__ double tile[2][4][ZP_PL];
  const int N = g.N, H = g.H;
  const int tm = threadIdx.x, ty = threadIdx.y, tid = ty * ZP_TM + tm;
  const int m0 = blockIdx.x * ZP_TM, j0 = blockIdx.y * ZP_TY;
  const int k0 = blockIdx.z * zchunk, k1 = min(k0 + zchunk, N);
  const int tme = min(ZP_TM, H - m0), tye = min(ZP_TY, N - j0);  // valid extent of this tile
  const bool own = tm < tme && ty < tye;
  const int m = m0 + tm, j = j0 + ty;
  const long long ob = (long long)(parity ^ 1) * g.V2, pb = (long long)parity * g.V2;
  // ring element of this thread (tid < ZP_RING): padded position (rx, ry) and half-row element (rm, rj)
  // rows above and below the tile (tme elements each), then the columns left
  // and right of it (tye rows each); corners are not needed
  int rx = 0, ry = 0, rm = 0, rj = 0;
  bool ring_live = false;
  if (tid < ZP_TM) {
    rx = 1 + tid, ry = 0, ring_live = tid < tme;
  } else if (tid < 2 * ZP_TM) {
    rx = 1 + tid - ZP_TM, ry = tye + 1, ring_live = tid - ZP_TM < tme;
  } else if (tid < 2 * ZP_TM + ZP_TY) {
    rx = 0, ry = 1 + tid - 2 * ZP_TM, ring_live = tid - 2 * ZP_TM < tye;
  } else if (tid < ZP_RING) {
    rx = tme + 1, ry = 1 + tid - 2 * ZP_TM - ZP_TY, ring_live = tid - 2 * ZP_TM - ZP_TY < tye;
  }
  if (ring_live) {
    rm = m0 + rx - 1;
    rj = j0 + ry - 1;
    rm = rm < 0 ? rm + H : (rm >= H ? rm - H : rm);
    rj = rj < 0 ? rj + N : (rj >= N ? rj - N : rj);
  }
  // the other parity's values of plane kk: own element -> o[], ring element -> smem
  auto load_other = [&](int kk, double (&o)[4], int buf) {
    const int kw = kk < 0 ? kk + N : (kk >= N ? kk - N : kk);
    if (own) {
      const long long off = ob + ((long long)kw * N + j) * H + m;
#pragma unroll
      for (int l = 0; l < 4; ++l) o[l] = f.c[l][off];
    }
    if (ring_live) {
      const long long off = ob + ((long long)kw * N + rj) * H + rm;
#pragma unroll
      for (int l = 0; l < 4; ++l) tile[buf][l][ry * ZP_W + rx] = f.c[l][off];
    }
  };
  double oz[4] = {0, 0, 0, 0}, oc[4] = {0, 0, 0, 0}, on[4] = {0, 0, 0, 0};
  load_other(k0 - 1, oz, 0);  // only the own element is used (z-1 neighbour); the ring is overwritten below
  load_other(k0, oc, 0);
  if (own) {
#pragma unroll
    for (int l = 0; l < 4; ++l) tile[0][l][(ty + 1) * ZP_W + tm + 1] = oc[l];
  }
  __syncthreads();
  MonLocal mon;
  for (int k = k0; k < k1; ++k) {
    const int b = (k - k0) & 1;
    load_other(k + 1, on, b ^ 1);
    if (own) {
      const int s = (parity + j + k) & 1;
      const double *T = &tile[b][0][0];
      const int c = (ty + 1) * ZP_W + tm + 1;
      const long long offp = pb + ((long long)k * N + j) * H + m;
      double po[4], heff[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const double *Tl = T + l * ZP_PL;
        // x neighbours: elements m-1+s and m+s of the other parity's row
        heff[l] = (Tl[c + s] + Tl[c - 1 + s]) + (Tl[c + ZP_W] + Tl[c - ZP_W]) + (on[l] + oz[l]);
        po[l] = f.c[l][offp];
      }
      const long long nat = ((long long)k * N + j) * N + 2 * m + s;
      HbDecision d;
      HbNoise z;
      if (!INJECTED) hb_noise<false>(a.sk, nat, z);
      hb_decide<INJECTED>(po, heff, a, nat, 2 * g.V2, z, d);
      if (d.accept) {
#pragma unroll
        for (int l = 0; l < 4; ++l) f.c[l][offp] = d.pn[l];
      }
      if (MON) mon_count(mon, d);
      if (a.flags) a.flags[nat] = d.flag;
#pragma unroll
      for (int l = 0; l < 4; ++l) tile[b ^ 1][l][c] = on[l];
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      oz[l] = oc[l];
      oc[l] = on[l];
    }
    __syncthreads();
  }
  if (MON) mon_flush(mon, a.mon);
}

// ----------------------------------------------------------------------------
// Phi heat bath, one or more whole sweeps (EulerLangevinHB::step,
// Stepper.cxx:287-389) in one persistent launch, ordered through the lattice
// by z-slabs so that the odd pass of a slab runs while its phi is still in
// L2.
//
// The lattice is cut into nslab slabs of S planes.  An item is one parity
// pass (phase p: sweep p/2, parity p&1) over one slab; it is split into cpi
// chunks of `spc` sites (sites of that parity in slab-local (k, j, m) order).
// A host-built schedule lists every chunk of every item in an order in which
// item (p, s) comes after the three items (p-1, s-1), (p-1, s), (p-1, s+1)
// (periodic in s) it depends on: the pass of phase p reads the sites of the
// other parity in planes sS-1 .. (s+1)S, which those items write, and writes
// sites those items read.  CTAs draw chunks in schedule order from an atomic
// ticket; a chunk of phase p >= 1 first waits until its three items have
// completed all their chunks.  Chunks are only ever handed to running CTAs
// and a chunk waits only on chunks with lower tickets, so the waits always
// end; each is still bounded, and a wait that gives up counts in
// sync[kSyncTimeouts], skips its sites and lets the host report
// LGV_ERR_TIMEOUT.  The result is that of the sequential passes bit for bit:
// every site sees exactly the neighbour values it sees there.
//
// phi moves 32 B/site in and 32 B/site out per sweep when the odd pass of a
// slab re-reads it from L2 (the two one-parity launches move 48 B/site each).
constexpr int kSyncTicket = 0, kSyncExit = 1, kSyncTimeouts = 2, kSyncDone = 3;
constexpr int kHbOrderedThreads = 128;

struct HbSched {
  const int *sched;            // ticket -> item * cpi + chunk, item = phase * nslab + slab
  unsigned long long *sync;    // [ticket, exits, timeouts, done[nphase * nslab]]
  int total;                   // tickets
  int cpi;                     // chunks per item
  int spc;                     // sites per chunk (a multiple of kHbOrderedThreads)
  int nslab, S, nphase;
  int limit;                   // polls before a dependency wait gives up
  uint64_t sk[4];              // counter keys of the sweeps (phase / 2)
};

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Thread 0 waits until the three items item (p, s) depends on have completed
// all their chunks; false (and a count in sync[kSyncTimeouts]) if a wait gives
// up.  `seen` caches the last two items already found ready.
__device__ __forceinline__ bool hb_deps_ready(const HbSched &s, int item, int (&seen)[2]) {
  const int phase = item / s.nslab, slab = item - phase * s.nslab;
  if (phase == 0 || item == seen[0] || item == seen[1]) return true;
  for (int d = -1; d <= 1; ++d) {
    const int dep = (phase - 1) * s.nslab + (slab + d + s.nslab) % s.nslab;
    const unsigned long long *p = &s.sync[kSyncDone + dep];
    int it = 0;
    while (ld_acquire(p) < (unsigned long long)s.cpi) {
      if (++it > s.limit) {
        atomicAdd(&s.sync[kSyncTimeouts], 1ull);
        return false;
      }
      __nanosleep(64);
    }
  }
  seen[1] = seen[0];
  seen[0] = item;
  return true;
}

template <bool INJECTED, bool MON>
__global__ void __launch_bounds__(kHbOrderedThreads) hb_ordered_kernel(Fields f, Geo g, HbArgs a, HbSched s) {
  __shared__ int s_work, s_ok;
  MonLocal mon;
  const long long item_sites = (long long)s.S * g.N * g.H;
  // Thread 0 draws the next ticket while the CTA works on the current chunk.
  // A CTA then holds at most two tickets, and each waits only on lower ones,
  // so the lowest unfinished chunk can always proceed.
  unsigned long long next = 0;
  int seen[2] = {-1, -1};
  if (threadIdx.x == 0) next = atomicAdd(&s.sync[kSyncTicket], 1ull);
  for (;;) {
    if (threadIdx.x == 0) {
      const int w = next < (unsigned long long)s.total ? __ldg(s.sched + next) : -1;
      s_ok = w >= 0 ? (int)hb_deps_ready(s, w / s.cpi, seen) : 1;
      s_work = w;
    }
    __syncthreads();
    const int w = s_work, ok = s_ok;
    if (w < 0) break;
    if (threadIdx.x == 0) next = atomicAdd(&s.sync[kSyncTicket], 1ull);
    const int item = w / s.cpi, chunk = w - item * s.cpi;
    const int phase = item / s.nslab, slab = item - phase * s.nslab;
    if (ok) {
      HbArgs aa = a;
      if (!INJECTED) {
        const int q = phase >> 1;  // constant indices: the key array stays in kernel parameters
        aa.sk = q == 0 ? s.sk[0] : q == 1 ? s.sk[1] : q == 2 ? s.sk[2] : s.sk[3];
      }
      const int parity = phase & 1;
      for (int r = threadIdx.x; r < s.spc; r += kHbOrderedThreads) {
        const long long q = (long long)chunk * s.spc + r;
        if (q >= item_sites) break;
        const unsigned u = (unsigned)q, H = (unsigned)g.H, N = (unsigned)g.N;
        const unsigned row = u / H;
        const int m = (int)(u - row * H);
        const unsigned kk = row / N;
        const int j = (int)(row - kk * N);
        hb_site<INJECTED, MON, true>(f, g, parity, aa, m, j, slab * s.S + (int)kk, mon);
      }
    }
    // The barrier orders every thread's stores before thread 0's fence, and
    // the fence (cumulative) before the completion count.
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(&s.sync[kSyncDone + item], 1ull);
    }
  }
  if (MON) mon_flush(mon, a.mon);
  // The last CTA out clears the ticket, exit and completion counters for the
  // next launch (the timeout count stays for the host to read).
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&s.sync[kSyncExit], 1ull) == gridDim.x - 1) {
      s.sync[kSyncTicket] = 0;
      s.sync[kSyncExit] = 0;
      for (int i = 0; i < s.nphase * s.nslab; ++i) s.sync[kSyncDone + i] = 0;
    }
  }
}

// ----------------------------------------------------------------------------
// Phi heat bath, one full checkerboard sweep (EulerLangevinHB::step,
// Stepper.cxx:287-389) in a single launch.  A CTA owns HB_TM x HB_TY
// pair-columns -- element m of both parity half-rows of row j, i.e. natural
// x = 2m and 2m+1 -- and marches up a z-chunk.  At plane p it
//   (1) runs the even pass on plane p over its tile plus a one-element ring,
//       from the old odd values of planes p-1, p, p+1 kept in shared memory
//       over a two-element ring;
//   (2) runs the odd pass on plane p-1 over its tile from the new even values
//       of planes p-2, p-1, p, and writes both parities of plane p-1.
// The ring's even updates are recomputed by the neighbouring CTAs bit for bit
// (same inputs, same counter stream), so no CTA waits for another.  phi is
// read once and written once (to `out`): 64 B per site per sweep.  cp.async
// brings plane p+2 (odd) and p+1 (even) in while plane p computes.
constexpr int HB_TM = 32, HB_TY = 8;
constexpr int HB_OW = HB_TM + 4, HB_OH = HB_TY + 4, HB_OP = HB_OW * HB_OH;  // old odd: two-element ring
constexpr int HB_EW = HB_TM + 2, HB_EH = HB_TY + 2, HB_EP = HB_EW * HB_EH;  // even: one-element ring
constexpr size_t HB_SMEM = (size_t)(4 * 4 * HB_OP + 2 * 4 * HB_EP + 3 * 4 * HB_EP) * sizeof(double);

template <bool INJECTED, bool MON>
__global__ void __launch_bounds__(HB_TM *HB_TY, 2) hb_sweep_kernel(Fields in, Fields out, Geo g, int zchunk, HbArgs a) {
  extern __shared__ double smem[];
  double *oo = smem;                     // [4 stages][4][HB_OP] old odd
  double *oe = oo + 4 * 4 * HB_OP;       // [2 stages][4][HB_EP] old even
  double *ne = oe + 2 * 4 * HB_EP;       // [3 stages][4][HB_EP] new even
  const int N = g.N, H = g.H;
  const long long V2 = g.V2, V = 2 * V2;
  const int tid = threadIdx.x;
  const int tm = tid % HB_TM, tj = tid / HB_TM;
  const int m0 = blockIdx.x * HB_TM, j0 = blockIdx.y * HB_TY;
  const int z0 = blockIdx.z * zchunk;
  const int z1 = min(z0 + zchunk, N);
  const int nit = (z1 - z0) + 2;
  MonLocal mon;

  auto issue_odd = [&](int plane, int stage) {
    for (int idx = tid; idx < HB_OP; idx += HB_TM * HB_TY) {
      const int qm = idx % HB_OW, qj = idx / HB_OW;
      const int m = wrapn(m0 - 2 + qm, H), j = wrapn(j0 - 2 + qj, N);
      const long long off = V2 + ((long long)plane * N + j) * H + m;
#pragma unroll
      for (int l = 0; l < 4; ++l) cp_async8(&oo[(stage * 4 + l) * HB_OP + idx], in.c[l] + off);
    }
  };
  auto issue_even = [&](int plane, int stage) {
    for (int idx = tid; idx < HB_EP; idx += HB_TM * HB_TY) {
      const int qm = idx % HB_EW, qj = idx / HB_EW;
      const int m = wrapn(m0 - 1 + qm, H), j = wrapn(j0 - 1 + qj, N);
      const long long off = ((long long)plane * N + j) * H + m;
#pragma unroll
      for (int l = 0; l < 4; ++l) cp_async8(&oe[(stage * 4 + l) * HB_EP + idx], in.c[l] + off);
    }
  };

  issue_odd(wrapn(z0 - 2, N), 0);
  issue_odd(wrapn(z0 - 1, N), 1);
  issue_odd(z0, 2);
  issue_even(wrapn(z0 - 1, N), 0);
  cp_async_commit();

  for (int it = 0; it < nit; ++it) {
    const int p = wrapn(z0 - 1 + it, N);
    cp_async_wait_all();
    __syncthreads();
    if (it + 1 < nit) {
      issue_odd(wrapn(p + 2, N), (it + 3) & 3);
      issue_even(wrapn(p + 1, N), (it + 1) & 1);
    }
    cp_async_commit();

    // (1) even pass on plane p over the tile and its one-element ring
    const double *oom = oo + ((it & 3) * 4) * HB_OP;        // plane p-1
    const double *ooc = oo + (((it + 1) & 3) * 4) * HB_OP;  // plane p
    const double *oop = oo + (((it + 2) & 3) * 4) * HB_OP;  // plane p+1
    const double *oec = oe + ((it & 1) * 4) * HB_EP;
    double *nec = ne + ((it % 3) * 4) * HB_EP;
    const bool in_chunk_e = (it >= 1) && (it <= nit - 2);
    for (int e = tid; e < HB_EP; e += HB_TM * HB_TY) {
      const int qm = e % HB_EW, qj = e / HB_EW;
      const int mr = m0 - 1 + qm, jr = j0 - 1 + qj;
      const int m = wrapn(mr, H), j = wrapn(jr, N);
      const int s0 = (j + p) & 1;
      const int oc = (qj + 1) * HB_OW + (qm + 1);
      double po[4], heff[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const double *C = ooc + l * HB_OP;
        heff[l] = (C[oc + s0] + C[oc - 1 + s0]) + (C[oc + HB_OW] + C[oc - HB_OW]) +
                  (oop[l * HB_OP + oc] + oom[l * HB_OP + oc]);
        po[l] = oec[l * HB_EP + e];
      }
      const long long nat = ((long long)p * N + j) * N + 2 * m + s0;
      HbDecision d;
      HbNoise z;
      if (!INJECTED) hb_noise<false>(a.sk, nat, z);
      hb_decide<INJECTED>(po, heff, a, nat, V, z, d);
#pragma unroll
      for (int l = 0; l < 4; ++l) nec[l * HB_EP + e] = d.accept ? d.pn[l] : po[l];
      const bool own = in_chunk_e && qm >= 1 && qm <= HB_TM && qj >= 1 && qj <= HB_TY && mr < H && jr < N;
      if (own) {
        if (MON) mon_count(mon, d);
        if (a.flags) a.flags[nat] = d.flag;
      }
    }
    __syncthreads();

    // (2) odd pass on plane q = p-1 over the tile; write both parities of q
    if (it >= 2) {
      const int q = wrapn(p - 1, N);
      const int mr = m0 + tm, jr = j0 + tj;
      const bool act = mr < H && jr < N;
      const int m = wrapn(mr, H), j = wrapn(jr, N);
      const int s1 = (1 + j + q) & 1;
      const int ec = (tj + 1) * HB_EW + (tm + 1);
      const double *nem = ne + (((it + 1) % 3) * 4) * HB_EP;  // plane p-2
      const double *neq = ne + (((it + 2) % 3) * 4) * HB_EP;  // plane p-1
      const double *oq = oom;                                  // old odd of plane p-1
      const int oc = (tj + 2) * HB_OW + (tm + 2);
      double po[4], heff[4], ev[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const double *C = neq + l * HB_EP;
        heff[l] = (C[ec + s1] + C[ec - 1 + s1]) + (C[ec + HB_EW] + C[ec - HB_EW]) +
                  (nec[l * HB_EP + ec] + nem[l * HB_EP + ec]);
        po[l] = oq[l * HB_OP + oc];
        ev[l] = C[ec];
      }
      const long long nat = ((long long)q * N + j) * N + 2 * m + s1;
      HbDecision d;
      HbNoise z;
      if (!INJECTED) hb_noise<false>(a.sk, nat, z);
      hb_decide<INJECTED>(po, heff, a, nat, V, z, d);
      if (act) {
        const long long row = ((long long)q * N + j) * H + m;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          out.c[l][row] = ev[l];
          out.c[l][V2 + row] = d.accept ? d.pn[l] : po[l];
        }
        if (MON) mon_count(mon, d);
        if (a.flags) a.flags[nat] = d.flag;
      }
    }
  }
  if (MON) mon_flush(mon, a.mon);
}

// ----------------------------------------------------------------------------
// Action change of moving q from A to B (modelg_update_charge_pair,
// Stepper.cxx:419-441): ((nA-q)^2 + (nB+q)^2 - nA^2 - nB^2) / (2 chi), the
// squares multiplied out.
__device__ __forceinline__ double charge_dS(double nA, double nB, double q, double invchi) {
  return (q * invchi) * (q + (nB - nA));
}
// Accept with the 32-bit uniform of hi.
__device__ __forceinline__ bool charge_accept(double dS, uint32_t hi) {
  return metropolis(hi, dS, [&] { return dS < 0 || u32(hi) < exp(-dS); });
}

// Charge heat bath, one face (direction `dir`, A-site parity eoA).  One thread
// per link (A, B = A + e_dir); the links of a face are disjoint, so the update
// is race free and conserves each charge exactly (Stepper.cxx:493-517).
template <bool INJECTED, bool MON, typename I = long long>
__device__ __forceinline__ void charge_link_site(const Fields &f, const Geo &g, int dir, int eoA, const ChargeArgs &a,
                                                 int m, int j, int k, MonLocal &mon) {
  const int H = g.H, N = g.N;
  const int s = (eoA + j + k) & 1;
  const int i = 2 * m + s;
  const I offA = (I)eoA * (I)g.V2 + ((I)k * N + j) * H + m;
  I offB;
  const I ob = (I)(eoA ^ 1) * (I)g.V2;
  if (dir == 0) {
    int mb = m + s;
    if (mb == H) mb = 0;
    offB = ob + ((I)k * N + j) * H + mb;
  } else if (dir == 1) {
    offB = ob + ((I)k * N + wrap_inc(j, N)) * H + m;
  } else {
    offB = ob + ((I)wrap_inc(k, g.Nz) * N + j) * H + m;
  }
  const long long nat = (long long)nat_index_t<I>(g, i, j, k);
  const long long V = global_sites(g);
  WordStream ws{};
  if (!INJECTED) ws = words_at(a.sk, 6 * (uint64_t)nat);
#pragma unroll
  for (int L = 0; L < 6; ++L) {
    double *P = f.c[4 + L];
    const double nA = P[offA], nB = P[offB];
    const long long ii = (long long)(a.pass * 6 + L) * V + nat;
    uint64_t ra = 0;
    double v;
    if (INJECTED) {
      v = a.q[ii];
    } else {
      ra = ws.next();
      v = v32(lo32(ra));
    }
    const double q = __dmul_rn(a.rms, v);
    const double dS = charge_dS(nA, nB, q, 2.0 * a.inv2chi);
    const bool accept = INJECTED ? dS < 0 || a.acc[ii] < exp(-dS) : charge_accept(dS, hi32(ra));
    const uint8_t fl = dS < 0 ? 1 : accept ? 2 : 0;
    if (MON) {
      if (fl == 1) mon.down(dS);
      else if (fl == 2) mon.up_yes(dS);
      else mon.up_no();
    }
    if (accept) {
      P[offA] = nA - q;
      P[offB] = nB + q;
    }
    if (a.flags) a.flags[ii] = fl;
  }
}

// Grid as hb_pass_kernel (pass_site).
// 16 blocks of 128 threads per SM (32 registers): the link updates are long
// integer / FP64 chains, and full occupancy hides them best.  With statistics
// eight: in 32 registers the tallies spill 300 to 600 bytes (a charge step of 48^3
// 102 us, 256^3 2917; in 64 registers 37 and 2350).
template <bool INJECTED, bool MON, bool ROWS, typename I>
__global__ void __launch_bounds__(128, MON ? 8 : 16) charge_pass_kernel(Fields f, Geo g, int dir, int eoA, ChargeArgs a) {
  pdl_launch();
  pdl_wait();
  int m, j, k;
  MonLocal mon;
  if (pass_site<ROWS>(g, m, j, k)) charge_link_site<INJECTED, MON, I>(f, g, dir, eoA, a, m, j, k, mon);
  if (MON) mon_flush(mon, a.mon);
}

// ----------------------------------------------------------------------------
// Charge heat bath, both faces of one direction per launch, one charge per
// thread (ModelGChargeHB::step, Stepper.cxx:471-518).  The six charges do not
// mix, so a thread takes one charge of a run of sites along the direction,
// applies the first face (dir, eo[0]) and then the second (dir, eo[1]) in
// registers and writes every site once: 16 B per site, charge and direction
// instead of the 32 that two one-face passes move.  Reads `in`, writes `out`.
// Links, words and outcomes are those of charge_link_site.  A charge step: 32^3
// 37 -> 10 us, 64^3 49 -> 22, 90^3 87 -> 56, 128^3 -> 127, 160^3 400 -> 252,
// 256^3 1684 -> 980 (5.0 TB/s of the 288 B/site that three directions move at
// least).  Issue bounds it (74-79 % active at 160^3: 78 instructions per link
// of one charge in y and z, 96 in x, most of them the word's two 64-bit
// products and shifts), then DRAM.
struct ChargeDirArgs {
  const double *in;  // charge 0 of six evenly spaced planes
  double *out;
  long long pitch_in, pitch_out;
  double rms, invchi;
  uint64_t sk[2];
  int eo[2];
};

// One link of one charge: word z of the face's sequence gives the proposal and
// the accept uniform; updates nA and nB.
__device__ __forceinline__ void charge_link(double &nA, double &nB, uint64_t z, double rms, double invchi) {
  const uint64_t r = mix64(z);
  const double q = __dmul_rn(rms, v32(lo32(r)));  // never contracted with the sums below: every kernel gives the same bits
  const bool yes = charge_accept(charge_dS(nA, nB, q, invchi), hi32(r));
  if (yes) {
    nA -= q;
    nB += q;
  }
}

// y (DIR 1) and z (DIR 2), one run: charge L of the sites b0 .. b0 + len - 1
// along the direction at fixed i and o (k or j); b0 = c0 or c0 + 1, the one
// whose site is an A site of the second face.  Its own second-face links are
// (b0, b0 + 1), (b0 + 2, b0 + 3), ..., and the first-face links they need
// (b0 - 1, b0), (b0 + 1, b0 + 2), ...: one more than its share, the link it has
// in common with the next run.  Offsets (I) are in bytes.  WRAP: the run may
// reach past N - 1.
template <int DIR, bool WRAP, typename I>
__device__ __forceinline__ void charge_run(const Geo &g, int L, int i, int o, int c0, int len, const ChargeDirArgs &a) {
  const int N = g.N, H = g.H;
  const int P0 = a.eo[1];  // parity of the sites b0, b0 + 2, ...
  const int b0 = c0 + ((P0 ^ (i + o)) & 1);
  const I base = 8 * ((DIR == 1 ? (I)o * N * H : (I)o * H) + (i >> 1));
  const I E = 8 * ((I)P0 * (I)g.V2) + base, O = 8 * ((I)(P0 ^ 1) * (I)g.V2) + base;
  const I str = 8 * (DIR == 1 ? (I)H : (I)N * H), adv = 2 * str, lap = (I)N * str;
  const double *in = a.in + L * a.pitch_in;
  double *out = a.out + L * a.pitch_out;
  auto ld = [&](I off) { return *(const double *)((const char *)in + off); };
  auto st = [&](I off, double x) { *(double *)((char *)out + off) = x; };
  auto wrap = [&](int c) { return c >= N ? c - N : c; };
  // word of the link whose A site has coordinate c: (6 nat + L + 1) golden
  const uint64_t ns = DIR == 1 ? (uint64_t)N : (uint64_t)N * N;
  const uint64_t nb = DIR == 1 ? (uint64_t)o * N * N + i : (uint64_t)o * N + i;
  const uint64_t dz = 12 * ns * kGolden, zlap = 6 * ns * N * kGolden, zb = (6 * nb + L + 1) * kGolden;
  const int cm = b0 == 0 ? N - 1 : b0 - 1, c1 = wrap(b0 + 1), c2 = wrap(b0 + 2);
  uint64_t z2 = a.sk[1] + zb + 6 * ns * b0 * kGolden;  // second face, A site c
  uint64_t z1 = a.sk[0] + zb + 6 * ns * c1 * kGolden;  // first face, A site c + 1
  const uint64_t zm = a.sk[0] + zb + 6 * ns * cm * kGolden;
  I se = E + (I)b0 * str, so = O + (I)c1 * str;  // where this pair of sites goes
  I le = E + (I)c2 * str;                        // the even site read last
  const I endE = E + lap, endO = O + lap;
  pdl_wait();
  double vm = ld(O + (I)cm * str), p = ld(se), x = ld(so), y = ld(le);
  charge_link(vm, p, zm, a.rms, a.invchi);
  for (int q = len >> 1; q > 0; --q) {
    I no = so + adv;
    le += adv;
    bool over = false;
    if (WRAP) {
      over = no >= endO;
      if (over) no -= lap;
      if (le >= endE) le -= lap;
    }
    double xn = 0, yn = 0;
    if (q > 1) {
      xn = ld(no);
      yn = ld(le);
    }
    charge_link(x, y, z1, a.rms, a.invchi);
    charge_link(p, x, z2, a.rms, a.invchi);
    st(se, p);
    st(so, x);
    p = y;
    x = xn;
    y = yn;
    se += adv;
    so = no;
    z2 += dz;
    z1 += dz;
    if (WRAP && over) z1 -= zlap;
  }
}

constexpr int kRunThreads = 128;

// Thread = site of the plane across the direction (lanes along m of one x
// parity), blockIdx.y = run, blockIdx.z = charge.
template <int DIR, typename I>
__global__ void __launch_bounds__(kRunThreads) charge_run_kernel(Geo g, ChargeDirArgs a, int seg) {
  pdl_launch();
  const unsigned idx = blockIdx.x * kRunThreads + threadIdx.x;
  const int N = g.N, L = g.zrev ? 5 - (int)blockIdx.z : (int)blockIdx.z;
  const int q = (int)(idx / (unsigned)N), t = (int)(idx - (unsigned)q * N);
  if (q >= N) return;
  const int o = g.zrev ? N - 1 - q : q, s = t >= g.H ? 1 : 0, i = 2 * (t - s * g.H) + s;
  const int c0 = (int)blockIdx.y * seg, len = min(seg, N - c0);
  if (c0 + len < N) charge_run<DIR, false, I>(g, L, i, o, c0, len, a);
  else charge_run<DIR, true, I>(g, L, i, o, c0, len, a);
}

// x.  A block holds whole rows (blockDim.x = N/2, blockDim.y rows) of charges
// L0 .. L0 + nl - 1, one after the other.  Thread m of a row holds the pair of
// sites that first-face link m joins, A and B; the second-face link joins its B
// with the A of thread m + 1, which comes through shared memory (two slots in
// turn, so one barrier per charge), and the thread writes both.
__device__ __forceinline__ void charge_row(const Geo &g, int L0, int nl, int m, int row, bool valid,
                                           const ChargeDirArgs &a, double *sh, int slot) {
  const int N = g.N, H = g.H;
  const int j = row % N, k = row / N, b = (a.eo[0] ^ (j + k)) & 1;  // A of link m is site 2m + b
  const int xb = 2 * m + b + 1 == N ? 0 : 2 * m + b + 1, mn = m + 1 == H ? 0 : m + 1;
  const long long r = (long long)row * H;
  const long long oa = (long long)a.eo[0] * g.V2 + r, ob = (long long)a.eo[1] * g.V2 + r + (xb >> 1);
  const uint64_t nat = (uint64_t)row * N;
  uint64_t z1 = a.sk[0] + (6 * (nat + 2 * m + b) + L0 + 1) * kGolden;
  uint64_t z2 = a.sk[1] + (6 * (nat + xb) + L0 + 1) * kGolden;
  const double *ia = a.in + L0 * a.pitch_in + oa + m, *ib = a.in + L0 * a.pitch_in + ob;
  double *wa = a.out + L0 * a.pitch_out + oa + mn, *wb = a.out + L0 * a.pitch_out + ob;
  pdl_wait();
  double an = 0, bn = 0;
  if (valid) {
    an = *ia;
    bn = *ib;
  }
  for (int l = 0; l < nl; ++l) {
    double A = an, B = bn;
    ia += a.pitch_in;
    ib += a.pitch_in;
    if (valid && l + 1 < nl) {
      an = *ia;
      bn = *ib;
    }
    charge_link(A, B, z1, a.rms, a.invchi);
    double *s = sh + (l & 1) * slot;
    s[m] = A;
    __syncthreads();
    A = s[mn];
    charge_link(B, A, z2, a.rms, a.invchi);
    if (valid) {
      *wb = B;
      *wa = A;
    }
    wa += a.pitch_out;
    wb += a.pitch_out;
    z1 += kGolden;
    z2 += kGolden;
  }
}

__global__ void __launch_bounds__(1024) charge_row_kernel(Geo g, ChargeDirArgs a, int nl) {
  extern __shared__ double xs[];  // [2][blockDim.y][H]
  pdl_launch();
  const int rows = g.N * g.N, id = blockIdx.x * blockDim.y + threadIdx.y;
  const int L0 = nl * (g.zrev ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y);
  const bool valid = id < rows;
  const int row = valid ? (g.zrev ? rows - 1 - id : id) : 0;
  charge_row(g, L0, nl, threadIdx.x, row, valid, a, xs + (size_t)threadIdx.y * g.H, blockDim.y * g.H);
}

// ----------------------------------------------------------------------------
// Blocks of the kernels that visit all sites: 256 threads cover 128 consecutive
// (j, m) elements of a plane, threads 0..127 in the even and 128..255 in the odd
// half.  Grid (ceil(N H / 128), planes).
constexpr int kSiteThreads = 256;
// resident blocks per SM of the Euler-Maruyama step with sums, its adjoint and the ideal step's adjoint (48, 80 and
// 86-128 registers)
constexpr int kEmBlocks = 5, kEmAdjBlocks = 3, kIdealAdjBlocks = 2;

__device__ __forceinline__ bool all_site(const Geo &g, int chunk, int &parity, int &m, int &j) {
  parity = threadIdx.x >> 7;
  const unsigned t = chunk * 128 + (threadIdx.x & 127), H = (unsigned)g.H;
  const unsigned jj = t / H;
  m = (int)(t - jj * H);
  j = (int)jj;
  return j < g.N;
}

inline dim3 site_grid(const Geo &g) { return dim3((unsigned)(((long long)g.N * g.H + 127) / 128), g.Nz); }

// The four normals of site nat in the sub-step of key sk.
__device__ __forceinline__ void site_normals(uint64_t sk, long long nat, double (&xi)[4]) {
  Xoro rng = stream_at(sk, (uint64_t)nat);
  const uint64_t r1 = rng.next(), r2 = rng.next(), r3 = rng.next(), r4 = rng.next();
  box_muller(r1, r2, xi[0], xi[1]);
  box_muller(r3, r4, xi[2], xi[3]);
}

// Euler-Maruyama Model A step at one site (Jacobi: reads `in`, writes phi of
// `out`); acc: the new phi.  The noise is drawn before the wait for the previous
// kernel.  I: the element offset type (int when idx32 holds).
template <bool INJECTED, typename I>
__device__ __forceinline__ void em_site(const Fields &in, const Fields &out, const Geo &g, const EmArgs &a, int parity,
                                        int m, int j, int k, double (&acc)[4]) {
  const long long nat = (long long)nat_index_t<I>(g, 2 * m + ((parity + j + k) & 1), j, k);
  double xi[4];
  if (!INJECTED) site_normals(a.sk, nat, xi);
  const Nbrs<I> o = nbrs_of<I>(g, parity, m, j, k);
  pdl_wait();
  if (INJECTED) {
#pragma unroll
    for (int l = 0; l < 4; ++l) xi[l] = a.xi[(long long)l * global_sites(g) + nat];
  }
  double c[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) c[l] = *at(in.c[l], o.own);
  const double p2 = c[0] * c[0] + c[1] * c[1] + c[2] * c[2] + c[3] * c[3];
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    double fo = -nbr_sum(in.c[l], o) + a.c6 * c[l] + a.lambda * p2 * c[l];
    if (l == 0) fo -= a.H;
    acc[l] = c[l] - a.dtg * fo + a.sq * xi[l];
    *at(out.c[l], o.own) = acc[l];
  }
}

// SUM: also the sums of the new phi, a row per block.  NB: resident blocks per SM.
template <bool INJECTED, bool SUM, typename I, int NB = kEmBlocks>
__global__ void __launch_bounds__(kSiteThreads, NB) em_kernel(Fields in, Fields out, Geo g, EmArgs a, double *partial) {
  pdl_launch();
  int parity, m, j;
  double acc[4] = {0, 0, 0, 0};
  if (all_site(g, blockIdx.x, parity, m, j)) em_site<INJECTED, I>(in, out, g, a, parity, m, j, blockIdx.y, acc);
  if (SUM) block_sum4<kSiteThreads>(acc, partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 4);
}

// Adjoint of the Euler-Maruyama step at one site (see em_adjoint_kernel); v: its
// shares of the parameter sums.  gl: the loss gradient added to the adjoint.
template <typename I, typename GL>
__device__ __forceinline__ void em_adjoint_site(const Fields &phi, const Fields &lin, const Fields &lout, const Geo &g,
                                                const EmAdjArgs &a, int parity, int m, int j, int k, GL gl,
                                                double (&v)[4]) {
  const long long nat = (long long)nat_index_t<I>(g, 2 * m + ((parity + j + k) & 1), j, k);
  double xi[4];
  site_normals(a.sk, nat, xi);
  const Nbrs<I> o = nbrs_of<I>(g, parity, m, j, k);
  pdl_wait();
  double c[4], l[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    c[b] = *at(phi.c[b], o.own);
    l[b] = *at(lin.c[b], o.own);
  }
  const double p2 = c[0] * c[0] + c[1] * c[1] + c[2] * c[2] + c[3] * c[3];
  const double dot = c[0] * l[0] + c[1] * l[1] + c[2] * l[2] + c[3] * l[3];
  double gg = 0;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const double hf = nbr_sum(phi.c[b], o), nl = nbr_sum(lin.c[b], o);
    const double jl = a.c6 * l[b] + a.lambda * (p2 * l[b] + 2.0 * c[b] * dot) - nl;
    *at(lout.c[b], o.own) = l[b] - a.dtg * jl + gl(b);
    double F = -hf + a.c6 * c[b] + a.lambda * p2 * c[b];
    if (b == 0) F -= a.H;
    gg += l[b] * (-a.dt * F + a.cxi * xi[b]);
  }
  v[0] = -a.dtg * dot;
  v[1] = -a.dtg * p2 * dot;
  v[2] = a.dtg * l[0];
  v[3] = gg;
}

// ----------------------------------------------------------------------------
// Fused ideal step (IdealPV2::step_no_reject, Stepper.cxx:68-176).
// A CTA owns a TX x TY column of sites and marches up a z-chunk.  At plane p
// it rotates phi by the half step (phi') for its sites and a one-site ring
// into shared memory (3 rotating plane buffers); for plane p-1 it advects the
// charges with the 7-point stencil on phi', applies the second half rotation
// with the updated charges and writes the site to `out`.  The 10 components
// of plane p+1 arrive by cp.async while plane p computes.  Each site is read
// once (80 B) and written once (80 B).
template <int TX, int TY>
struct IdealTile {
  static constexpr int SX = TX + 2, SY = TY + 2, SP = SX * SY;
  static constexpr int NHALO = 2 * SX + 2 * TY;
  static constexpr size_t SMEM = (size_t)(2 * 10 * SP + 3 * 4 * SP) * sizeof(double);
};

template <int TX, int TY>
__device__ __forceinline__ void ideal_tile(const Fields &in, const Fields &out, const Geo &g, int zchunk,
                                           const IdealArgs &a, int bx, int by, int bz) {
  using T = IdealTile<TX, TY>;
  constexpr int SX = T::SX, SY = T::SY, SP = T::SP, NHALO = T::NHALO;
  static_assert(NHALO <= TX * TY, "halo ring larger than the CTA");
  extern __shared__ double smem[];
  double *raw = smem;               // [2 stages][10][SP]
  double *phs = raw + 2 * 10 * SP;  // [3][4][SP]
  const int N = g.N;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int x0 = bx * TX, y0 = by * TY;
  const int z0 = bz * zchunk;
  const int z1 = min(z0 + zchunk, g.Nz);
  const int nit = (z1 - z0) + 2;
  const bool act = (x0 + tx < N) && (y0 + ty < N);
  const int xi = (x0 + tx) % N, yj = (y0 + ty) % N;
  const int sc = (ty + 1) * SX + tx + 1;

  int hs = -1, hxg = 0, hyg = 0;
  if (threadIdx.x < NHALO) {
    const int h = threadIdx.x;
    int hx, hy;
    if (h < SX) { hx = h; hy = 0; }
    else if (h < 2 * SX) { hx = h - SX; hy = SY - 1; }
    else if (h < 2 * SX + TY) { hx = 0; hy = 1 + (h - 2 * SX); }
    else { hx = SX - 1; hy = 1 + (h - 2 * SX - TY); }
    hs = hy * SX + hx;
    hxg = wrapn(x0 - 1 + hx, N);
    hyg = wrapn(y0 - 1 + hy, N);
  }

  // Planes z0-1 .. z1 of the march, tracked incrementally (within two wraps
  // of the buffer: nit <= Nz + 2), and rb_off split into its in-plane part
  // and plane part, so the march does no integer division.
  const int zfirst = z0 == 0 ? g.Nz - 1 : z0 - 1;
  auto plane_of = [&](int q) {
    int pl = zfirst + q;
    if (pl >= g.Nz) pl -= g.Nz;
    if (pl >= g.Nz) pl -= g.Nz;
    return pl;
  };
  const long long NH = (long long)N * g.H;
  const int own_xy = yj * g.H + (xi >> 1), own_par = (xi + yj) & 1;
  const int ring_xy = hyg * g.H + (hxg >> 1), ring_par = (hxg + hyg) & 1;
  auto issue = [&](int plane, int stage, bool halo) {
    const long long o = (long long)((own_par + plane) & 1) * g.V2 + (long long)plane * NH + own_xy;
#pragma unroll
    for (int c = 0; c < 10; ++c) cp_async8(&raw[(stage * 10 + c) * SP + sc], in.c[c] + o);
    if (halo && hs >= 0) {
      const long long oh = (long long)((ring_par + plane) & 1) * g.V2 + (long long)plane * NH + ring_xy;
#pragma unroll
      for (int c = 0; c < 10; ++c) cp_async8(&raw[(stage * 10 + c) * SP + hs], in.c[c] + oh);
    }
  };

  issue(zfirst, 0, false);
  cp_async_commit();

  double pm[4], pc[4], pn[4], qc[6], qn[6];
  int pprev = zfirst;  // plane p - 1 (used from it >= 2)
  for (int it = 0; it < nit; ++it) {
    const int p = plane_of(it);
    cp_async_wait_all();
    __syncthreads();
    if (it + 1 < nit) issue(plane_of(it + 1), (it + 1) & 1, true);
    cp_async_commit();

    const double *rw = raw + (it & 1) * 10 * SP;
    double *ph = phs + (it % 3) * 4 * SP;
#pragma unroll
    for (int l = 0; l < 4; ++l) pn[l] = rw[l * SP + sc];
#pragma unroll
    for (int s = 0; s < 6; ++s) qn[s] = rw[(4 + s) * SP + sc];
    rotate_site(pn, qn, a.dto2chi);
#pragma unroll
    for (int l = 0; l < 4; ++l) ph[l * SP + sc] = pn[l];
    if (hs >= 0 && it >= 1) {
      double phh[4], qh[6];
#pragma unroll
      for (int l = 0; l < 4; ++l) phh[l] = rw[l * SP + hs];
#pragma unroll
      for (int s = 0; s < 6; ++s) qh[s] = rw[(4 + s) * SP + hs];
      rotate_site(phh, qh, a.dto2chi);
#pragma unroll
      for (int l = 0; l < 4; ++l) ph[l * SP + hs] = phh[l];
    }

    if (it >= 2 && act) {
      const double *pp = phs + ((it + 2) % 3) * 4 * SP;  // phi' of plane p-1 (written last iteration)
      double xp[4], xm[4], yp[4], ym[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        xp[l] = pp[l * SP + sc + 1];
        xm[l] = pp[l * SP + sc - 1];
        yp[l] = pp[l * SP + sc + SX];
        ym[l] = pp[l * SP + sc - SX];
      }
      const double *c = pc, *zp = pn, *zm = pm;
      double S[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) S[l] = ((xp[l] + xm[l]) + (yp[l] + ym[l])) + (zp[l] + zm[l]);
      charge_currents(c, S, a.dt, a.a2, a.H, qc);
      // second half rotation on a copy: pc (phi') stays the z-1 neighbour of the next plane
      double pf[4] = {pc[0], pc[1], pc[2], pc[3]};
      rotate_site(pf, qc, a.dto2chi);
      const long long o = (long long)((own_par + pprev) & 1) * g.V2 + (long long)pprev * NH + own_xy;
#pragma unroll
      for (int l = 0; l < 4; ++l) out.c[l][o] = pf[l];
#pragma unroll
      for (int s = 0; s < 6; ++s) out.c[4 + s][o] = qc[s];
    }
    pprev = p;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      pm[l] = pc[l];
      pc[l] = pn[l];
    }
#pragma unroll
    for (int s = 0; s < 6; ++s) qc[s] = qn[s];
  }
}

template <int TX, int TY>
__global__ void __launch_bounds__(TX *TY, 2) ideal_kernel(Fields in, Fields out, Geo g, int zchunk, IdealArgs a) {
  pdl_launch();
  pdl_wait();
  ideal_tile<TX, TY>(in, out, g, zchunk, a, blockIdx.x, blockIdx.y,
                    g.zrev ? (int)(gridDim.z - 1 - blockIdx.z) : (int)blockIdx.z);
}

// ----------------------------------------------------------------------------
// Energy (IdealPV2::computeEnergy, Stepper.cxx:204-268): forward differences.
__global__ void energy_kernel(Fields f, Geo g, double *partial) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double grad2 = 0, nab2 = 0, hphi = 0;
  if (t < 2 * g.V2) {
    const int N = g.N;
    const long long n = t;
    const int i = (int)(n % N);
    const long long r = n / N;
    const int j = (int)(r % N), k = (int)(r / N);
    const long long o = rb_off(g, i, j, k);
    const long long ox = rb_off(g, wrap_inc(i, N), j, k);
    const long long oy = rb_off(g, i, wrap_inc(j, N), k);
    const long long oz = rb_off(g, i, j, wrap_inc(k, N));
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const double pm = f.c[s][o];
      const double a = f.c[s][oz] - pm, b = f.c[s][oy] - pm, c = f.c[s][ox] - pm;
      grad2 += a * a + b * b + c * c;
    }
    hphi = f.c[0][o];
#pragma unroll
    for (int s = 0; s < 6; ++s) nab2 += f.c[4 + s][o] * f.c[4 + s][o];
  }
  __shared__ double s3[3][kThreads / 32];
  warp_sum(grad2);
  warp_sum(nab2);
  warp_sum(hphi);
  if ((threadIdx.x & 31) == 0) {
    s3[0][threadIdx.x >> 5] = grad2;
    s3[1][threadIdx.x >> 5] = nab2;
    s3[2][threadIdx.x >> 5] = hphi;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t2 = 0;
    for (int w = 0; w < kThreads / 32; ++w) t2 += s3[threadIdx.x][w];
    partial[(long long)blockIdx.x * 3 + threadIdx.x] = t2;
  }
}

__global__ void energy_final_kernel(const double *partial, int nblk, double H, double half_over_chi,
                                    double *out) {
  __shared__ double s[3];
  const int c = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (c < 3) {
    double t = 0;
    for (int b = l; b < nblk; b += 32) t += partial[(long long)b * 3 + c];
    warp_sum(t);
    if (l == 0) s[c] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) out[0] = half_over_chi * s[1] + 0.5 * s[0] - H * s[2];
}

// ----------------------------------------------------------------------------
// Measurer.  The 25 per-site observables: 11 of computeSliceAverage
// (phi_a, A, V, phi^2; measurer.cxx:46-69) then 14 of computeSliceAveragePhase
// (sigma, n_a, A_a, V_a, sigma^2; measurer.cxx:152-192).
constexpr int kNObs = 25;

__device__ __forceinline__ void site_obs(const double f[10], double o[kNObs]) {
  double phi2 = 0.0;
#pragma unroll
  for (int l = 0; l < 10; ++l) o[l] = f[l];
#pragma unroll
  for (int l = 0; l < 4; ++l) phi2 += f[l] * f[l];
  o[10] = phi2;
  const double sigma = sqrt(phi2);
  double n[4];
  if (phi2 > 100. * 2.2250738585072014e-308) {
    // one division instead of four (equal to phi_a / sigma up to an ulp)
    const double inv = 1.0 / sigma;
#pragma unroll
    for (int l = 0; l < 4; ++l) n[l] = f[l] * inv;
  } else {
    n[0] = 1;
    n[1] = n[2] = n[3] = 0;
  }
  const double *rho = f + 4;  // (A1..3, V1..3)
  // contract_rho(n, rho) and contract_rho(n, dual rho) (measurer.cxx:101-114)
  const double A0 = -(n[1] * rho[0]) - n[2] * rho[1] - n[3] * rho[2];
  const double A1 = n[0] * rho[0] + n[3] * rho[4] - n[2] * rho[5];
  const double A2 = n[0] * rho[1] - n[3] * rho[3] + n[1] * rho[5];
  const double A3 = n[0] * rho[2] + n[2] * rho[3] - n[1] * rho[4];
  const double V0 = -(n[1] * rho[3]) - n[2] * rho[4] - n[3] * rho[5];
  const double V1 = n[0] * rho[3] + n[3] * rho[1] - n[2] * rho[2];
  const double V2 = n[0] * rho[4] - n[3] * rho[0] + n[1] * rho[2];
  const double V3 = n[0] * rho[5] + n[2] * rho[0] - n[1] * rho[1];
  o[11] = sigma;
#pragma unroll
  for (int l = 0; l < 4; ++l) o[12 + l] = n[l];
  o[16] = A0; o[17] = A1; o[18] = A2; o[19] = A3;
  o[20] = V0; o[21] = V1; o[22] = V2; o[23] = V3;
  o[24] = sigma * sigma;
}

__device__ __forceinline__ void load_site(const Fields &f, const Geo &g, int i, int j, int k, double s[10]) {
  const long long o = rb_off(g, i, j, k);
#pragma unroll
  for (int L = 0; L < 10; ++L) s[L] = f.c[L][o];
}

// T[o][kout + k - klo][i] = sum_j obs(i, j, k) for local planes k in [klo, klo + nk);
// T is [25][Ng][N]
__global__ void meas_sum_j_kernel(Fields f, Geo g, double *T, int klo, int nk, int kout) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int N = g.N;
  if (t >= (long long)N * nk) return;
  const int i = (int)(t % N), kl = (int)(t / N), k = klo + kl;
  double acc[kNObs];
#pragma unroll
  for (int o = 0; o < kNObs; ++o) acc[o] = 0;
  for (int j = 0; j < N; ++j) {
    double s[10], ob[kNObs];
    load_site(f, g, i, j, k, s);
    site_obs(s, ob);
#pragma unroll
    for (int o = 0; o < kNObs; ++o) acc[o] += ob[o];
  }
  const long long NT = (long long)g.Ng * N;
#pragma unroll
  for (int o = 0; o < kNObs; ++o) T[o * NT + (long long)(kout + kl) * N + i] = acc[o];
}

// U[o][j][i] = sum_k obs(i, j, k) over local planes [klo, klo + nk)
__global__ void meas_sum_k_kernel(Fields f, Geo g, double *U, int klo, int nk) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int N = g.N;
  if (t >= (long long)N * N) return;
  const int i = (int)(t % N), j = (int)(t / N);
  double acc[kNObs];
#pragma unroll
  for (int o = 0; o < kNObs; ++o) acc[o] = 0;
  for (int k = klo; k < klo + nk; ++k) {
    double s[10], ob[kNObs];
    load_site(f, g, i, j, k, s);
    site_obs(s, ob);
#pragma unroll
    for (int o = 0; o < kNObs; ++o) acc[o] += ob[o];
  }
  const long long NN = (long long)N * N;
#pragma unroll
  for (int o = 0; o < kNObs; ++o) U[o * NN + (long long)j * N + i] = acc[o];
}

struct MeasOut {
  double *oavg;
  double *wall[3], *wk[3], *wkr[3], *ph[3], *phk[3];
};

__host__ __device__ inline MeasOut meas_layout(double *base, int N) {
  const int NK = N / 2 + 1;
  MeasOut m;
  double *p = base;
  m.oavg = p;
  p += 11;
  for (int a = 0; a < 3; ++a) { m.wall[a] = p; p += 11 * N; }
  for (int a = 0; a < 3; ++a) { m.wk[a] = p; p += 11 * NK * 2; }
  for (int a = 0; a < 3; ++a) { m.wkr[a] = p; p += 14 * NK * 2; }
  for (int a = 0; a < 3; ++a) { m.ph[a] = p; p += 14 * N; }
  for (int a = 0; a < 3; ++a) { m.phk[a] = p; p += 14 * NK * 2; }
  return m;
}

// walls: axis 0 (X): sum_k T[o][k][i]; axis 2 (Z): sum_i T[o][k][i];
// axis 1 (Y): sum_i U[o][j][i]; divided by N^2 (measurer.cxx:78-80).
__global__ void meas_walls_kernel(const double *T, const double *U, int N, MeasOut mo) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * kNObs * N) return;
  const int pos = t % N;
  const int o = (t / N) % kNObs;
  const int axis = t / (N * kNObs);
  const long long NN = (long long)N * N;
  double s = 0;
  if (axis == 0) {
    for (int k = 0; k < N; ++k) s += T[o * NN + (long long)k * N + pos];
  } else if (axis == 2) {
    for (int i = 0; i < N; ++i) s += T[o * NN + (long long)pos * N + i];
  } else {
    for (int i = 0; i < N; ++i) s += U[o * NN + (long long)pos * N + i];
  }
  s /= (double)(N * N);
  if (o < 11) mo.wall[axis][o * N + pos] = s;
  else mo.ph[axis][(o - 11) * N + pos] = s;
}

// rotate_to_vev (measurer.cxx:231-286), complex arithmetic as the reference.
// One mode kk of one axis: w its k walls, o its rotated k walls.
__device__ __forceinline__ void rotate_mode(const double *w, double *o, int NK, int kk) {
  // the walls may come from other blocks of this launch (meas_finish_kernel): read at L2
  auto re = [&](int a, int k) { return __ldcg(w + (a * NK + k) * 2); };
  auto im = [&](int a, int k) { return __ldcg(w + (a * NK + k) * 2 + 1); };
  double nr[4], ni[4];
  double nrm = 0;
  for (int a = 0; a < 4; ++a) {
    nr[a] = re(a, 0);
    ni[a] = im(a, 0);
    nrm += nr[a] * nr[a] + ni[a] * ni[a];
  }
  nrm = sqrt(nrm);
  if (nrm < 2.2250738585072014e-308) {
    nr[0] = 1; ni[0] = 0;
    for (int a = 1; a < 4; ++a) nr[a] = ni[a] = 0;
  } else {
    for (int a = 0; a < 4; ++a) { nr[a] /= nrm; ni[a] /= nrm; }
  }
  double pr[4], pi[4], rr[6], ri[6];
  for (int a = 0; a < 4; ++a) { pr[a] = re(a, kk); pi[a] = im(a, kk); }
  for (int b = 0; b < 6; ++b) { rr[b] = re(4 + b, kk); ri[b] = im(4 + b, kk); }
  // phis = sum_a n_a phi_a (complex, no conjugation)
  double sr = 0, si = 0;
  for (int a = 0; a < 4; ++a) {
    sr += nr[a] * pr[a] - ni[a] * pi[a];
    si += nr[a] * pi[a] + ni[a] * pr[a];
  }
  auto put = [&](int a, double x, double y) { o[(a * NK + kk) * 2] = x; o[(a * NK + kk) * 2 + 1] = y; };
  put(0, sr, si);
  for (int a = 0; a < 4; ++a) {
    // phir = phi - n * phis
    put(1 + a, pr[a] - (nr[a] * sr - ni[a] * si), pi[a] - (nr[a] * si + ni[a] * sr));
  }
  // complex products c = n_a * rho_b
#define CMR(a, b) (nr[a] * rr[b] - ni[a] * ri[b])
#define CMI(a, b) (nr[a] * ri[b] + ni[a] * rr[b])
  // contract_rho(n, rho)
  put(5, -CMR(1, 0) - CMR(2, 1) - CMR(3, 2), -CMI(1, 0) - CMI(2, 1) - CMI(3, 2));
  put(6, CMR(0, 0) + CMR(3, 4) - CMR(2, 5), CMI(0, 0) + CMI(3, 4) - CMI(2, 5));
  put(7, CMR(0, 1) - CMR(3, 3) + CMR(1, 5), CMI(0, 1) - CMI(3, 3) + CMI(1, 5));
  put(8, CMR(0, 2) + CMR(2, 3) - CMR(1, 4), CMI(0, 2) + CMI(2, 3) - CMI(1, 4));
  // contract_rho(n, dualize_rho(rho)), dual = (rho3..5, rho0..2)
  put(9, -CMR(1, 3) - CMR(2, 4) - CMR(3, 5), -CMI(1, 3) - CMI(2, 4) - CMI(3, 5));
  put(10, CMR(0, 3) + CMR(3, 1) - CMR(2, 2), CMI(0, 3) + CMI(3, 1) - CMI(2, 2));
  put(11, CMR(0, 4) - CMR(3, 0) + CMR(1, 2), CMI(0, 4) - CMI(3, 0) + CMI(1, 2));
  put(12, CMR(0, 5) + CMR(2, 0) - CMR(1, 1), CMI(0, 5) + CMI(2, 0) - CMI(1, 1));
#undef CMR
#undef CMI
  put(13, re(10, kk), im(10, kk));
}

__global__ void meas_rotate_kernel(int N, MeasOut mo) {
  const int NK = N / 2 + 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * NK) return;
  rotate_mode(mo.wk[t / NK], mo.wkr[t / NK], NK, t % NK);
}

constexpr int kWallThreads = 256;   // block of meas_dft_kernel
constexpr int kFinishThreads = 512;  // block of meas_finish_kernel

// OAverage[l] = mean_x wallX(l, x) (measurer.cxx:292-300) and the r2c DFT of
// one wall row (lgv_dft.cuh), W(k) = (1/N) sum_x W(x) e^{-2 pi i k x / N}, k =
// 0..N/2, by one block: `row` is the row in shared memory, after a barrier.
__device__ __forceinline__ void wall_modes(const double *row, const dft::Plan &p, double2 *tw, double2 *Z, int axis,
                                           int o, const MeasOut &mo) {
  const int N = p.N, NK = N / 2 + 1;
  if (axis == 0 && o < 11 && threadIdx.x < 32) {
    double s = 0;
    for (int i = threadIdx.x; i < N; i += 32) s += row[i];
    warp_sum(s);
    if (threadIdx.x == 0) mo.oavg[o] = s / (double)N;
  }
  for (int u = threadIdx.x; u < p.K1 * p.N2; u += blockDim.x) {
    const int k1[1] = {u / p.N2}, n2 = u - k1[0] * p.N2;
    double2 z[1];
    dft::inner<1>(row + n2, p, tw, n2, k1, z);
    Z[u] = z[0];
  }
  __syncthreads();
  double *dst = (o < 11) ? mo.wk[axis] + (size_t)o * NK * 2 : mo.phk[axis] + (size_t)(o - 11) * NK * 2;
  const int n2h = p.N2 / 2 + 1;
  for (int u = threadIdx.x; u < p.K1 * n2h; u += blockDim.x) {
    const int k1 = u / n2h, k2[1] = {u - k1 * n2h};
    double2 W[1], M[1];
    dft::outer<1>(Z + k1 * p.N2, p, tw, k2, W, M);
    dft::store(p, k1, k2[0], W[0], dst);
    if (k2[0] > 0 && 2 * k2[0] < p.N2) dft::store(p, k1, p.N2 - k2[0], M[0], dst);
  }
}

// dynamic shared memory of a block that transforms one row
inline size_t wall_smem(const dft::Plan &p) {
  return ((size_t)p.N + (size_t)p.K1 * p.N2) * sizeof(double2) + (size_t)p.N * sizeof(double);
}

// The modes of every wall row already in place; block = (row o, axis).
__global__ void __launch_bounds__(kWallThreads) meas_dft_kernel(dft::Plan p, MeasOut mo) {
  extern __shared__ __align__(16) double2 sm2[];
  double2 *tw = sm2, *Z = sm2 + p.N;
  double *row = (double *)(Z + p.K1 * p.N2);
  const int o = blockIdx.x, axis = blockIdx.y;
  const double *src = (o < 11) ? mo.wall[axis] + (size_t)o * p.N : mo.ph[axis] + (size_t)(o - 11) * p.N;
  dft::fill_twiddles(tw, p.N);
  for (int x = threadIdx.x; x < p.N; x += kWallThreads) row[x] = src[x];
  __syncthreads();
  wall_modes(row, p, tw, Z, axis, o, mo);
}

// ---- one-pass measurement ----------------------------------------------------
// The 25 observables of every site are formed once and summed towards all
// three axes: a block takes a brick of 32 sites in x (lanes) by TJ rows by 8
// planes (warps).  A thread adds its site's observables over the rows (towards
// x); each row of 32 sites goes through a warp's own [25][32] table in shared
// memory, where lane l adds the row of observable l (towards y; a butterfly of
// shuffles cost 2.3 times the instructions); and the sums over rows, added
// over the lanes once at the end the same way, go towards z.  Each brick
// writes its share of the walls and meas_finish_kernel adds the bricks in a
// fixed order.  The two passes it replaces read the state twice and had N^2
// threads, each adding N sites in a chain: a measurement took 92 us at 32^3,
// 157 at 64^3, 295 at 120^3, 395 at 160^3 and 725 at 256^3; now 19, 25, 83,
// 141 and 468.  It is bound by shared-memory bandwidth (73 % of the wavefronts
// at 120^3) and the 24 % of the warps that its 128 registers leave.
constexpr int kMtI = 32, kMtK = 8, kMtRows = 8, kMtLanes = 32;
constexpr int kMtW = 34;  // doubles per table row: an odd number of 16-byte words, lanes on distinct banks
constexpr size_t kMtSmem = (size_t)kMtK * (kNObs * kMtW + kMtRows * kMtLanes) * sizeof(double);

struct MeasTiles {
  int it, jt, kt, tj;
  __host__ __device__ int npart(int axis) const { return axis == 0 ? kt * jt : axis == 1 ? kt * it : jt * it; }
  __host__ __device__ int pitch(int axis) const { return axis == 0 ? it * kMtI : axis == 1 ? jt * tj : kt * kMtK; }
  // doubles of the shares towards `axis`
  __host__ __device__ size_t len(int axis) const { return (size_t)kNObs * npart(axis) * pitch(axis); }
};

// Rows per brick: as many as leave two bricks per SM, since a brick's shares
// cost 1100 to 1900 doubles whatever its rows; at least 4.
inline MeasTiles meas_tiles(int N) {
  MeasTiles t;
  t.it = (N + kMtI - 1) / kMtI;
  t.kt = (N + kMtK - 1) / kMtK;
  for (t.tj = 32; t.tj > 4; t.tj >>= 1)
    if (t.it * t.kt * ((N + t.tj - 1) / t.tj) >= 2 * 148) break;
  t.jt = (N + t.tj - 1) / t.tj;
  return t;
}

// Sum over the warp of v[0..24] through its table: lane l < 25 returns the sum of v[l].
__device__ __forceinline__ double warp_sum25(const double (&v)[kNObs], double *tab, int lane) {
  __syncwarp();
#pragma unroll
  for (int o = 0; o < kNObs; ++o) tab[o * kMtW + lane] = v[o];
  __syncwarp();
  const double2 *r = (const double2 *)(tab + min(lane, kNObs - 1) * kMtW);
  double a[4] = {0, 0, 0, 0};
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const double2 t = r[q];
    a[q & 3] += t.x + t.y;
  }
  return (a[0] + a[1]) + (a[2] + a[3]);
}

__global__ void __launch_bounds__(256, 2) meas_tile_kernel(Fields f, Geo g, MeasTiles mt, double *__restrict__ xp,
                                                        double *__restrict__ yp, double *__restrict__ zp) {
  extern __shared__ __align__(16) double2 sm2[];
  pdl_launch();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *tab = (double *)sm2 + (size_t)warp * kNObs * kMtW;       // [warp][25][kMtW]
  double *ys = (double *)sm2 + (size_t)kMtK * kNObs * kMtW;        // [warp][row][lane]
  const int ix = blockIdx.x, jy = blockIdx.y, kz = blockIdx.z;
  const int N = g.N, i = ix * kMtI + 2 * (lane & 15) + (lane >> 4);  // a half warp's sites share the x parity
  const int k = kz * kMtK + warp, j0 = jy * mt.tj, j1 = min(j0 + mt.tj, N);
  const bool own = i < N && k < N;
  const int V2 = (int)g.V2, base = (k * N + j0) * g.H + (i >> 1), par0 = (i + j0 + k) & 1;
  double acc[kNObs], nx[10];
#pragma unroll
  for (int o = 0; o < kNObs; ++o) acc[o] = 0;
  auto load = [&](int j) {
    if (own && j < j1) {
      const int off = ((par0 + j - j0) & 1) * V2 + base + (j - j0) * g.H;
#pragma unroll
      for (int L = 0; L < 10; ++L) nx[L] = f.c[L][off];
    }
  };
  load(j0);
  for (int jc = j0; jc < j1; jc += kMtRows) {
    const int rows = min(min(kMtRows, mt.tj), j1 - jc);
    for (int jj = 0; jj < rows; ++jj) {
      double s[10], ob[kNObs];
#pragma unroll
      for (int L = 0; L < 10; ++L) s[L] = nx[L];
      load(jc + jj + 1);
      if (own) {
        site_obs(s, ob);
      } else {
#pragma unroll
        for (int o = 0; o < kNObs; ++o) ob[o] = 0;
      }
#pragma unroll
      for (int o = 0; o < kNObs; ++o) acc[o] += ob[o];
      ys[(warp * kMtRows + jj) * kMtLanes + lane] = warp_sum25(ob, tab, lane);
    }
    __syncthreads();
    const size_t P = mt.npart(1), pitch = mt.pitch(1), q = (size_t)kz * mt.it + ix;
    for (int e = threadIdx.x; e < rows * kMtLanes; e += 256) {
      const int jj = e / kMtLanes, o = e % kMtLanes;
      double t = 0;
#pragma unroll
      for (int w = 0; w < kMtK; ++w) t += ys[(w * kMtRows + jj) * kMtLanes + o];
      if (o < kNObs) yp[((size_t)o * P + q) * pitch + jc + jj] = t;
    }
    __syncthreads();
  }
  const double zs = warp_sum25(acc, tab, lane);
  if (lane < kNObs && k < N) zp[((size_t)lane * mt.npart(2) + (size_t)jy * mt.it + ix) * mt.pitch(2) + k] = zs;
  // towards x: the warps' tables hold their sums over rows; thread t adds column t of the 25 x 32 over the planes
  __syncthreads();
  for (int e = threadIdx.x; e < kNObs * 32; e += 256) {
    const int o = e >> 5, l = e & 31, x = ix * kMtI + 2 * (l & 15) + (l >> 4);
    double t = 0;
#pragma unroll
    for (int w = 0; w < kMtK; ++w) t += ((const double *)sm2)[((size_t)w * kNObs + o) * kMtW + l];
    if (x < N) xp[((size_t)o * mt.npart(0) + (size_t)kz * mt.jt + jy) * mt.pitch(0) + x] = t;
  }
}

// Block (o, axis): wall row o towards `axis` from the bricks' shares, each
// position by G groups of threads (fixed order), then its modes; the block that
// ends last of an axis's first 11 rows then rotates that axis's modes.
// done[3]: zero on entry, re-armed.
__global__ void __launch_bounds__(kFinishThreads) meas_finish_kernel(const double *xp, const double *yp,
                                                                    const double *zp, MeasTiles mt, dft::Plan p,
                                                                    int logP, MeasOut mo, unsigned *done) {
  extern __shared__ __align__(16) double2 sm2[];
  __shared__ double part[kFinishThreads];
  __shared__ bool last;
  double2 *tw = sm2, *Z = sm2 + p.N;
  double *row = (double *)(Z + p.K1 * p.N2);
  const int N = p.N, o = blockIdx.x, axis = blockIdx.y;
  const int np = mt.npart(axis), pitch = mt.pitch(axis);
  const double *src = (axis == 0 ? xp : axis == 1 ? yp : zp) + (size_t)o * np * pitch;
  pdl_launch();
  dft::fill_twiddles(tw, N);
  pdl_wait();
  const int P = 1 << logP, G = kFinishThreads >> logP, grp = threadIdx.x >> logP;
  double *dst = (o < 11) ? mo.wall[axis] + (size_t)o * N : mo.ph[axis] + (size_t)(o - 11) * N;
  for (int x0 = 0; x0 < N; x0 += P) {
    const int x = x0 + (threadIdx.x & (P - 1));
    double s = 0;
    if (x < N) {
#pragma unroll 16
      for (int q = grp; q < np; q += G) s += src[q * pitch + x];
    }
    part[threadIdx.x] = s;
    __syncthreads();
    if (grp == 0 && x < N) {
      for (int q = 1; q < G; ++q) s += part[(q << logP) + threadIdx.x];
      s /= (double)(N * N);
      row[x] = s;
      dst[x] = s;
    }
    __syncthreads();
  }
  wall_modes(row, p, tw, Z, axis, o, mo);
  if (o >= 11) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done + axis, 1u) == 10u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int kk = threadIdx.x; kk < N / 2 + 1; kk += kFinishThreads)
    rotate_mode(mo.wk[axis], mo.wkr[axis], N / 2 + 1, kk);
  if (threadIdx.x == 0) done[axis] = 0u;
}

// Sums of the 25 observables over a lattice given in the host-order AoS layout
// u[k][j][i][10] (used by the allocation-free measurement entry point).
// T[o][k][i] = sum_j obs(i, j, k)
__global__ void meas_sum_j_aos_kernel(const double *__restrict__ aos, int N, double *T) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)N * N) return;
  const int i = (int)(t % N), k = (int)(t / N);
  double acc[kNObs];
#pragma unroll
  for (int o = 0; o < kNObs; ++o) acc[o] = 0;
  for (int j = 0; j < N; ++j) {
    const double *src = aos + (((long long)k * N + j) * N + i) * 10;
    double s[10], ob[kNObs];
#pragma unroll
    for (int L = 0; L < 10; ++L) s[L] = src[L];
    site_obs(s, ob);
#pragma unroll
    for (int o = 0; o < kNObs; ++o) acc[o] += ob[o];
  }
  const long long NN = (long long)N * N;
#pragma unroll
  for (int o = 0; o < kNObs; ++o) T[o * NN + (long long)k * N + i] = acc[o];
}

// U[o][j][i] = sum_k obs(i, j, k)
__global__ void meas_sum_k_aos_kernel(const double *__restrict__ aos, int N, double *U) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)N * N) return;
  const int i = (int)(t % N), j = (int)(t / N);
  double acc[kNObs];
#pragma unroll
  for (int o = 0; o < kNObs; ++o) acc[o] = 0;
  for (int k = 0; k < N; ++k) {
    const double *src = aos + (((long long)k * N + j) * N + i) * 10;
    double s[10], ob[kNObs];
#pragma unroll
    for (int L = 0; L < 10; ++L) s[L] = src[L];
    site_obs(s, ob);
#pragma unroll
    for (int o = 0; o < kNObs; ++o) acc[o] += ob[o];
  }
  const long long NN = (long long)N * N;
#pragma unroll
  for (int o = 0; o < kNObs; ++o) U[o * NN + (long long)j * N + i] = acc[o];
}

// ----------------------------------------------------------------------------
// Batched kernels: one launch advances every replica of an ensemble.  The
// flat grid is partitioned into per-replica block ranges (rep[b] is the
// replica of block b, first[r] its first block; the order of the ranges is
// the packing order chosen by the autotuner).  Each block rebuilds its
// replica's arguments exactly as the single-lattice host code does (same
// expressions, no FMA contraction), so a replica evolves bit for bit like a
// lattice of its own; sub-step keys come from the device-resident counter.
// the replica's planes: phi from buffer pphi, charges from buffer pq
__device__ __forceinline__ Fields rep_fields(const RepDesc &r, int pphi, int pq) {
  Fields f;
#pragma unroll
  for (int L = 0; L < 10; ++L) f.c[L] = r.base[L < 4 ? pphi : pq] + (long long)L * r.pstride;
  return f;
}

// The counter and the clock, which the kernel before this one may have written:
// volatile, so that the read stays behind pdl_wait.
__device__ __forceinline__ EnsDyn load_dyn(const EnsDyn *dyn) {
  EnsDyn y;
  y.ctr = *(const volatile unsigned long long *)&dyn->ctr;
  y.t = *(const volatile double *)&dyn->t;
  return y;
}

__device__ __forceinline__ double rep_mass(const RepDesc &r, const EnsDyn &dyn) {
  return __dadd_rn(r.mass0, __dmul_rn(r.dmassdt, dyn.t));
}

// plane kernels: 128 threads cover 128 consecutive (j, m) elements of a plane
__device__ __forceinline__ bool plane_coords(const RepDesc &r, int local, int &m, int &j, int &k) {
  const int chunk = local % r.nchunk;
  k = local / r.nchunk;
  const int t = chunk * 128 + (int)threadIdx.x;
  j = t / r.g.H;
  m = t - j * r.g.H;
  return j < r.g.N;
}

// slab kernels: a block covers 128 consecutive (j, m) elements of kBatchPlanes
// consecutive planes of one replica, so the block-map and descriptor loads
// (two dependent round trips before the first site load) are paid once per
// kBatchPlanes planes
__device__ __forceinline__ bool slab_coords(const RepDesc &r, int local, int lane, int &m, int &j, int &k0) {
  const int chunk = local % r.nchunk;
  k0 = (local / r.nchunk) * kBatchPlanes;
  const int t = chunk * 128 + lane;
  j = t / r.g.H;
  m = t - j * r.g.H;
  return j < r.g.N;
}

// Items of the batched heat-bath and charge sub-steps: block blk of the slab
// map, lane 0..127 of its 128 threads (a kernel of their own, or half of a
// CTA of the persistent step).
__device__ __forceinline__ HbArgs rep_hb_args(const RepDesc &R, const EnsDyn &y, double dt, int ctr_off) {
  HbArgs a{};
  a.rdtg = sqrt(2. * dt * R.gamma);
  a.Lambda2 = 0.5 * (2. * 3. + rep_mass(R, y));
  a.lam4 = R.lambda / 4.;
  a.H = R.H;
  a.sk = sub_key(R.key, y.ctr + (unsigned long long)ctr_off);
  return a;
}

// The planes of a slab block, one after the other: unrolled (the planes' loads
// interleaved) the ensemble step measured 4 % slower.
template <typename I>
__device__ __forceinline__ void batch_hb_planes(const RepDesc &R, int phase, int parity, const HbArgs &a, int m, int j,
                                                int k0) {
  const Fields f = rep_fields(R, phase, phase);
  MonLocal mon;
#pragma unroll 1
  for (int q = 0; q < kBatchPlanes; ++q)
    if (k0 + q < R.g.N) hb_site<false, false, false, I>(f, R.g, parity, a, m, j, k0 + q, mon);
}

template <typename I>
__device__ __forceinline__ void batch_hb_item(const RepDesc *__restrict__ d, const EnsDyn *dyn,
                                              const int *__restrict__ rep, const int *__restrict__ first, int blk,
                                              int lane, int phase, int parity, double dt, int ctr_off) {
  const int r = rep[blk];
  const RepDesc &R = d[r];
  int m, j, k0;
  if (!slab_coords(R, blk - first[r], lane, m, j, k0)) return;
  batch_hb_planes<I>(R, phase, parity, rep_hb_args(R, load_dyn(dyn), dt, ctr_off), m, j, k0);
}

template <typename I>
__global__ void __launch_bounds__(128) batch_hb_kernel(const RepDesc *__restrict__ d, const EnsDyn *dyn,
                                                       const int *__restrict__ rep, const int *__restrict__ first,
                                                       int phase, int parity, double dt, int ctr_off) {
  pdl_launch();
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  int m, j, k0;
  const bool ok = slab_coords(R, blockIdx.x - first[r], threadIdx.x, m, j, k0);
  pdl_wait();  // the previous sub-step writes the fields, the clock kernel *dyn
  __shared__ HbArgs sa;  // once per block: a square root and a key
  if (threadIdx.x == 0) sa = rep_hb_args(R, load_dyn(dyn), dt, ctr_off);
  __syncthreads();
  if (ok) batch_hb_planes<I>(R, phase, parity, sa, m, j, k0);
}

// The replica's pass order (counter mode of ModelGChargeHB::step): the direction
// in place ixyz and the first face's A-site parity.
__device__ __forceinline__ void rep_charge_order(const RepDesc &R, unsigned long long c0, int ixyz, int &dir, int &e0) {
  const uint64_t w = split_word(sub_key(R.key, c0), 0);
  const int pi = (int)((w & 0xffffffffull) % 6ull);
  // lexicographic permutation pi of (0, 1, 2): first element pi / 2, then the
  // remaining two in order (pi even) or swapped (pi odd)
  const int p0 = pi / 2;
  const int lo = (p0 == 0) ? 1 : 0, hi = (p0 == 2) ? 1 : 2;
  dir = ixyz == 0 ? p0 : (ixyz == 1 ? ((pi & 1) ? hi : lo) : ((pi & 1) ? lo : hi));
  e0 = (int)(w >> 63);
}

template <typename I>
__device__ __forceinline__ void batch_charge_item(const RepDesc *__restrict__ d, const EnsDyn *dyn,
                                                  const int *__restrict__ rep, const int *__restrict__ first, int blk,
                                                  int lane, int phase, int pass, double dt, int ctr_off_order) {
  const int r = rep[blk];
  const RepDesc &R = d[r];
  const EnsDyn y = load_dyn(dyn);
  int m, j, k0;
  if (!slab_coords(R, blk - first[r], lane, m, j, k0)) return;
  const unsigned long long c0 = y.ctr + (unsigned long long)ctr_off_order;
  int dir, e0;
  rep_charge_order(R, c0, pass / 2, dir, e0);
  const int eoA = (pass & 1) ? (e0 ^ 1) : e0;
  ChargeArgs a{};
  a.rms = sqrt(2. * dt * (R.diffusion * R.chi));
  a.inv2chi = 1.0 / (2. * R.chi);
  a.sk = sub_key(R.key, c0 + 1 + pass);
  a.pass = pass;
  const Fields f = rep_fields(R, phase, phase);
  MonLocal mon;
#pragma unroll 1
  for (int q = 0; q < kBatchPlanes; ++q)
    if (k0 + q < R.g.N) charge_link_site<false, false, I>(f, R.g, dir, eoA, a, m, j, k0 + q, mon);
}

// Both faces of the direction in place ixyz of every replica's order, from the
// charges of buffer `phase` to those of the other one.  Block blk of the run
// map, whose share of a replica is batch_run_blocks(N): along x a block holds
// whole rows (all six charges in turn), along y and z runs of kBatchSeg sites of
// one charge (charge_run).
// kBatchRowSets sets of rows per block: both forms then need about as many
// blocks (a charge step of 52 replicas, 20^3 to 64^3: 240 us at one set and 222
// at two with runs of 32, 236 with runs of 16, 237 at four sets).  Twelve blocks
// per SM (40 registers, 40 bytes of spill): 222 -> 207 us, since the step waits
// on its replicas' memory; 48 registers 213, 32 registers 219.
constexpr int kBatchSeg = 32, kBatchRowSets = 2;

__device__ __forceinline__ void batch_charge_rows(const Geo &g, int blk, const ChargeDirArgs &a, double *sh) {
  const int N = g.N, H = g.H, rows = N * N;
  if (H <= kRunThreads) {  // a pair per thread, as charge_row_kernel
    const int by = kRunThreads / H, y = (int)threadIdx.x / H, m = (int)threadIdx.x - y * H;
    for (int r0 = blk * kBatchRowSets * by; r0 < min(rows, (blk + 1) * kBatchRowSets * by); r0 += by) {
      const bool valid = y < by && r0 + y < rows;
      charge_row(g, 0, 6, m, valid ? r0 + y : 0, valid, a, sh + y * H, (by + 1) * H);
      __syncthreads();
    }
    return;
  }
  if (blk >= rows) return;
  double *sA = sh, *sB = sh + H;
  const int k = blk / N, b = (a.eo[0] ^ (blk - k * N + k)) & 1;
  const long long ra = (long long)a.eo[0] * g.V2 + (long long)blk * H, rb = (long long)a.eo[1] * g.V2 + (long long)blk * H;
  pdl_wait();
  for (int L = 0; L < 6; ++L) {
    const double *in = a.in + L * a.pitch_in;
    double *out = a.out + L * a.pitch_out;
    for (int m = threadIdx.x; m < H; m += kRunThreads) {
      const int xb = 2 * m + b + 1 == N ? 0 : 2 * m + b + 1;
      double A = in[ra + m], B = in[rb + (xb >> 1)];
      charge_link(A, B, a.sk[0] + (6 * ((uint64_t)blk * N + 2 * m + b) + L + 1) * kGolden, a.rms, a.invchi);
      sA[m] = A;
      sB[m] = B;
    }
    __syncthreads();
    for (int m = threadIdx.x; m < H; m += kRunThreads) {
      const int xb = 2 * m + b + 1 == N ? 0 : 2 * m + b + 1, mn = m + 1 == H ? 0 : m + 1;
      double A = sA[mn], B = sB[m];
      charge_link(B, A, a.sk[1] + (6 * ((uint64_t)blk * N + xb) + L + 1) * kGolden, a.rms, a.invchi);
      out[ra + mn] = A;
      out[rb + (xb >> 1)] = B;
    }
    __syncthreads();
  }
}

template <typename I>
__global__ void __launch_bounds__(kRunThreads, 12) batch_charge_dir_kernel(const RepDesc *__restrict__ d,
                                                                       const EnsDyn *dyn,
                                                                       const int *__restrict__ rep,
                                                                       const int *__restrict__ first, int phase,
                                                                       int ixyz, double dt, int ctr_off_order) {
  extern __shared__ double xs[];
  pdl_launch();
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  const int blk = blockIdx.x - first[r], N = R.g.N;
  pdl_wait();
  __shared__ ChargeDirArgs a;  // once per block: the order, keys, a square root and a division
  __shared__ int s_dir;
  if (threadIdx.x == 0) {
    const unsigned long long c0 = load_dyn(dyn).ctr + (unsigned long long)ctr_off_order;
    int dir, e0;
    rep_charge_order(R, c0, ixyz, dir, e0);
    s_dir = dir;
    a.in = R.base[phase] + 4 * R.pstride;
    a.out = R.base[phase ^ 1] + 4 * R.pstride;
    a.pitch_in = a.pitch_out = R.pstride;
    a.rms = sqrt(2. * dt * (R.diffusion * R.chi));
    a.invchi = 2.0 * (1.0 / (2. * R.chi));
    a.sk[0] = sub_key(R.key, c0 + 1 + 2 * ixyz);
    a.sk[1] = sub_key(R.key, c0 + 2 + 2 * ixyz);
    a.eo[0] = e0;
    a.eo[1] = e0 ^ 1;
  }
  __syncthreads();
  const int dir = s_dir;
  if (dir == 0) {
    batch_charge_rows(R.g, blk, a, xs);
    return;
  }
  const int nrun = (N + kBatchSeg - 1) / kBatchSeg, L = blk % 6, q = blk / 6, run = q % nrun;
  const int idx = (q / nrun) * kRunThreads + (int)threadIdx.x, o = idx / N, t = idx - o * N;
  if (o >= N) return;
  const int s = t >= R.g.H ? 1 : 0, i = 2 * (t - s * R.g.H) + s;
  const int seg0 = run * kBatchSeg, len = min(kBatchSeg, N - seg0);
  if (dir == 1) charge_run<1, true, I>(R.g, L, i, o, seg0, len, a);
  else charge_run<2, true, I>(R.g, L, i, o, seg0, len, a);
}

// ---- differentiable Euler-Maruyama runs of an ensemble ---------------------
__device__ __forceinline__ Fields diff_planes(double *base, long long V, long long first) {
  Fields f{};
#pragma unroll
  for (int l = 0; l < 4; ++l) f.c[l] = base + (first + l) * V;
  return f;
}

__device__ __forceinline__ EmArgs rep_em_args(const RepDesc &R, unsigned long long ctr, double t, double dt) {
  EmArgs a{};
  a.c6 = 6.0 + __dadd_rn(R.mass0, __dmul_rn(R.dmassdt, t));
  a.dtg = dt * R.gamma;
  a.sq = sqrt(2.0 * R.gamma * dt);
  a.lambda = R.lambda;
  a.H = R.H;
  a.sk = sub_key(R.key, ctr);
  return a;
}

// Blocks of the plane map: 256 threads, both halves of 128 elements (as all_site).
__device__ __forceinline__ bool rep_site(const RepDesc &R, int local, int &parity, int &m, int &j, int &k) {
  k = local / R.nchunk;
  return all_site(R.g, local - k * R.nchunk, parity, m, j);
}

// Forward step: phi of the lattice buffer `phase` -> phase ^ 1, the sums of the
// new phi into the block's row of `partial`.
template <typename I>
__global__ void __launch_bounds__(kSiteThreads, kEmBlocks) batch_em_fwd_kernel(const RepDesc *__restrict__ d,
                                                                    const int *__restrict__ rep,
                                                                    const int *__restrict__ first, int phase,
                                                                    unsigned long long ctr, double t, double dt,
                                                                    double *partial) {
  pdl_launch();
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  __shared__ EmArgs sa;  // once per block: a square root and a key
  if (threadIdx.x == 0) sa = rep_em_args(R, ctr, t, dt);
  __syncthreads();
  int parity, m, j, k;
  double acc[4] = {0, 0, 0, 0};
  if (rep_site(R, blockIdx.x - first[r], parity, m, j, k))
    em_site<false, I>(rep_fields(R, phase, phase), rep_fields(R, phase ^ 1, phase ^ 1), R.g, sa,
                      parity, m, j, k, acc);
  block_sum4<kSiteThreads>(acc, partial + (size_t)blockIdx.x * 4);
}

template <typename I>
__global__ void __launch_bounds__(kSiteThreads, kEmBlocks) batch_em_seg_kernel(const RepDesc *__restrict__ d,
                                                                    const DiffDesc *__restrict__ dd,
                                                                    const int *__restrict__ rep,
                                                                    const int *__restrict__ first, int slot,
                                                                    unsigned long long ctr, double t, double dt) {
  pdl_launch();
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  __shared__ EmArgs sa;  // once per block: a square root and a key
  if (threadIdx.x == 0) sa = rep_em_args(R, ctr, t, dt);
  __syncthreads();
  const DiffDesc &D = dd[r];
  int parity, m, j, k;
  if (!rep_site(R, blockIdx.x - first[r], parity, m, j, k)) return;
  double acc[4];
  em_site<false, I>(diff_planes(D.seg, D.V, 4LL * slot), diff_planes(D.seg, D.V, 4LL * (slot + 1)), R.g,
                    sa, parity, m, j, k, acc);
}

// Sums of phi of the lattice buffer `phase`, a row per block.
__global__ void __launch_bounds__(kSiteThreads) batch_phi_sum_kernel(const RepDesc *__restrict__ d,
                                                                     const int *__restrict__ rep,
                                                                     const int *__restrict__ first, int phase,
                                                                     double *partial) {
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  int parity, m, j, k;
  double v[4] = {0, 0, 0, 0};
  if (rep_site(R, blockIdx.x - first[r], parity, m, j, k)) {
    const long long o = (long long)parity * R.g.V2 + ((long long)k * R.g.N + j) * R.g.H + m;
#pragma unroll
    for (int l = 0; l < 4; ++l) v[l] = R.base[phase][(long long)l * R.pstride + o];
  }
  block_sum4<kSiteThreads>(v, partial + (size_t)blockIdx.x * 4);
}

// Block (replica r, slot): the rows of r's blocks in src[slot][nblocks][4] into
// row row0 + slot of r's averages (WHAT 0, scaled by 1 / V) or of its gradient
// rows (1); WHAT 2: r's n gradient rows into its gradient.
template <int WHAT>
__global__ void __launch_bounds__(kSumThreads) batch_sum_kernel(const DiffDesc *__restrict__ dd,
                                                                const int *__restrict__ first,
                                                                const int *__restrict__ count, const double *src,
                                                                int nblocks, int row0, int n) {
  const int r = blockIdx.x;
  const DiffDesc &D = dd[r];
  if (WHAT == 2) {
    sum_rows(D.gs, 0, n, 1.0, D.grad);
    return;
  }
  const size_t row = ((size_t)row0 + blockIdx.y) * 4;
  sum_rows(src + (size_t)blockIdx.y * nblocks * 4, first[r], first[r] + count[r], WHAT == 0 ? 1.0 / (double)D.V : 1.0,
           (WHAT == 0 ? D.avg : D.gs) + row);
}

// dJ/dphi_a(n) of J = w0 obs0 + w1 obs1 (the per-replica averages of the run)
__device__ __forceinline__ double rep_gl(const DiffDesc &D, int n, int b, int S, int a) {
  if (n <= b) return 0.0;
  const double M = (double)(S - b);
  return a == 0 ? D.w[0] / ((double)D.V * M) : D.w[1] * 2.0 * D.avg[(size_t)n * 4 + a] / M;
}

template <typename I>
__global__ void __launch_bounds__(kSiteThreads, kEmAdjBlocks) batch_em_adj_kernel(const RepDesc *__restrict__ d,
                                                                    const DiffDesc *__restrict__ dd,
                                                                    const int *__restrict__ rep,
                                                                    const int *__restrict__ first, int slot, int cur,
                                                                    int n, int b, int S, unsigned long long ctr,
                                                                    double t, double dt, double *partial) {
  pdl_launch();
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  const DiffDesc &D = dd[r];
  __shared__ EmAdjArgs sa;  // once per block: square roots, a key, and the divisions of the loss gradient
  if (threadIdx.x == 0) {
    sa.c6 = 6.0 + __dadd_rn(R.mass0, __dmul_rn(R.dmassdt, t));
    sa.dtg = dt * R.gamma;
    sa.dt = dt;
    sa.lambda = R.lambda;
    sa.H = R.H;
    sa.cxi = sqrt(2.0 * dt) / (2.0 * sqrt(R.gamma));
    sa.sk = sub_key(R.key, ctr);
  }
  // avg and w were complete before the first adjoint launch
  if (threadIdx.x >= 32 && threadIdx.x < 36) sa.gl[threadIdx.x - 32] = rep_gl(D, n, b, S, threadIdx.x - 32);
  __syncthreads();
  double v[4] = {0, 0, 0, 0};
  int parity, m, j, k;
  if (rep_site(R, blockIdx.x - first[r], parity, m, j, k))
    em_adjoint_site<I>(diff_planes(D.seg, D.V, 4LL * slot), diff_planes(D.lam, D.V, 4LL * cur),
                       diff_planes(D.lam, D.V, 4LL * (cur ^ 1)), R.g, sa, parity, m, j, k,
                       [&](int q) { return sa.gl[q]; }, v);
  block_sum4<kSiteThreads>(v, partial + (size_t)blockIdx.x * 4);
}

__global__ void __launch_bounds__(128) batch_diff_copy_kernel(const RepDesc *__restrict__ d,
                                                              const DiffDesc *__restrict__ dd,
                                                              const int *__restrict__ rep,
                                                              const int *__restrict__ first, int dir, int phase, int s,
                                                              int b, int S) {
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  const DiffDesc &D = dd[r];
  int m, j, k;
  if (!plane_coords(R, blockIdx.x - first[r], m, j, k)) return;
  const long long row = ((long long)k * R.g.N + j) * R.g.H + m;
  double gl[4] = {0, 0, 0, 0};
  if (dir == 2)
    for (int l = 0; l < 4; ++l) gl[l] = rep_gl(D, S, b, S, l);
#pragma unroll
  for (int l = 0; l < 4; ++l)
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      const long long o = par * R.g.V2 + row;
      if (dir == 0) D.ckpt[((long long)s * 4 + l) * D.V + o] = R.base[phase][l * R.pstride + o];
      else if (dir == 1) D.seg[(long long)l * D.V + o] = D.ckpt[((long long)s * 4 + l) * D.V + o];
      else D.lam[(long long)l * D.V + o] = gl[l];
    }
}

template <typename I>
__global__ void __launch_bounds__(kSiteThreads, kEmBlocks) batch_em_kernel(const RepDesc *__restrict__ d,
                                                                const EnsDyn *dyn,
                                                                const int *__restrict__ rep,
                                                                const int *__restrict__ first, int phase_in, double dt,
                                                                int ctr_off) {
  pdl_launch();
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  int parity, m, j, k;
  const bool ok = rep_site(R, blockIdx.x - first[r], parity, m, j, k);
  // Warps without a site leave (the first stays, for the arguments): a plane below
  // 12^2 fills less than half of its block (a step of 500 of 8^3 25.0 -> 19.0 us,
  // of 1000 of 4^3 24.0 -> 18.2; with 128 threads of two sites each 23.3 and 23.4).
  if (threadIdx.x >= 32 && !__any_sync(0xffffffffu, ok)) return;
  pdl_wait();
  const EnsDyn y = load_dyn(dyn);
  __shared__ EmArgs sa;
  if (threadIdx.x == 0) sa = rep_em_args(R, y.ctr + (unsigned long long)ctr_off, y.t, dt);
  __syncthreads();
  if (!ok) return;
  double acc[4];
  em_site<false, I>(rep_fields(R, phase_in, phase_in), rep_fields(R, phase_in ^ 1, phase_in ^ 1), R.g,
                    sa, parity, m, j, k, acc);
}

template <int TX, int TY>
__device__ __forceinline__ void batch_ideal_item(const RepDesc *__restrict__ d, const int *__restrict__ rep,
                                                 const int *__restrict__ first, int blk, int pphi, int pq, double dt) {
  const int r = rep[blk];
  const RepDesc &R = d[r];
  const int l = blk - first[r];
  const int bx = l % R.igx, by = (l / R.igx) % R.igy, bz = l / (R.igx * R.igy);
  IdealArgs a;
  a.dto2chi = (dt / 2.0) / R.chi;
  a.dt = dt;
  a.a2 = R.a2;
  a.H = R.H;
  ideal_tile<TX, TY>(rep_fields(R, pphi, pq), rep_fields(R, pphi ^ 1, pq ^ 1), R.g, R.izc, a, bx, by, bz);
}

template <int TX, int TY>
__global__ void __launch_bounds__(TX *TY, 2) batch_ideal_kernel(const RepDesc *__restrict__ d,
                                                                const int *__restrict__ rep,
                                                                const int *__restrict__ first, int pphi, int pq,
                                                                double dt) {
  pdl_launch();
  pdl_wait();
  batch_ideal_item<TX, TY>(d, rep, first, blockIdx.x, pphi, pq, dt);
}

// ---- persistent ensemble step -------------------------------------------------
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier over the co-resident CTAs of a cooperative launch.  bar[0]
// counts the arrivals of the current generation, bar[1] is the generation and
// bar[2] an error flag.  One thread per CTA reads the generation, publishes
// the CTA's writes (fence) and arrives; the last to arrive resets the count
// and advances the generation, the others poll it -- at most `limit` times,
// after which the CTA raises the error flag, counts a timed-out wait and
// gives up.  A CTA that sees the error flag gives up too, so every CTA leaves
// the launch after a bounded number of polls whatever happened to the
// others.  Returns false when the launch should stop.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned nblocks, int limit, unsigned long long *waits) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned gen = ld_acquire_u32(bar + 1);
    __threadfence();
    if (atomicAdd(bar, 1u) == nblocks - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      for (int i = 0;; ++i) {
        if (ld_acquire_u32(bar + 1) != gen) break;
        if (ld_acquire_u32(bar + 2) != 0u) {
          ok = 0;
          break;
        }
        if (i >= limit) {
          ok = 0;
          atomicExch(bar + 2, 1u);
          if (waits) atomicAdd(waits, 1ull);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

constexpr size_t kPersistSmem = (tma::kSmemBytes > IdealTile<32, 8>::SMEM)
                                    ? (tma::kSmemBytes > IdealTile<16, 16>::SMEM ? tma::kSmemBytes
                                                                                 : IdealTile<16, 16>::SMEM)
                                    : (IdealTile<32, 8>::SMEM > IdealTile<16, 16>::SMEM ? IdealTile<32, 8>::SMEM
                                                                                        : IdealTile<16, 16>::SMEM);

// The persistent step's bodies as calls, so that each keeps the register
// allocation of its own kernel instead of the union of all of them.
__device__ __noinline__ void persist_tma_tile(const PersistPtrs &q, int w, const PersistPhase &ph, int limit) {
  tma::batch_tma_item(q.d, reinterpret_cast<const CUtensorMap *>(q.gmaps), q.tma_rep, q.tma_first, w, ph.pphi, ph.pq,
                      ph.dt, q.waits, limit);
}
template <int TX, int TY>
__device__ __noinline__ void persist_cp_tile(const PersistPtrs &q, int w, const PersistPhase &ph) {
  batch_ideal_item<TX, TY>(q.d, q.cp_rep, q.cp_first, w, ph.pphi, ph.pq, ph.dt);
}
template <typename I>
__device__ __noinline__ void persist_phi_item(const PersistPtrs &q, int blk, int lane, const PersistPhase &ph) {
  batch_hb_item<I>(q.d, q.dyn, q.slab_rep, q.slab_first, blk, lane, ph.pphi, ph.arg, ph.dt, ph.ctr_off);
}
template <typename I>
__device__ __noinline__ void persist_charge_item(const PersistPtrs &q, int blk, int lane, const PersistPhase &ph) {
  batch_charge_item<I>(q.d, q.dyn, q.slab_rep, q.slab_first, blk, lane, ph.pq, ph.arg, ph.dt, ph.ctr_off);
}

// One step of an ensemble in one launch of 256-thread CTAs, two per SM (the
// ideal step's CTA bodies set the shape).  Each phase hands its items out
// round robin over the grid: ideal tiles (TMA replicas first, through the
// same CTA bodies as batch_ideal_tma_kernel and batch_ideal_kernel), or pairs
// of 128-lane slab items of the heat-bath and charge sub-steps (each half of
// the CTA one item: batch_hb_item, batch_charge_item).  Phases are
// separated by grid_barrier; after the last one block 0 advances the
// ensemble's counter and clock, as launch_ens_advance does after the
// one-launch-per-sub-step sequence.  Results equal that sequence's bit for
// bit (same device functions, same noise indexing).
template <typename I>
__global__ void __launch_bounds__(256, 2) ens_persistent_kernel(const __grid_constant__ PersistPlan P,
                                                                const PersistPtrs q) {
  const int lane = threadIdx.x & 127, half = threadIdx.x >> 7;
  for (int f = 0; f < P.nphase; ++f) {
    const PersistPhase &ph = P.ph[f];
    if (ph.kind == kPersistIdeal) {
      const int n = P.nb_tma + P.nb_cp;
      for (int w = blockIdx.x; w < n; w += gridDim.x) {
        if (w < P.nb_tma) {
          // the TMA loads (async proxy) read what the previous phase stored
          if (threadIdx.x == 0) asm volatile("fence.proxy.async.global;\n" ::: "memory");
          persist_tma_tile(q, w, ph, P.wait_limit);
        } else if (P.tile == LGV_TILE_16x16) {
          persist_cp_tile<16, 16>(q, w - P.nb_tma, ph);
        } else {
          persist_cp_tile<32, 8>(q, w - P.nb_tma, ph);
        }
        __syncthreads();  // the tile's shared memory and barriers are reused by the next one
      }
    } else {
      const int n = (P.nb_slab + 1) / 2;
      for (int w = blockIdx.x; w < n; w += gridDim.x) {
        const int blk = 2 * w + half;
        if (blk < P.nb_slab) {
          if (ph.kind == kPersistPhi) persist_phi_item<I>(q, blk, lane, ph);
          else persist_charge_item<I>(q, blk, lane, ph);
        }
      }
    }
    if (!grid_barrier(q.bar, gridDim.x, P.wait_limit, q.waits)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    q.dyn->ctr += P.dctr;
    q.dyn->t += P.dt_step;
  }
}

__global__ void ens_set_kernel(EnsDyn *dyn, unsigned long long ctr, double t) {
  dyn->ctr = ctr;
  dyn->t = t;
}
__global__ void ens_advance_kernel(EnsDyn *dyn, unsigned long long dctr, double dt) {
  pdl_launch();
  pdl_wait();
  dyn->ctr += dctr;
  dyn->t += dt;
}

// Volume averages of the 11 OAverage observables per replica.
__global__ void __launch_bounds__(128) batch_oavg_kernel(const RepDesc *__restrict__ d, const int *__restrict__ rep,
                                                         const int *__restrict__ first, int pphi, int pq,
                                                         double *partial) {
  const int r = rep[blockIdx.x];
  const RepDesc &R = d[r];
  int m, j, k;
  double acc[11];
#pragma unroll
  for (int o = 0; o < 11; ++o) acc[o] = 0;
  if (plane_coords(R, blockIdx.x - first[r], m, j, k)) {
    const long long row = ((long long)k * R.g.N + j) * R.g.H + m;
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      const long long o = par * R.g.V2 + row;
      double p2 = 0;
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const double v = R.base[pphi][(long long)l * R.pstride + o];
        acc[l] += v;
        p2 += v * v;
      }
#pragma unroll
      for (int l = 4; l < 10; ++l) acc[l] += R.base[pq][(long long)l * R.pstride + o];
      acc[10] += p2;
    }
  }
  __shared__ double sm[11][4];
#pragma unroll
  for (int o = 0; o < 11; ++o) {
    warp_sum(acc[o]);
    if ((threadIdx.x & 31) == 0) sm[o][threadIdx.x >> 5] = acc[o];
  }
  __syncthreads();
  if (threadIdx.x < 11) {
    const int o = threadIdx.x;
    partial[(long long)blockIdx.x * 11 + o] = ((sm[o][0] + sm[o][1]) + sm[o][2]) + sm[o][3];
  }
}

__global__ void batch_oavg_final_kernel(const RepDesc *__restrict__ d, const int *__restrict__ first, int nrep,
                                        const int *__restrict__ count, const double *partial, double *out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nrep * 11) return;
  const int r = t / 11, o = t % 11;
  double s = 0;
  for (int b = 0; b < count[r]; ++b) s += partial[(long long)(first[r] + b) * 11 + o];
  out[t] = s / (2.0 * (double)d[r].g.V2);
}

// ----------------------------------------------------------------------------
// Adjoint of the Euler-Maruyama step (noise fixed).  The step is
//   phi'_a = phi_a - dt G F_a(phi) + sqrt(2 G dt) xi_a,
//   F_a = -sum_nbr phi_a + (6 + m^2) phi_a + lambda phi^2 phi_a - H delta_a0,
// so with lam = dL/dphi' (lam_in) the adjoint of the state is
//   lam_b - dt G [(6 + m^2) lam_b + lambda (phi^2 lam_b + 2 phi_b (phi . lam))
//                 - sum_nbr lam_b] + gl_b
// (the lattice Laplacian is symmetric), and the parameter sensitivities are
//   dL/dm^2 += -dtG (phi . lam),  dL/dlambda += -dtG phi^2 (phi . lam),
//   dL/dH += dtG lam_0,  dL/dG += lam . (-dt F + sqrt(2dt)/(2 sqrt G) xi).
// One thread per site; the parameter sums leave as a row per block.
template <typename I>
__global__ void __launch_bounds__(kSiteThreads, kEmAdjBlocks) em_adjoint_kernel(Fields phi, Fields lin, Fields lout, Geo g,
                                                                  EmAdjArgs a, double *partial) {
  pdl_launch();
  double v[4] = {0, 0, 0, 0};
  int parity, m, j;
  if (all_site(g, blockIdx.x, parity, m, j))
    em_adjoint_site<I>(phi, lin, lout, g, a, parity, m, j, blockIdx.y, [&](int q) { return a.gl[q]; }, v);
  block_sum4<kSiteThreads>(v, partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 4);
}

// ----------------------------------------------------------------------------
// Adjoint of the ideal step (IdealPV2::step_no_reject, Stepper.cxx:68-176):
//   phi1 = rot(phi, n), n' = n + dt J(phi1), phi2 = rot(phi1, n'),
// with the currents J, summed over directions,
//   J_A,l = a2 (phi1_0 S_l - phi1_l S_0) - H phi1_l,
//   J_V,s = a2 (phi1_s1 S_s2 - phi1_s2 S_s1),   S_a = sum_nbr phi1_a.
// Three passes: rot_phi_kernel writes phi1; ideal_adj_a_kernel recomputes n'
// exactly as the forward does and back-propagates through the second
// rotation (phi1_bar partial -> PB, n'_bar -> QB, dL/dH); ideal_adj_b_kernel
// adds the currents' adjoint (a stencil over QB * phi1), back-propagates
// through the first rotation and writes lam_out = (phi_bar + gl, n_bar).
// Pair (a, b, c): charge c gets a2 (phi1_a S_b - phi1_b S_a).
__host__ __device__ constexpr int pair_a(int c) { return c < 3 ? 0 : (c == 3 ? 2 : (c == 4 ? 3 : 1)); }
__host__ __device__ constexpr int pair_b(int c) { return c < 3 ? c + 1 : (c == 3 ? 3 : (c == 4 ? 1 : 2)); }

__global__ void __launch_bounds__(kThreads) rot_phi_kernel(Fields u, Fields P1, long long V, double k) {
  pdl_launch();
  pdl_wait();
  const long long n = (long long)blockIdx.x * kThreads + threadIdx.x;
  if (n >= V) return;
  double ph[4], q[6];
#pragma unroll
  for (int l = 0; l < 4; ++l) ph[l] = u.c[l][n];
#pragma unroll
  for (int s = 0; s < 6; ++s) q[s] = u.c[4 + s][n];
  rotate_site(ph, q, k);
#pragma unroll
  for (int l = 0; l < 4; ++l) P1.c[l][n] = ph[l];
}

// The ideal step of a small lattice in two launches: rot_phi_kernel writes phi'
// to P1, and this one, a thread per site, advects the charges with the stencil
// on phi' and rotates phi' by the second half step.  Reads the charges of `in`,
// writes `out`, which may be `in`.  Byte offsets: the lattices it takes have planes
// far below 4 GB (ideal_flat).
__global__ void __launch_bounds__(kSiteThreads, 3) ideal_flat_kernel(Fields in, Fields P1, Fields out, Geo g, IdealArgs a) {
  pdl_launch();
  int parity, m, j;
  const bool ok = all_site(g, blockIdx.x, parity, m, j);
  const Nbrs<unsigned> o = nbrs_of<unsigned>(g, parity, m, j, blockIdx.y);
  pdl_wait();
  if (!ok) return;
  double c[4], S[4], q[6];
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    c[l] = *at(P1.c[l], o.own);
    S[l] = nbr_sum(P1.c[l], o);
  }
#pragma unroll
  for (int s = 0; s < 6; ++s) q[s] = *at(in.c[4 + s], o.own);
  charge_currents(c, S, a.dt, a.a2, a.H, q);
  rotate_site(c, q, a.dto2chi);
#pragma unroll
  for (int l = 0; l < 4; ++l) *at(out.c[l], o.own) = c[l];
#pragma unroll
  for (int s = 0; s < 6; ++s) *at(out.c[4 + s], o.own) = q[s];
}

__global__ void __launch_bounds__(kSiteThreads, kIdealAdjBlocks) ideal_adj_a_kernel(Fields u, Fields lin, Fields P1, Fields PB, Fields QB,
                                                                   Geo g, IdealAdjArgs a, double *partial) {
  pdl_launch();
  pdl_wait();
  double v[4] = {0, 0, 0, 0};
  int parity, m, j;
  if (all_site(g, blockIdx.x, parity, m, j)) {
    const Nbrs<long long> o = nbrs_of<long long>(g, parity, m, j, blockIdx.y);
    // n' exactly as the forward computes it (ideal_tile, ideal_tma_kernel)
    double c[4], q2[6], S[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      c[l] = *at(P1.c[l], o.own);
      S[l] = nbr_sum(P1.c[l], o);
    }
#pragma unroll
    for (int s = 0; s < 6; ++s) q2[s] = *at(u.c[4 + s], o.own);
    charge_currents(c, S, a.dt, a.a2, a.H, q2);
    double ob[4], pb[4], qb[6];
#pragma unroll
    for (int l = 0; l < 4; ++l) ob[l] = *at(lin.c[l], o.own);
    rotate_site_adj(c, q2, a.k, ob, pb, qb);
#pragma unroll
    for (int l = 0; l < 4; ++l) *at(PB.c[l], o.own) = pb[l];
    double hb = 0;
#pragma unroll
    for (int s = 0; s < 6; ++s) {
      const double Q = *at(lin.c[4 + s], o.own) + qb[s];
      *at(QB.c[s], o.own) = Q;
      if (s < 3) hb += -a.dt * Q * c[s + 1];
    }
    v[2] = hb;
  }
  block_sum4<kSiteThreads>(v, partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 4);
}

__global__ void __launch_bounds__(kSiteThreads, kIdealAdjBlocks) ideal_adj_b_kernel(Fields u, Fields lout, Fields P1, Fields PB, Fields QB,
                                                                   Geo g, IdealAdjArgs a) {
  pdl_launch();
  pdl_wait();
  int parity, m, j;
  if (!all_site(g, blockIdx.x, parity, m, j)) return;
  const Nbrs<long long> o = nbrs_of<long long>(g, parity, m, j, blockIdx.y);
  const long long od[6] = {o.xp, o.xm, o.jp, o.jm, o.kp, o.km};
  double S[4] = {0, 0, 0, 0}, Na[6] = {0, 0, 0, 0, 0, 0}, Nb[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    double P[4], Q[6];
#pragma unroll
    for (int l = 0; l < 4; ++l) P[l] = P1.c[l][od[d]];
#pragma unroll
    for (int s = 0; s < 6; ++s) Q[s] = QB.c[s][od[d]];
#pragma unroll
    for (int l = 0; l < 4; ++l) S[l] += P[l];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      Na[c] += Q[c] * P[pair_b(c)];
      Nb[c] += Q[c] * P[pair_a(c)];
    }
  }
  double pb[4], Qc[6];
#pragma unroll
  for (int l = 0; l < 4; ++l) pb[l] = *at(PB.c[l], o.own);
#pragma unroll
  for (int s = 0; s < 6; ++s) Qc[s] = *at(QB.c[s], o.own);
  const double da = a.dt * a.a2;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int ia = pair_a(c), ib = pair_b(c);
    pb[ia] += da * (Qc[c] * S[ib] - Na[c]);
    pb[ib] += da * (Nb[c] - Qc[c] * S[ia]);
  }
#pragma unroll
  for (int l = 0; l < 3; ++l) pb[l + 1] += -a.dt * a.H * Qc[l];
  double ph[4], q[6], phb[4], qb[6];
#pragma unroll
  for (int l = 0; l < 4; ++l) ph[l] = *at(u.c[l], o.own);
#pragma unroll
  for (int s = 0; s < 6; ++s) q[s] = *at(u.c[4 + s], o.own);
  rotate_site_adj(ph, q, a.k, pb, phb, qb);
#pragma unroll
  for (int l = 0; l < 4; ++l) *at(lout.c[l], o.own) = phb[l] + a.gl[l];
#pragma unroll
  for (int s = 0; s < 6; ++s) *at(lout.c[4 + s], o.own) = Qc[s] + qb[s];
}

// sums of phi_0..3, a row per block
__global__ void __launch_bounds__(kSiteThreads) phi_sum_kernel(Fields f, Geo g, double *partial) {
  int parity, m, j;
  double v[4] = {0, 0, 0, 0};
  if (all_site(g, blockIdx.x, parity, m, j)) {
    const long long o = (long long)parity * g.V2 + ((long long)blockIdx.y * g.N + j) * g.H + m;
#pragma unroll
    for (int b = 0; b < 4; ++b) v[b] = f.c[b][o];
  }
  block_sum4<kSiteThreads>(v, partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 4);
}

__global__ void fill_phi_kernel(Fields f, long long V, double v0, double v1, double v2, double v3) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= V) return;
  f.c[0][n] = v0;
  f.c[1][n] = v1;
  f.c[2][n] = v2;
  f.c[3][n] = v3;
}

inline unsigned nblocks(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace

// ============================================================================
// Launchers.
cudaError_t launch_aos_to_rb(const double *aos, Fields f, const Geo &g, cudaStream_t st) {
  aos_to_rb_kernel<<<nblocks(2 * g.V2, kThreads), kThreads, 0, st>>>(aos, f, g);
  return cudaGetLastError();
}
cudaError_t launch_aos_to_rb(const double *aos, Fields f, int N, cudaStream_t st) {
  return launch_aos_to_rb(aos, f, make_geo(N), st);
}

cudaError_t launch_rb_to_aos(Fields f, double *aos, const Geo &g, cudaStream_t st) {
  rb_to_aos_kernel<<<nblocks(2 * g.V2, kAosSites), kAosSites, 0, st>>>(f, aos, g);
  return cudaGetLastError();
}
cudaError_t launch_rb_to_aos(Fields f, double *aos, int N, cudaStream_t st) {
  return launch_rb_to_aos(f, aos, make_geo(N), st);
}

cudaError_t launch_init_phi(Fields f, int N, uint64_t sk, double scale, cudaStream_t st) {
  const Geo g = make_geo(N);
  init_phi_kernel<<<nblocks(2 * g.V2, kThreads), kThreads, 0, st>>>(f, g, sk, scale);
  return cudaGetLastError();
}

cudaError_t launch_init_charges(Fields f, int N, uint64_t sk, double sqrtchi, double *scratch,
                                cudaStream_t st) {
  const Geo g = make_geo(N);
  const long long V = 2 * g.V2;
  const unsigned nb = nblocks(V, kThreads);
  double *partial = scratch;
  double *mean = scratch + (size_t)nb * 6;
  init_charge_kernel<<<nb, kThreads, 0, st>>>(f, g, sk, sqrtchi, partial);
  charge_mean_kernel<<<1, 6 * 32, 0, st>>>(partial, (int)nb, 1.0 / (double)V, mean);
  // the red-black planes are contiguous in V, so subtract on the flat planes
  charge_sub_kernel<<<nb, kThreads, 0, st>>>(f, V, mean);
  return cudaGetLastError();
}

template <typename K>
static cudaError_t allow_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// The z-marching pass is opt-in (LGV_HB_ZPASS=1 in the environment, for half
// rows of at least one tile): on B200 at 256^3 it measured 0.22 ms per pass
// against 0.19 ms for hb_pass_kernel -- at 80 registers three CTAs of 8 warps
// per SM wait out the load of the plane above on every plane.
static bool hb_zpass_default(int N) {
  static const bool on = [] {
    const char *v = std::getenv("LGV_HB_ZPASS");
    return v && v[0] == '1';
  }();
  return on && N / 2 >= ZP_TM;
}

cudaError_t launch_hb_zpass(Fields f, int N, int parity, const HbArgs &a, cudaStream_t st) {
  const Geo g = make_geo(N);
  const long long bxy = (long long)((g.H + ZP_TM - 1) / ZP_TM) * ((N + ZP_TY - 1) / ZP_TY);
  long long zc = (long long)N * bxy / (148 * 4 * 3);  // about three waves of 4 CTAs per SM
  zc = std::max(4LL, std::min(32LL, zc));
  zc = std::min<long long>(zc, N);
  const dim3 grid((g.H + ZP_TM - 1) / ZP_TM, (N + ZP_TY - 1) / ZP_TY, (unsigned)((N + zc - 1) / zc));
  const dim3 block(ZP_TM, ZP_TY);
  const bool inj = a.prop != nullptr, mon = a.mon != nullptr;
  if (inj) {
    if (mon) hb_zpass_kernel<true, true><<<grid, block, 0, st>>>(f, g, parity, (int)zc, a);
    else hb_zpass_kernel<true, false><<<grid, block, 0, st>>>(f, g, parity, (int)zc, a);
  } else {
    if (mon) hb_zpass_kernel<false, true><<<grid, block, 0, st>>>(f, g, parity, (int)zc, a);
    else hb_zpass_kernel<false, false><<<grid, block, 0, st>>>(f, g, parity, (int)zc, a);
  }
  return cudaGetLastError();
}

cudaError_t launch_hb_pass(Fields f, int N, int parity, const HbArgs &a, cudaStream_t st) {
  if (hb_zpass_default(N)) return launch_hb_zpass(f, N, parity, a, st);
  return launch_hb_pass(f, make_geo(N), parity, a, st);
}

cudaError_t launch_hb_pass(Fields f, const Geo &g, int parity, const HbArgs &a, cudaStream_t st) {
  const bool inj = a.prop != nullptr, mon = a.mon != nullptr;
  const bool gauss = a.gauss && !inj;  // injected proposals are used as given
  if (!gauss && g.Nz == g.Ng && g.kg == 0 && hb_zpass_default(g.N)) return launch_hb_zpass(f, g.N, parity, a, st);
  const bool rows = g.H % 128 == 0;
  const dim3 grid = pass_grid(g, rows);
  const bool i32 = idx32(g), el = idx_el(g);
  if (!inj && !mon && !rows && hb_small(g, gauss))  // 32-bit offsets hold
    return launch_pdl(gauss ? hb_pass_small_kernel<true> : hb_pass_small_kernel<false>, grid, dim3(128), 0, st, f, g, parity,
                      a);
#define LGV_HBP(I, M, R, T, G) \
  return launch_pdl(hb_pass_kernel<I, M, R, T, G>, grid, dim3(128), 0, st, f, g, parity, a)
#define LGV_HBP_R(I, M, T, G) \
  if (rows) LGV_HBP(I, M, true, T, G); \
  else LGV_HBP(I, M, false, T, G)
#define LGV_HBP_T(I, M, G)                                     \
  if (i32) LGV_HBP_R(I, M, unsigned, G);                       \
  else if (el) LGV_HBP_R(I, M, int, G);                        \
  else LGV_HBP_R(I, M, long long, G)
  if (inj) {
    if (mon) LGV_HBP_T(true, true, false);
    else LGV_HBP_T(true, false, false);
  } else if (gauss) {
    if (mon) LGV_HBP_T(false, true, true);
    else LGV_HBP_T(false, false, true);
  } else if (mon) {
    LGV_HBP_T(false, true, false);
  } else {
    LGV_HBP_T(false, false, false);
  }
#undef LGV_HBP_T
#undef LGV_HBP_R
#undef LGV_HBP
}

// ---- ordered sweeps ---------------------------------------------------------
// Slab thickness: the largest divisor of N not above `target` that leaves at
// least three slabs (an item depends on three distinct neighbours).
static int hb_slab_planes(int N, int target) {
  for (int S = std::min(target, N / 3); S >= 1; --S)
    if (N % S == 0) return S;
  return 0;
}

cudaError_t hb_plan_build(HbPlan &pl, int N, int slab_target, int spc, int lag) {
  hb_plan_free(pl);
  const int S = hb_slab_planes(N, slab_target);
  if (S < 1 || spc < kHbOrderedThreads || spc % kHbOrderedThreads || lag < 1) return cudaErrorInvalidValue;
  pl.N = N;
  pl.S = S;
  pl.nslab = N / S;
  pl.spc = spc;
  const long long item_sites = (long long)S * N * (N / 2);
  pl.cpi = (int)((item_sites + spc - 1) / spc);
  const int n = pl.nslab;
  cudaError_t e;
  for (int ns = 1; ns <= kHbMaxSweeps; ++ns) {
    // T(0, s) = s; T(p, s) = lag + max T(p-1, s-1 .. s+1); items grouped by T,
    // chunks of one group interleaved item by item.
    const int P = 2 * ns;
    std::vector<int> T((size_t)P * n);
    for (int sl = 0; sl < n; ++sl) T[sl] = sl;
    for (int ph = 1; ph < P; ++ph)
      for (int sl = 0; sl < n; ++sl) {
        int t = 0;
        for (int d = -1; d <= 1; ++d) t = std::max(t, T[(size_t)(ph - 1) * n + (sl + d + n) % n]);
        T[(size_t)ph * n + sl] = t + lag;
      }
    std::vector<int> items((size_t)P * n);
    for (int i = 0; i < P * n; ++i) items[i] = i;
    std::stable_sort(items.begin(), items.end(), [&](int x, int y) { return T[x] < T[y]; });
    std::vector<int> sched;
    sched.reserve((size_t)P * n * pl.cpi);
    for (size_t a = 0; a < items.size();) {
      size_t b = a;
      while (b < items.size() && T[items[b]] == T[items[a]]) ++b;
      for (int c = 0; c < pl.cpi; ++c)
        for (size_t q = a; q < b; ++q) sched.push_back(items[q] * pl.cpi + c);
      a = b;
    }
    pl.total[ns - 1] = (int)sched.size();
    if ((e = cudaMalloc((void **)&pl.sched[ns - 1], sched.size() * sizeof(int))) != cudaSuccess) return e;
    if ((e = cudaMemcpy(pl.sched[ns - 1], sched.data(), sched.size() * sizeof(int), cudaMemcpyHostToDevice)) !=
        cudaSuccess)
      return e;
  }
  const size_t nsync = kSyncDone + (size_t)2 * kHbMaxSweeps * n;
  if ((e = cudaMalloc((void **)&pl.sync, nsync * sizeof(unsigned long long))) != cudaSuccess) return e;
  if ((e = cudaMemset(pl.sync, 0, nsync * sizeof(unsigned long long))) != cudaSuccess) return e;
  int dev = 0, sms = 0, occ = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, hb_ordered_kernel<false, false>, kHbOrderedThreads,
                                                          0)) != cudaSuccess)
    return e;
  pl.grid = std::max(1, sms * std::max(1, occ));
  return cudaSuccess;
}

void hb_plan_free(HbPlan &pl) {
  for (int i = 0; i < kHbMaxSweeps; ++i) {
    if (pl.sched[i]) cudaFree(pl.sched[i]);
    pl.sched[i] = nullptr;
    pl.total[i] = 0;
  }
  if (pl.sync) cudaFree(pl.sync);
  pl.sync = nullptr;
  pl.N = 0;
}

cudaError_t launch_hb_ordered(Fields f, int N, const HbArgs &a, const HbPlan &pl, int nsweeps, const uint64_t *sk,
                              cudaStream_t st) {
  if (pl.N != N || nsweeps < 1 || nsweeps > kHbMaxSweeps) return cudaErrorInvalidValue;
  const bool inj = a.prop != nullptr, mon = a.mon != nullptr;
  if ((inj || a.flags) && nsweeps != 1) return cudaErrorInvalidValue;
  HbSched s{};
  s.sched = pl.sched[nsweeps - 1];
  s.sync = pl.sync;
  s.total = pl.total[nsweeps - 1];
  s.cpi = pl.cpi;
  s.spc = pl.spc;
  s.nslab = pl.nslab;
  s.S = pl.S;
  s.nphase = 2 * nsweeps;
  s.limit = pl.wait_limit;
  for (int q = 0; q < nsweeps; ++q) s.sk[q] = sk ? sk[q] : a.sk;
  const Geo g = make_geo(N);
  const int grid = std::min(pl.grid, s.total);
  if (inj) {
    if (mon) hb_ordered_kernel<true, true><<<grid, kHbOrderedThreads, 0, st>>>(f, g, a, s);
    else hb_ordered_kernel<true, false><<<grid, kHbOrderedThreads, 0, st>>>(f, g, a, s);
  } else {
    if (mon) hb_ordered_kernel<false, true><<<grid, kHbOrderedThreads, 0, st>>>(f, g, a, s);
    else hb_ordered_kernel<false, false><<<grid, kHbOrderedThreads, 0, st>>>(f, g, a, s);
  }
  return cudaGetLastError();
}

cudaError_t hb_plan_timeouts(const HbPlan &pl, cudaStream_t st, unsigned long long *out, bool clear) {
  *out = 0;
  if (!pl.sync) return cudaSuccess;
  cudaError_t e = cudaMemcpyAsync(out, pl.sync + kSyncTimeouts, sizeof(*out), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && clear && *out) e = cudaMemsetAsync(pl.sync + kSyncTimeouts, 0, sizeof(*out), st);
  return e;
}

static int hb_zchunk(int N) {
  const int H = N / 2;
  const long long bxy = (long long)((H + HB_TM - 1) / HB_TM) * ((N + HB_TY - 1) / HB_TY);
  long long z = (long long)N * bxy / 1184;  // aim at >= 4 CTAs per SM slot
  if (z > 32) z = 32;
  if (z < 4) z = 4;
  if (z > N) z = N;
  return (int)z;
}

cudaError_t launch_hb_sweep(Fields in, Fields out, int N, const HbArgs &a, cudaStream_t st) {
  const Geo g = make_geo(N);
  const int zc = hb_zchunk(N);
  dim3 grid((g.H + HB_TM - 1) / HB_TM, (N + HB_TY - 1) / HB_TY, (N + zc - 1) / zc);
  const bool inj = a.prop != nullptr, mon = a.mon != nullptr;
  cudaError_t e;
  if (inj) {
    if (mon) {
      if ((e = allow_smem(hb_sweep_kernel<true, true>, HB_SMEM)) != cudaSuccess) return e;
      hb_sweep_kernel<true, true><<<grid, HB_TM * HB_TY, HB_SMEM, st>>>(in, out, g, zc, a);
    } else {
      if ((e = allow_smem(hb_sweep_kernel<true, false>, HB_SMEM)) != cudaSuccess) return e;
      hb_sweep_kernel<true, false><<<grid, HB_TM * HB_TY, HB_SMEM, st>>>(in, out, g, zc, a);
    }
  } else {
    if (mon) {
      if ((e = allow_smem(hb_sweep_kernel<false, true>, HB_SMEM)) != cudaSuccess) return e;
      hb_sweep_kernel<false, true><<<grid, HB_TM * HB_TY, HB_SMEM, st>>>(in, out, g, zc, a);
    } else {
      if ((e = allow_smem(hb_sweep_kernel<false, false>, HB_SMEM)) != cudaSuccess) return e;
      hb_sweep_kernel<false, false><<<grid, HB_TM * HB_TY, HB_SMEM, st>>>(in, out, g, zc, a);
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_charge_pass(Fields f, int N, int dir, int eoA, const ChargeArgs &a, cudaStream_t st) {
  return launch_charge_pass(f, make_geo(N), dir, eoA, a, st);
}

cudaError_t launch_charge_pass(Fields f, const Geo &g, int dir, int eoA, const ChargeArgs &a, cudaStream_t st) {
  const bool rows = g.H % 128 == 0;
  const dim3 grid = pass_grid(g, rows);
  const bool inj = a.q != nullptr, mon = a.mon != nullptr;
  const bool i32 = idx_el(g);
#define LGV_CHP1(I, M, T)                                                                                    \
  return launch_pdl(rows ? charge_pass_kernel<I, M, true, T> : charge_pass_kernel<I, M, false, T>, grid, dim3(128), 0, \
                    st, f, g, dir, eoA, a)
#define LGV_CHP(I, M)                                                                                        \
  if (i32) { LGV_CHP1(I, M, int); } else { LGV_CHP1(I, M, long long); }
  if (inj) { if (mon) { LGV_CHP(true, true); } else { LGV_CHP(true, false); } }
  else { if (mon) { LGV_CHP(false, true); } else { LGV_CHP(false, false); } }
#undef LGV_CHP
#undef LGV_CHP1
  return cudaGetLastError();
}

// Sites per run along y and z: a run of `seg` sites repeats one of its seg
// links, shorter runs are more threads.  The longest of 32, 16 and 8 that leaves
// two rounds of resident threads (a charge step measured at 8 / 16 / 32 / 64:
// 64^3 23.6 / 28.7 / - / 39 us, 128^3 143 / 138 / - / 148, 256^3 1205 / 1143 /
// 1097 / 1106).
static int charge_seg(int N) {
  int seg = 32;
  while (seg > 8 && 6LL * N * N * ((N + seg - 1) / seg) < 2LL * 148 * 2048) seg >>= 1;
  return std::min(seg, N);
}

// Charges per thread along x: all six (the row's indices are worked out once;
// 256^3 982 us a charge step against 1152 at one each) unless that leaves the
// chip short of threads (64^3: 22.4 us at three, 23.0 at six, 25.1 at one).
static int charge_row_nl(const Geo &g) { return g.V2 >= 148LL * 2048 ? 6 : 3; }

cudaError_t launch_charge_dir(Fields in, Fields out, const Geo &g, int dir, const ChargeDirPair &p, cudaStream_t st) {
  ChargeDirArgs a{};
  a.in = in.c[4];
  a.out = out.c[4];
  a.pitch_in = in.c[5] - in.c[4];
  a.pitch_out = out.c[5] - out.c[4];
  for (int L = 0; L < 6; ++L)
    if (in.c[4 + L] != a.in + L * a.pitch_in || out.c[4 + L] != a.out + L * a.pitch_out) return cudaErrorInvalidValue;
  a.rms = p.rms;
  a.invchi = 2.0 * p.inv2chi;
  for (int i = 0; i < 2; ++i) {
    a.sk[i] = p.sk[i];
    a.eo[i] = p.eo[i];
  }
  if (dir == 0) {
    const int by = std::max(1, kRunThreads / g.H), nl = charge_row_nl(g);
    const dim3 block(g.H, by), grid((unsigned)(((long long)g.N * g.N + by - 1) / by), 6 / nl);
    return launch_pdl(charge_row_kernel, grid, block, 2 * (size_t)by * g.H * sizeof(double), st, g, a, nl);
  }
  const bool i32 = 16 * g.V2 <= 0xffffffffLL;  // byte offsets within a plane
  const int seg = charge_seg(g.N);
  const dim3 grid(nblocks((long long)g.N * g.N, kRunThreads), (g.N + seg - 1) / seg, 6);
#define LGV_RUN(D)                                                                                                  \
  launch_pdl(i32 ? charge_run_kernel<D, unsigned> : charge_run_kernel<D, long long>, grid, dim3(kRunThreads), 0, st, g, \
             a, seg)
  return dir == 1 ? LGV_RUN(1) : LGV_RUN(2);
#undef LGV_RUN
}

cudaError_t launch_em(Fields in, Fields out, int N, const EmArgs &a, cudaStream_t st) {
  return launch_em(in, out, make_geo(N), a, st);
}

cudaError_t launch_em(Fields in, Fields out, const Geo &g, const EmArgs &a, cudaStream_t st) {
  // Five blocks per SM (48 registers) where that is one round of blocks (24^3 to
  // 56^3 0.2 to 0.3 us faster than six), six beyond (128^3 51.1 -> 50.3 us, 300^3
  // 675 -> 643, 400^3 1602 -> 1533, 720^3 10.3 -> 9.9 ms), and eight (32 registers)
  // for the largest lattices' int offsets (814^3 16.3 -> 15.4 ms).
  const bool one_round = 2 * g.V2 <= 148LL * kEmBlocks * kSiteThreads;
#define LGV_EM(J)                                                                      \
  (one_round ? em_kernel<J, false, unsigned>                                           \
             : idx32(g) ? em_kernel<J, false, unsigned, 6>                             \
                        : idx_el(g) ? em_kernel<J, false, int, 8> : em_kernel<J, false, long long, 6>)
  const auto kern = a.xi ? LGV_EM(true) : LGV_EM(false);
#undef LGV_EM
  return launch_pdl(kern, site_grid(g), dim3(kSiteThreads), 0, st, in, out, g, a, nullptr);
}

cudaError_t launch_em_sum(Fields in, Fields out, int N, const EmArgs &a, double *partial, cudaStream_t st) {
  const Geo g = make_geo(N);
  const auto kern = idx32(g) ? em_kernel<false, true, unsigned> : em_kernel<false, true, long long>;
  return launch_pdl(kern, site_grid(g), dim3(kSiteThreads), 0, st, in, out, g, a, partial);
}

// Where the march's chunks of a few planes are a chain of latencies and the
// fields sit in L2, two flat launches are faster although phi' takes 112 B/site
// more: 32^3 11.6 -> 5.4 us, 64^3 15.0 -> 10.4, 96^3 42.6 -> 35.0; 128^3 92.0 and
// 91.5, 160^3 161 and 177, 256^3 601 and 748.  Sides that 32 does not divide
// march without TMA: 90^3 45.3 -> 28.1, 120^3 96 -> 76, 150^3 175 -> 155, 200^3
// 402 -> 348, 250^3 713 and 749.
bool ideal_flat(int N) { return N % 32 == 0 ? N < 128 : N <= 200; }

cudaError_t launch_ideal_flat(Fields in, Fields P1, Fields out, const Geo &g, const IdealArgs &a, cudaStream_t st) {
  const long long V = 2 * g.V2;
  const cudaError_t e =
      launch_pdl(rot_phi_kernel, dim3(nblocks(V, kThreads)), dim3(kThreads), 0, st, in, P1, V, a.dto2chi);
  if (e != cudaSuccess) return e;
  return launch_pdl(ideal_flat_kernel, site_grid(g), dim3(kSiteThreads), 0, st, in, P1, out, g, a);
}

cudaError_t launch_ideal(Fields in, Fields out, int N, const IdealArgs &a, cudaStream_t st) {
  return launch_ideal(in, out, make_geo(N), a, st);
}

cudaError_t launch_ideal(Fields in, Fields out, const Geo &g, const IdealArgs &a, cudaStream_t st) {
  const int N = g.N;
  constexpr int TX = 32, TY = 8;
  using T = IdealTile<TX, TY>;
  const long long bxy = (long long)((N + TX - 1) / TX) * ((N + TY - 1) / TY);
  long long zc = (long long)g.Nz * bxy / 1184;
  if (zc > 32) zc = 32;
  if (zc < 4) zc = 4;
  if (zc > g.Nz) zc = g.Nz;
  static const bool tma_off = [] {
    const char *v = std::getenv("LGV_IDEAL_TMA");
    return v && v[0] == '0';
  }();
  if (!tma_off && ideal_tma_supported(N)) return launch_ideal_tma(in, out, g, (int)zc, a, st);
  dim3 grid((N + TX - 1) / TX, (N + TY - 1) / TY, (unsigned)((g.Nz + zc - 1) / zc));
  cudaError_t e = allow_smem(ideal_kernel<TX, TY>, T::SMEM);
  if (e != cudaSuccess) return e;
  return launch_pdl(ideal_kernel<TX, TY>, grid, dim3(TX * TY), T::SMEM, st, in, out, g, (int)zc, a);
}

size_t energy_scratch_doubles(int N) {
  const long long V = (long long)N * N * N;
  return (size_t)nblocks(V, kThreads) * 3 + 8;
}

cudaError_t launch_energy(Fields f, int N, double H, double half_over_chi, double *scratch, double *dev_out,
                          cudaStream_t st) {
  const Geo g = make_geo(N);
  const unsigned nb = nblocks(2 * g.V2, kThreads);
  energy_kernel<<<nb, kThreads, 0, st>>>(f, g, scratch);
  energy_final_kernel<<<1, 96, 0, st>>>(scratch, (int)nb, H, half_over_chi, dev_out);
  return cudaGetLastError();
}

size_t measure_size(int N) {
  const size_t NK = N / 2 + 1;
  return 11 + 75 * (size_t)N + 234 * NK;
}

// The one-pass measurement's shares grow as N^3 / 128 (they would be 1 GB at
// N = 1024, where the tables of the two-pass sums take 0.4 GB); beyond
// kMeasTileMaxN the two passes have N^2 threads enough to fill the chip.
constexpr int kMeasTileMaxN = 512;

size_t measure_scratch_doubles(int N) {
  if (N > kMeasTileMaxN) return 2 * (size_t)kNObs * N * N;
  const MeasTiles t = meas_tiles(N);
  return t.len(0) + t.len(1) + t.len(2);
}

cudaError_t launch_measure(Fields f, int N, double *scratch, unsigned *done, double *dev_out, cudaStream_t st) {
  const Geo g = make_geo(N);
  const long long NN = (long long)N * N;
  if (N > kMeasTileMaxN) {
    double *T = scratch, *U = scratch + (size_t)kNObs * NN;
    meas_sum_j_kernel<<<nblocks(NN, 128), 128, 0, st>>>(f, g, T, 0, N, 0);
    meas_sum_k_kernel<<<nblocks(NN, 128), 128, 0, st>>>(f, g, U, 0, N);
    return launch_measure_finish(T, U, N, dev_out, st);
  }
  const MeasTiles t = meas_tiles(N);
  double *xp = scratch, *yp = xp + t.len(0), *zp = yp + t.len(1);
  cudaError_t e = allow_smem(meas_tile_kernel, kMtSmem);
  if (e != cudaSuccess) return e;
  if ((e = launch_pdl(meas_tile_kernel, dim3(t.it, t.jt, t.kt), dim3(256), kMtSmem, st, f, g, t, xp, yp, zp)) !=
      cudaSuccess)
    return e;
  const MeasOut mo = meas_layout(dev_out, N);
  const dft::Plan p = dft::make_plan(N);
  int logP = 3;
  while (logP < 8 && (1 << logP) < N) ++logP;
  return launch_pdl(meas_finish_kernel, dim3(kNObs, 3), dim3(kFinishThreads), wall_smem(p), st, xp, yp, zp, t, p, logP, mo,
                    done);
}

cudaError_t launch_measure_partials(Fields f, const Geo &g, int klo, int nk, int kout, double *T, double *U,
                                    cudaStream_t st) {
  const long long NN = (long long)g.N * g.N;
  meas_sum_j_kernel<<<nblocks((long long)g.N * nk, 128), 128, 0, st>>>(f, g, T, klo, nk, kout);
  meas_sum_k_kernel<<<nblocks(NN, 128), 128, 0, st>>>(f, g, U, klo, nk);
  return cudaGetLastError();
}

cudaError_t launch_measure_sums_aos(const double *aos, int N, double *T, double *U, cudaStream_t st) {
  const long long NN = (long long)N * N;
  meas_sum_j_aos_kernel<<<nblocks(NN, 128), 128, 0, st>>>(aos, N, T);
  meas_sum_k_aos_kernel<<<nblocks(NN, 128), 128, 0, st>>>(aos, N, U);
  return cudaGetLastError();
}

cudaError_t launch_measure_finish(const double *T, const double *U, int N, double *dev_out, cudaStream_t st) {
  const MeasOut mo = meas_layout(dev_out, N);
  meas_walls_kernel<<<nblocks(3LL * kNObs * N, 128), 128, 0, st>>>(T, U, N, mo);
  const dft::Plan p = dft::make_plan(N);
  const size_t smem = wall_smem(p);
  if (smem > 48 * 1024) {
    const cudaError_t e = allow_smem(meas_dft_kernel, smem);
    if (e != cudaSuccess) return e;
  }
  meas_dft_kernel<<<dim3(kNObs, 3), kWallThreads, smem, st>>>(p, mo);
  meas_rotate_kernel<<<nblocks(3LL * (N / 2 + 1), 128), 128, 0, st>>>(N, mo);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Batched launchers.
int ideal_tile_dims(int tile, int *tx, int *ty) {
  if (tile == LGV_TILE_16x16) {
    *tx = 16;
    *ty = 16;
  } else {
    *tx = 32;
    *ty = 8;
  }
  return 0;
}

cudaError_t launch_batch_ideal(const RepDesc *d, const int *rep, const int *first, int nblocks, int tile,
                               int phase_phi, int phase_q, double dt, cudaStream_t st) {
  cudaError_t e;
  if (tile == LGV_TILE_16x16) {
    using T = IdealTile<16, 16>;
    if ((e = allow_smem(batch_ideal_kernel<16, 16>, T::SMEM)) != cudaSuccess) return e;
    return launch_pdl(batch_ideal_kernel<16, 16>, dim3(nblocks), dim3(256), T::SMEM, st, d, rep, first, phase_phi, phase_q,
                      dt);
  } else {
    using T = IdealTile<32, 8>;
    if ((e = allow_smem(batch_ideal_kernel<32, 8>, T::SMEM)) != cudaSuccess) return e;
    return launch_pdl(batch_ideal_kernel<32, 8>, dim3(nblocks), dim3(256), T::SMEM, st, d, rep, first, phase_phi, phase_q,
                      dt);
  }
}

bool batch_idx32(const RepDesc *hd, int nrep) {
  for (int r = 0; r < nrep; ++r)
    if (!idx32(hd[r].g)) return false;
  return true;
}

cudaError_t launch_batch_hb(const RepDesc *d, const EnsDyn *dyn, const int *rep, const int *first, int nblocks,
                            int phase, int parity, double dt, int ctr_off, bool i32, cudaStream_t st) {
  return launch_pdl(i32 ? batch_hb_kernel<unsigned> : batch_hb_kernel<long long>, dim3(nblocks), dim3(128), 0, st, d, dyn, rep,
                    first, phase, parity, dt, ctr_off);
}

int batch_run_blocks(int N) {
  const int H = N / 2, by = H <= kRunThreads ? kBatchRowSets * (kRunThreads / H) : 1, nrun = (N + kBatchSeg - 1) / kBatchSeg;
  const long long NN = (long long)N * N;
  return (int)std::max<long long>((NN + by - 1) / by, 6LL * nrun * ((NN + kRunThreads - 1) / kRunThreads));
}

size_t batch_run_smem(int N) {
  const int H = N / 2;
  return 2 * (size_t)(H <= kRunThreads ? (kRunThreads / H + 1) * H : H) * sizeof(double);
}

cudaError_t launch_batch_charge_dir(const RepDesc *d, const EnsDyn *dyn, const int *rep, const int *first, int nblocks,
                                    size_t smem, int phase, int ixyz, double dt, int ctr_off_order, bool small,
                                    cudaStream_t st) {
  return launch_pdl(small ? batch_charge_dir_kernel<unsigned> : batch_charge_dir_kernel<long long>, dim3(nblocks),
                    dim3(kRunThreads), smem, st, d, dyn, rep, first, phase, ixyz, dt, ctr_off_order);
}

int persist_grid(bool i32) {
  // per device (the shared-memory attribute is set on the current device)
  constexpr int kMaxDevices = 64;
  static int cached[kMaxDevices][2];
  static std::once_flag once;
  std::call_once(once, [] {
    for (auto &d : cached) d[0] = d[1] = -1;
  });
  int dev = 0, coop = 0, sms = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  int &c = cached[dev][i32 ? 1 : 0];
  if (c >= 0) return c;
  c = 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  const void *kern = i32 ? (const void *)ens_persistent_kernel<unsigned> : (const void *)ens_persistent_kernel<long long>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPersistSmem) != cudaSuccess)
    return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, 256, kPersistSmem) != cudaSuccess) return 0;
  c = per * sms;
  return c;
}

cudaError_t launch_ens_persistent(const PersistPlan &plan, const PersistPtrs &q, bool i32, cudaStream_t st) {
  const int grid = persist_grid(i32);
  if (grid <= 0) return cudaErrorCooperativeLaunchTooLarge;
  const void *kern = i32 ? (const void *)ens_persistent_kernel<unsigned> : (const void *)ens_persistent_kernel<long long>;
  void *args[] = {const_cast<PersistPlan *>(&plan), const_cast<PersistPtrs *>(&q)};
  return cudaLaunchCooperativeKernel(kern, grid, 256, args, kPersistSmem, st);
}

cudaError_t launch_batch_em(const RepDesc *d, const EnsDyn *dyn, const int *rep, const int *first, int nblocks,
                            int phase_in, double dt, int ctr_off, bool i32, cudaStream_t st) {
  return launch_pdl(i32 ? batch_em_kernel<unsigned> : batch_em_kernel<long long>, dim3(nblocks), dim3(kSiteThreads), 0, st, d,
                    dyn, rep, first, phase_in, dt, ctr_off);
}

cudaError_t launch_batch_em_fwd(const RepDesc *d, const int *rep, const int *first, int nblocks, int phase,
                                unsigned long long ctr, double t, double dt, double *partial, bool i32,
                                cudaStream_t st) {
  return launch_pdl(i32 ? batch_em_fwd_kernel<unsigned> : batch_em_fwd_kernel<long long>, dim3(nblocks), dim3(kSiteThreads),
                    0, st, d, rep, first, phase, ctr, t, dt, partial);
}

cudaError_t launch_batch_em_seg(const RepDesc *d, const DiffDesc *dd, const int *rep, const int *first, int nblocks,
                                int m, unsigned long long ctr, double t, double dt, bool i32, cudaStream_t st) {
  return launch_pdl(i32 ? batch_em_seg_kernel<unsigned> : batch_em_seg_kernel<long long>, dim3(nblocks), dim3(kSiteThreads),
                    0, st, d, dd, rep, first, m, ctr, t, dt);
}

cudaError_t launch_batch_em_adj(const RepDesc *d, const DiffDesc *dd, const int *rep, const int *first, int nblocks,
                                int m, int cur, int n, int b, int S, unsigned long long ctr, double t, double dt,
                                double *partial, bool i32, cudaStream_t st) {
  return launch_pdl(i32 ? batch_em_adj_kernel<unsigned> : batch_em_adj_kernel<long long>, dim3(nblocks), dim3(kSiteThreads),
                    0, st, d, dd, rep, first, m, cur, n, b, S, ctr, t, dt, partial);
}

cudaError_t launch_batch_phi_sum(const RepDesc *d, const int *rep, const int *first, int nblocks, int phase,
                                 double *partial, cudaStream_t st) {
  batch_phi_sum_kernel<<<nblocks, kSiteThreads, 0, st>>>(d, rep, first, phase, partial);
  return cudaGetLastError();
}

cudaError_t launch_batch_sum(const DiffDesc *dd, const int *first, const int *count, int nrep, int what,
                             const double *src, int nblocks, int row0, int nslot, cudaStream_t st) {
  const dim3 grid(nrep, nslot);
  if (what == 0) batch_sum_kernel<0><<<grid, kSumThreads, 0, st>>>(dd, first, count, src, nblocks, row0, 0);
  else if (what == 1) batch_sum_kernel<1><<<grid, kSumThreads, 0, st>>>(dd, first, count, src, nblocks, row0, 0);
  else batch_sum_kernel<2><<<nrep, kSumThreads, 0, st>>>(dd, first, count, nullptr, 0, 0, row0);
  return cudaGetLastError();
}

cudaError_t launch_batch_diff_copy(const RepDesc *d, const DiffDesc *dd, const int *rep, const int *first,
                                   int nblocks, int dir, int phase, int s, int b, int S, cudaStream_t st) {
  batch_diff_copy_kernel<<<nblocks, 128, 0, st>>>(d, dd, rep, first, dir, phase, s, b, S);
  return cudaGetLastError();
}

cudaError_t launch_ens_set(EnsDyn *dyn, unsigned long long ctr, double t, cudaStream_t st) {
  ens_set_kernel<<<1, 1, 0, st>>>(dyn, ctr, t);
  return cudaGetLastError();
}

cudaError_t launch_ens_advance(EnsDyn *dyn, unsigned long long dctr, double dt, cudaStream_t st) {
  return launch_pdl(ens_advance_kernel, dim3(1), dim3(1), 0, st, dyn, dctr, dt);
}

cudaError_t launch_batch_oavg(const RepDesc *d, const int *rep, const int *first, int nblocks, int phase_phi,
                              int phase_q, double *partial, int nrep, double *out, cudaStream_t st) {
  // per-replica block counts sit after the partial sums: count[r] = first[r+1] - first[r] in map order
  batch_oavg_kernel<<<nblocks, 128, 0, st>>>(d, rep, first, phase_phi, phase_q, partial);
  return cudaGetLastError();
}

cudaError_t launch_batch_oavg_final(const RepDesc *d, const int *first, const int *count, int nrep,
                                    const double *partial, double *out, cudaStream_t st) {
  batch_oavg_final_kernel<<<nblocks((long long)nrep * 11, 128), 128, 0, st>>>(d, first, nrep, count, partial, out);
  return cudaGetLastError();
}


// ---------------------------------------------------------------------------
// Euler-Maruyama adjoint launchers.
int sum_blocks(int N) {
  const dim3 g = site_grid(make_geo(N));
  return (int)(g.x * g.y);
}

int sum_slots(int nblocks) { return (int)std::max<long long>(1, std::min<long long>(32, (8LL << 20) / (32LL * nblocks))); }

cudaError_t launch_sum_rows(const double *src, int nslot, int nb, double scale, double *rows, double *tmp,
                            cudaStream_t st) {
  if (nb <= 4096) {
    sum_rows_kernel<<<nslot, kSumThreads, 0, st>>>(src, nb, scale, rows);
  } else {
    sum_rows_kernel<<<dim3(nslot, kSumSegs), kSumThreads, 0, st>>>(src, nb, 1.0, tmp);
    sum_rows_kernel<<<nslot, kSumThreads, 0, st>>>(tmp, kSumSegs, scale, rows);
  }
  return cudaGetLastError();
}

cudaError_t launch_em_adjoint(Fields phi, Fields lam_in, Fields lam_out, int N, const EmAdjArgs &a, double *partial,
                              cudaStream_t st) {
  const Geo g = make_geo(N);
  return launch_pdl(idx32(g) ? em_adjoint_kernel<unsigned> : em_adjoint_kernel<long long>, site_grid(g), dim3(kSiteThreads), 0,
                    st, phi, lam_in, lam_out, g, a, partial);
}

cudaError_t launch_ideal_adjoint(Fields u, Fields lam_in, Fields lam_out, Fields P1, Fields PB, Fields QB, int N,
                                 const IdealAdjArgs &a, double *partial, cudaStream_t st) {
  const Geo g = make_geo(N);
  const long long V = 2 * g.V2;
  cudaError_t e = launch_pdl(rot_phi_kernel, dim3(nblocks(V, kThreads)), dim3(kThreads), 0, st, u, P1, V, a.k);
  if (e == cudaSuccess)
    e = launch_pdl(ideal_adj_a_kernel, site_grid(g), dim3(kSiteThreads), 0, st, u, lam_in, P1, PB, QB, g, a, partial);
  if (e == cudaSuccess)
    e = launch_pdl(ideal_adj_b_kernel, site_grid(g), dim3(kSiteThreads), 0, st, u, lam_out, P1, PB, QB, g, a);
  return e;
}

cudaError_t launch_phi_sum(Fields f, int N, double *partial, cudaStream_t st) {
  const Geo g = make_geo(N);
  phi_sum_kernel<<<site_grid(g), kSiteThreads, 0, st>>>(f, g, partial);
  return cudaGetLastError();
}

cudaError_t launch_fill_phi(Fields f, int N, const double v[4], cudaStream_t st) {
  const Geo g = make_geo(N);
  const long long V = 2 * g.V2;
  fill_phi_kernel<<<nblocks(V, 256), 256, 0, st>>>(f, V, v[0], v[1], v[2], v[3]);
  return cudaGetLastError();
}

}  // namespace lgv
