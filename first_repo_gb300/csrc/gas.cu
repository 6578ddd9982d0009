// The reference's box gas step (grid.cpp) on the GPU, FP64, coupled to a pstep
// handle: the two-way-coupled gas response that turns the particle step's
// deposits into the gas disturbance (the learned correction's training runs).
//
// Compiled with -fmad=false; every element is computed with the reference's operand order
// except where a comment says otherwise. A kernel computes the interior cells and writes every
// value to its periodic ghost images too (what communicator.cpp:177-278's x, y, z passes leave),
// so stencils read the ghost layers and no refresh pass runs. GB300's FP64 rate (two lanes per
// SM and clock) bounds the step once the passes are fused: an operation a cell at 128^3 costs
// 3.3 us. The Poisson solve is the reference's fixed-point iteration on constant-coefficient FFT
// solves (poisson.cpp:391-462), five kernels an iteration: residual + x transform, y, z with the
// division by the wavenumbers and the way back, y, x + the update of P and its largest change.
// Interior sums (mean) and maxima are two-pass reductions in a fixed order of their own, so they
// round differently from the reference's sequential i-outer loop; together with the transform
// that is the source of difference from the CPU restatement.
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include "pstep_gas.h"
#include "pstep_internal.cuh"

namespace pgas {

constexpr double kPre[4] = {0.5, 0.5, 1., 1. / 6.};  // grid.cpp:16-23
constexpr double kPost[4] = {1. / 6., 1. / 3., 1. / 3., 1. / 6.};
constexpr int kT = 256;

enum {
  F_RU = 0, F_RU_INT = 3, F_RU_NEW = 6, F_RU_NP1 = 9, F_RHS_RU = 12, F_U = 15, F_IRF = 18 /* 1 / Rho_face */,
  F_P = 21, F_RHS_POIS, F_C, F_RHO, F_RHO_INT, F_RHO_NEW, F_RHO_NP1, F_IRHO /* 1 / Rho_new */, F_T, F_DIV, F_RHS_PT,
  F_CENTER, F_NF
};
// device scalars: P0 and its stage copies, mean of RHS_Part_Temp, scratch means (3), solve
// error (as bits), P0_new / R, -R / (Cp P0_new Vcell)
enum { S_P0, S_P0_INT, S_P0_NEW, S_P0_NP1, S_MEAN_E, S_MEAN, S_MEAN_Y, S_MEAN_Z, S_ERR, S_T, S_SRC, S_N };

struct Dim {
  int n, G;
  double idx, idx2;
};

__device__ __forceinline__ size_t ix(const Dim &d, int i, int j, int k) {
  return ((size_t)k * d.G + (size_t)j) * d.G + (size_t)i;
}

__device__ __forceinline__ int64_t gtid() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }

// interior cell of a thread of a (32, 8) block on a (n/32, n/8, n) grid
__device__ __forceinline__ bool cell_of(const Dim &d, int &i, int &j, int &k) {
  i = blockIdx.x * 32 + threadIdx.x + 1;
  j = blockIdx.y * 8 + threadIdx.y + 1;
  k = blockIdx.z + 1;
  return i <= d.n && j <= d.n;
}

// v at interior cell (i, j, k) and its periodic images in the ghost layers
struct Images {
  int i2, j2, k2;
  __device__ __forceinline__ Images(const Dim &d, int i, int j, int k)
      : i2(i == 1 ? d.n + 1 : (i == d.n ? 0 : -1)), j2(j == 1 ? d.n + 1 : (j == d.n ? 0 : -1)),
        k2(k == 1 ? d.n + 1 : (k == d.n ? 0 : -1)) {}
  __device__ __forceinline__ void put(const Dim &d, double *f, int i, int j, int k, double v) const {
    f[ix(d, i, j, k)] = v;
    if (i2 < 0 && j2 < 0 && k2 < 0) return;
    for (int c = 0; c < 2; ++c) {
      const int kk = c ? k2 : k;
      if (kk < 0) continue;
      for (int b = 0; b < 2; ++b) {
        const int jj = b ? j2 : j;
        if (jj < 0) continue;
        for (int a = 0; a < 2; ++a) {
          const int ii = a ? i2 : i;
          if (ii >= 0 && (a | b | c)) f[ix(d, ii, jj, kk)] = v;
        }
      }
    }
  }
};

struct V3 {
  double *p[3];
};
struct CV3 {
  const double *p[3];
};

// x / y with r = 1 / y at hand: one Newton step on the quotient (Markstein), which gives the
// correctly rounded quotient at 3 FP64 operations instead of a division's ten where nothing on the way
// leaves the normal range: both magnitudes in [2^-423, 2^424). Anything else (zeros, infinities,
// extremes) is divided.
__device__ __noinline__ double divide(double x, double y) { return x / y; }
__device__ __forceinline__ double quotient(double x, double y, double r) {
  constexpr uint32_t lo = 600u << 20, span = (1447u - 600u) << 20;
  const uint32_t ex = (uint32_t)__double2hiint(x) & 0x7fffffffu, ey = (uint32_t)__double2hiint(y) & 0x7fffffffu;
  const double q = x * r;
  if (ex - lo >= span || ey - lo >= span) {
    if ((ex | (uint32_t)__double2loint(x)) == 0u && ey - lo < span) return q;  // +-0, gas at rest
    return divide(x, y);
  }
  return fma(fma(-q, y, x), r, q);
}

// Update_Rho (grid.cpp:327-333): RHS_Rho = div(RU_int), Rho_np1, Rho_new; 1 / Rho_new beside it
__global__ void k_update_rho(Dim d, CV3 ru, const double *rho, double *np1, double *rnew, double *irho, double a_post,
                             double a_pre, int last) {
  int i, j, k;
  if (!cell_of(d, i, j, k)) return;
  const Images im(d, i, j, k);
  const size_t c = ix(d, i, j, k), off[3] = {1, (size_t)d.G, (size_t)d.G * d.G};
  const double rate = (ru.p[0][c + off[0]] - ru.p[0][c]) * d.idx + (ru.p[1][c + off[1]] - ru.p[1][c]) * d.idx +
                      (ru.p[2][c + off[2]] - ru.p[2][c]) * d.idx;
  const double a = np1[c] + a_post * rate;
  const double v = last ? a : rho[c] + a_pre * rate;
  im.put(d, np1, i, j, k, a);
  im.put(d, rnew, i, j, k, v);
  im.put(d, irho, i, j, k, 1. / v);
}

// U = RU_int / Rho_face(rho) (grid.cpp:662), T = (P0_new / R) / Rho_new (grid.cpp:676) and
// div(U) (the viscous term's, grid.cpp:389)
__global__ void k_velocity(Dim d, CV3 ru, CV3 irf, const double *rho, const double *rnew, const double *irho,
                           const double *sc, V3 u, double *T, double *div) {
  int i, j, k;
  if (!cell_of(d, i, j, k)) return;
  const Images im(d, i, j, k);
  const size_t c = ix(d, i, j, k), off[3] = {1, (size_t)d.G, (size_t)d.G * d.G};
  double s = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const size_t o = off[a];
    const double lo = quotient(ru.p[a][c], (rho[c] + rho[c - o]) * 0.5, irf.p[a][c]);
    const double hi = quotient(ru.p[a][c + o], (rho[c + o] + rho[c]) * 0.5, irf.p[a][c + o]);
    im.put(d, u.p[a], i, j, k, lo);
    s = a ? s + (hi - lo) * d.idx : (hi - lo) * d.idx;
  }
  im.put(d, div, i, j, k, s);
  im.put(d, T, i, j, k, quotient(sc[S_T], rnew[c], irho[c]));
}

// 1 / Rho_face(rho) of the start (grid::Initialize), and U, T there
__global__ void k_init_fields(Dim d, CV3 ru, const double *rho, const double *sc, V3 irf, V3 u, double *T) {
  int i, j, k;
  if (!cell_of(d, i, j, k)) return;
  const Images im(d, i, j, k);
  const size_t c = ix(d, i, j, k), off[3] = {1, (size_t)d.G, (size_t)d.G * d.G};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double f = (rho[c] + rho[c - off[a]]) * 0.5;
    im.put(d, irf.p[a], i, j, k, 1. / f);
    im.put(d, u.p[a], i, j, k, ru.p[a][c] / f);
  }
  im.put(d, T, i, j, k, sc[S_T] / rho[c]);
}

struct RuConst {
  double part, mu3_idx, mu_idx2, quarter, a_force, a_const, rho0, g[3], post, pre;
  int force, gravity, last;
};

// Update_RU_WOP (grid.cpp:387-425): RHS_RU = particle source + mu/3 grad(div U) + mu del2(U)
// - div(U RU) + forcing + buoyancy, RU_np1 and RU_new; 1 / Rho_face(Rho_new) beside it. Bound by
// its FP64 operations: sums before their common factor and fused operations, about 135 a cell
// (each product and sum by itself: 200 operations, 770 us at 128^3; this way 578 us).
__global__ void __launch_bounds__(256) k_update_ru(Dim d, RuConst q, CV3 u, CV3 rui, CV3 ru, const double *div,
                                                   const double *rho, const double *rnew, V3 rhs, V3 np1, V3 runew,
                                                   V3 irf) {
  int i, j, k;
  if (!cell_of(d, i, j, k)) return;
  const Images im(d, i, j, k);
  const size_t c = ix(d, i, j, k), off[3] = {1, (size_t)d.G, (size_t)d.G * d.G};
  const double dc = div[c], rc = rnew[c];
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const double *ue = u.p[e];
    const double uc = ue[c];
    double lap = 0.0, conv = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const size_t o = off[a];
      const double up = ue[c + o], um = ue[c - o], hi = up + uc, lo = uc + um;
      const double l = fma(-2.0, uc, up) + um;
      lap = a ? lap + l : l;
      // face(U_e, a) face(RU_a, e) at c + a and at c, each without its factor 1/4
      conv = fma(hi, rui.p[a][c + o] + rui.p[a][c + o - off[e]], conv);
      conv = fma(-lo, rui.p[a][c] + rui.p[a][c - off[e]], conv);
    }
    double r = q.part * rhs.p[e][c];
    r = fma(q.mu3_idx, dc - div[c - off[e]], r);
    r = fma(q.mu_idx2, lap, r);
    r = fma(-q.quarter, conv, r);
    if (q.force) {
      r += q.a_force * rui.p[e][c];
      if (e == 0) r += q.a_const;
    }
    if (q.gravity) r += ((rho[c] + rho[c - off[e]]) * 0.5 - q.rho0) * q.g[e];
    const double a = fma(q.post, r, np1.p[e][c]);
    im.put(d, rhs.p[e], i, j, k, r);
    im.put(d, np1.p[e], i, j, k, a);
    im.put(d, runew.p[e], i, j, k, q.last ? a : fma(q.pre, r, ru.p[e][c]));
    im.put(d, irf.p[e], i, j, k, 2. / (rc + rnew[c - off[e]]));
  }
}

// Compute_Div_U_new (grid.cpp:556-563) and Compute_RHS_Pois (:629-637) without its mean:
// divergence = k/Cp del2(1/Rho_new) - R/(Cp P0_new Vcell) RHS_Part_Temp, U = RU_new / Rho_face,
// RHS = (div(U) - divergence) / (dt pre); and the solve's centre coefficient
// -1 / I_F2C(1 / Rho_face) (poisson.cpp:391-400)
__global__ void __launch_bounds__(256) k_rhs_pois(Dim d, CV3 runew, CV3 irf, const double *rnew, const double *irho,
                                                  const double *pt, const double *sc, double kcp, double inv_dt,
                                                  int cooling, V3 u, double *div, double *rhs, double *centre) {
  int i, j, k;
  if (!cell_of(d, i, j, k)) return;
  const Images im(d, i, j, k);
  const size_t c = ix(d, i, j, k), off[3] = {1, (size_t)d.G, (size_t)d.G * d.G};
  const double two = 2 * irho[c];
  double lap = 0.0, s = 0.0, m = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const size_t o = off[a];
    const double l = (irho[c + o] - two + irho[c - o]) * d.idx2;
    lap = a ? lap + l : l;
    const double fl = irf.p[a][c], fh = irf.p[a][c + o];
    const double lo = quotient(runew.p[a][c], (rnew[c] + rnew[c - o]) * 0.5, fl);
    const double hi = quotient(runew.p[a][c + o], (rnew[c + o] + rnew[c]) * 0.5, fh);
    im.put(d, u.p[a], i, j, k, lo);
    s = a ? s + (hi - lo) * d.idx : (hi - lo) * d.idx;
    m = a ? m + (fl + fh) * 0.5 : (fl + fh) * 0.5;
  }
  const double src = cooling ? pt[c] - sc[S_MEAN] : pt[c];
  const double dv = kcp * lap + sc[S_SRC] * src;
  im.put(d, div, i, j, k, dv);
  rhs[c] = (s - dv) * inv_dt;
  centre[c] = -1. / ((1. / 3.) * m);
}

// Update_RU_WP (grid.cpp:651-657) and TimeAdvance_RK4 (:705-712)
__global__ void k_pressure_step(Dim d, const double *P, CV3 runew, V3 np1, V3 rui, const double *rnew, double *rhoi,
                                double a_post, double a_pre, int last) {
  int i, j, k;
  if (!cell_of(d, i, j, k)) return;
  const Images im(d, i, j, k);
  const size_t c = ix(d, i, j, k), off[3] = {1, (size_t)d.G, (size_t)d.G * d.G};
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const double g = (P[c] - P[c - off[e]]) * d.idx;
    const double a = np1.p[e][c] + a_post * g;
    im.put(d, np1.p[e], i, j, k, a);
    im.put(d, rui.p[e], i, j, k, last ? a : runew.p[e][c] + a_pre * g);
  }
  im.put(d, rhoi, i, j, k, rnew[c]);
}

// Correct_mean_RU (grid.cpp:566-572) and TimeAdvance (:315-325)
__global__ void k_end_step(Dim d, V3 np1, V3 ru, const double *rho_np1, double *rho, const double *sc, double mean_x) {
  int i, j, k;
  if (!cell_of(d, i, j, k)) return;
  const Images im(d, i, j, k);
  const size_t c = ix(d, i, j, k);
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    double v = np1.p[e][c] - sc[S_MEAN + e];
    if (e == 0) v += mean_x;
    im.put(d, np1.p[e], i, j, k, v);
    im.put(d, ru.p[e], i, j, k, v);
  }
  im.put(d, rho, i, j, k, rho_np1[c]);
}

__global__ void k_fill(double *x, double s, int64_t n) {
  int64_t q = gtid();
  if (q < n) x[q] = s;
}

// ----------------------------------------------------------- reductions
// one warp per (j, k) interior row; blockIdx.y picks the field
__global__ void k_rows(Dim d, CV3 f, double *rows) {
  const int64_t w = gtid() >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t nr = (int64_t)d.n * d.n;
  if (w >= nr) return;
  const int j = (int)(w % d.n) + 1, k = (int)(w / d.n) + 1;
  const double *r = f.p[blockIdx.y] + ix(d, 0, j, k);
  double s = 0.0;
  for (int i = lane + 1; i <= d.n; i += 32) s += r[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) rows[blockIdx.y * nr + w] = s;
}

// Update_P0 (grid.cpp:539-554) from the mean of RHS_Part_Temp
struct P0Const {
  int on, k3, cooling;
  double post, pre, r, cv, cp, vcell;
};
__device__ __forceinline__ void update_p0(double *sc, const P0Const &q) {
  const double dp0 = q.cooling ? 0.0 : -q.r / q.cv * sc[S_MEAN_E];
  sc[S_P0_NP1] += q.post * dp0;
  sc[S_P0_NEW] = q.k3 ? sc[S_P0_NP1] : sc[S_P0] + q.pre * dp0;
  sc[S_T] = sc[S_P0_NEW] / q.r;
  sc[S_SRC] = -q.r / (q.cp * sc[S_P0_NEW] * q.vcell);
}

// one block per field: sum of its row sums times inv into sc[slot + field]; then Update_P0
__global__ void __launch_bounds__(1024) k_rows_total(const double *rows, int64_t nr, double inv, double *sc, int slot,
                                                     P0Const q) {
  __shared__ double sm[32];
  const double *r0 = rows + blockIdx.x * nr;
  double s = 0.0;
  for (int64_t r = threadIdx.x; r < nr; r += 1024) s += r0[r];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = sm[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) {
      sc[slot + blockIdx.x] = s * inv;
      if (q.on) update_p0(sc, q);
    }
  }
}
__global__ void k_scalar_copy(double *sc, int dst, int src) { sc[dst] = sc[src]; }

// ------------------------------------------------------------------ FFT
// The right-hand side is real: two rows go through one complex transform along x and half the
// spectrum (n/2 + 1 bins) through y and z, 1/2 the FP64 work of a complex transform. Lines are
// transformed in shared memory, W of them side by side (element e of line w at e W + w), so that
// y and z move W neighbouring bins per row. Radix 2 in time with a +- w b as six fused
// operations (a + w b in four, the other sum as 2 a - that), the first two levels free of
// products: 38 operations a pair of points at n = 128 instead of 70.
__device__ __forceinline__ void fft_lines(double2 *s, int n, int logn, int W, const double2 *__restrict__ tw, int inv) {
  const double sg = inv ? -1.0 : 1.0;
  for (int t = threadIdx.x; t < W * (n >> 2); t += blockDim.x) {
    const int w = t % W, e = (t / W) << 2;
    double2 *p = s + e * W + w;
    const double2 a0 = p[0], a1 = p[W], a2 = p[2 * W], a3 = p[3 * W];
    const double2 b0 = make_double2(a0.x + a1.x, a0.y + a1.y), b1 = make_double2(a0.x - a1.x, a0.y - a1.y);
    const double2 b2 = make_double2(a2.x + a3.x, a2.y + a3.y), b3 = make_double2(a2.x - a3.x, a2.y - a3.y);
    // w = -i forward, +i backward
    const double2 m = inv ? make_double2(-b3.y, b3.x) : make_double2(b3.y, -b3.x);
    p[0] = make_double2(b0.x + b2.x, b0.y + b2.y);
    p[W] = make_double2(b1.x + m.x, b1.y + m.y);
    p[2 * W] = make_double2(b0.x - b2.x, b0.y - b2.y);
    p[3 * W] = make_double2(b1.x - m.x, b1.y - m.y);
  }
  __syncthreads();
  for (int lh = 2; lh < logn; ++lh) {
    const int half = 1 << lh, step = n >> (lh + 1);
    for (int t = threadIdx.x; t < W * (n >> 1); t += blockDim.x) {
      const int w = t % W, q = t / W, kk = q & (half - 1);
      double2 *pa = s + ((((q & ~(half - 1)) << 1) | kk)) * W + w, *pb = pa + half * W;
      const double2 f = tw[kk * step], a = *pa, b = *pb;
      const double wy = sg * f.y;
      const double rx = fma(-wy, b.y, fma(f.x, b.x, a.x)), ry = fma(wy, b.x, fma(f.x, b.y, a.y));
      *pa = make_double2(rx, ry);
      *pb = make_double2(fma(2.0, a.x, -rx), fma(2.0, a.y, -ry));
    }
    __syncthreads();
  }
}
__device__ __forceinline__ int bitrev(int e, int logn) { return (int)(__brev((unsigned)e) >> (32 - logn)); }

// One iteration's right-hand side (poisson.cpp:405-420), ((div(C grad P) - (RHS - mean)) centre),
// and its transform along x: W pairs of rows per CTA. The flux differences are summed with
// fused operations and scaled by idx^2 once.
__global__ void __launch_bounds__(256) k_res_fft_x(Dim d, int logn, int W, const double2 *__restrict__ tw,
                                                   const double *P, CV3 irf, const double *rhs, const double *centre,
                                                   double *sc, double2 *z) {
  extern __shared__ double2 s[];
  const int n = d.n, nh = n / 2 + 1;
  const int64_t row0 = (int64_t)blockIdx.x * 2 * W;
  if (blockIdx.x == 0 && threadIdx.x == 0) sc[S_ERR] = 0.0;
  const double mean = sc[S_MEAN], idx2 = d.idx * d.idx;
  const size_t oy = (size_t)d.G, oz = (size_t)d.G * d.G;
  for (int t = threadIdx.x; t < 2 * W * n; t += blockDim.x) {
    const int i = t & (n - 1), r = t >> logn;
    const int64_t row = row0 + r;
    const size_t c = ix(d, i + 1, (int)(row & (n - 1)) + 1, (int)(row >> logn) + 1);
    const double pc = P[c];
    double a = irf.p[0][c + 1] * (P[c + 1] - pc);
    a = fma(-irf.p[0][c], pc - P[c - 1], a);
    a = fma(irf.p[1][c + oy], P[c + oy] - pc, a);
    a = fma(-irf.p[1][c], pc - P[c - oy], a);
    a = fma(irf.p[2][c + oz], P[c + oz] - pc, a);
    a = fma(-irf.p[2][c], pc - P[c - oz], a);
    const double v = fma(a, idx2, mean - rhs[c]) * centre[c];
    reinterpret_cast<double *>(s)[2 * (bitrev(i, logn) * W + (r >> 1)) + (r & 1)] = v;
  }
  __syncthreads();
  fft_lines(s, n, logn, W, tw, 0);
  // the two rows' spectra, each twice (the factor 1/2 is in k_fft_x_back's scale)
  for (int t = threadIdx.x; t < W * nh; t += blockDim.x) {
    const int kx = t % nh, w = t / nh;
    const double2 a = s[kx * W + w], b = s[((n - kx) & (n - 1)) * W + w];
    double2 *o = z + (row0 + 2 * w) * nh + kx;
    o[0] = make_double2(a.x + b.x, a.y - b.y);
    o[nh] = make_double2(a.y + b.y, b.x - a.x);
  }
}

// along y, in place: CTA (tile of W bins, plane)
__global__ void __launch_bounds__(256) k_fft_y(int n, int logn, int W, const double2 *__restrict__ tw, int inv,
                                               double2 *z) {
  extern __shared__ double2 s[];
  const int nh = n / 2 + 1, x0 = blockIdx.x * W;
  double2 *pl = z + (int64_t)blockIdx.y * n * nh;
  for (int t = threadIdx.x; t < W * n; t += blockDim.x) {
    const int w = t % W, e = t / W;
    s[bitrev(e, logn) * W + w] = x0 + w < nh ? pl[(int64_t)e * nh + x0 + w] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  fft_lines(s, n, logn, W, tw, inv);
  for (int t = threadIdx.x; t < W * n; t += blockDim.x) {
    const int w = t % W, e = t / W;
    if (x0 + w < nh) pl[(int64_t)e * nh + x0 + w] = s[t];
  }
}

// along z, division by the modified wavenumbers (the zero mode is left alone) and back
__global__ void __launch_bounds__(256) k_fft_z(int n, int logn, int W, const double2 *__restrict__ tw,
                                               const double *__restrict__ kmod, double2 *z) {
  extern __shared__ double2 s[];
  const int nh = n / 2 + 1;
  const int64_t plane = (int64_t)n * nh;
  double2 *col = z + (int64_t)blockIdx.x * W;
  for (int t = threadIdx.x; t < W * n; t += blockDim.x) {
    const int w = t % W, e = t / W;
    s[bitrev(e, logn) * W + w] = col[e * plane + w];
  }
  __syncthreads();
  fft_lines(s, n, logn, W, tw, 0);
  for (int t = threadIdx.x; t < W * n; t += blockDim.x) {
    const int w = t % W, e = t / W, r = bitrev(e, logn);
    if (r < e) continue;  // this thread takes both of a pair
    const int c = (int)blockIdx.x * W + w;
    const double kxy = kmod[c % nh] + kmod[c / nh];
    const double de = kxy + kmod[e], dr = kxy + kmod[r];
    const double fe = c + e > 0 ? 1.0 / de : 1.0, fr = r == e ? fe : 1.0 / dr;
    const double2 a = s[e * W + w], b = s[r * W + w];
    s[r * W + w] = make_double2(a.x * fe, a.y * fe);
    if (r != e) s[e * W + w] = make_double2(b.x * fr, b.y * fr);
  }
  __syncthreads();
  fft_lines(s, n, logn, W, tw, 1);
  for (int t = threadIdx.x; t < W * n; t += blockDim.x) {
    const int w = t % W, e = t / W;
    col[e * plane + w] = s[t];
  }
}

// back along x: P += the solution, sc[S_ERR] = its largest magnitude (non-negative doubles order
// like their bits)
__global__ void __launch_bounds__(256) k_fft_x_back(Dim d, int logn, int W, const double2 *__restrict__ tw,
                                                    const double2 *z, double scale, double *P, double *sc) {
  extern __shared__ double2 s[];
  __shared__ double top[8];
  const int n = d.n, nh = n / 2 + 1;
  const int64_t row0 = (int64_t)blockIdx.x * 2 * W;
  for (int t = threadIdx.x; t < W * nh; t += blockDim.x) {
    const int kx = t % nh, w = t / nh;
    const double2 *o = z + (row0 + 2 * w) * nh + kx;
    const double2 a = o[0], b = o[nh];
    s[bitrev(kx, logn) * W + w] = make_double2(a.x - b.y, a.y + b.x);
    if (kx > 0 && kx < n / 2) s[bitrev(n - kx, logn) * W + w] = make_double2(a.x + b.y, b.x - a.y);
  }
  __syncthreads();
  fft_lines(s, n, logn, W, tw, 1);
  double m = 0.0;
  for (int t = threadIdx.x; t < 2 * W * n; t += blockDim.x) {
    const int i = t & (n - 1), r = t >> logn;
    const int64_t row = row0 + r;
    const int j = (int)(row & (n - 1)) + 1, k = (int)(row >> logn) + 1;
    const double v = reinterpret_cast<const double *>(s)[2 * (i * W + (r >> 1)) + (r & 1)] * scale;
    const Images im(d, i + 1, j, k);
    im.put(d, P, i + 1, j, k, P[ix(d, i + 1, j, k)] + v);
    m = fmax(m, fabs(v));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) top[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) m = fmax(m, top[q]);
    atomicMax(reinterpret_cast<unsigned long long *>(sc + S_ERR), (unsigned long long)__double_as_longlong(m));
  }
}

// interior n^3 (i fastest) -> ghosted
__global__ void k_scatter(Dim d, double *out, const double *lin) {
  int i, j, k;
  if (!cell_of(d, i, j, k)) return;
  const Images im(d, i, j, k);
  im.put(d, out, i, j, k, lin[((size_t)(k - 1) * d.n + (j - 1)) * d.n + (i - 1)]);
}

}  // namespace pgas

struct pgas_ctx {
  pgas_config c;
  pgas::Dim d;
  int device;
  cudaStream_t stream;
  double *f[pgas::F_NF];
  double *sc;      // device scalars
  double *rows;    // reduction scratch (n^2)
  double2 *z;      // half spectrum, n^2 (n/2 + 1)
  double2 *tw;     // twiddles, forward
  double *kmod;
  double r, vcell;
  int logn, last_iterations;
  int64_t size;
  char msg[256];
};

namespace {

using namespace pgas;

int gfail(pgas_ctx *g, int code, const char *what, cudaError_t e = cudaSuccess) {
  if (g) {
    if (e != cudaSuccess) snprintf(g->msg, sizeof g->msg, "%s: %s", what, cudaGetErrorString(e));
    else snprintf(g->msg, sizeof g->msg, "%s", what);
  }
  cudaGetLastError();
  return code;
}

#define GCUDA(g, x)                                                 \
  do {                                                              \
    cudaError_t e_ = (x);                                           \
    if (e_ != cudaSuccess) return gfail(g, PSTEP_ERR_CUDA, #x, e_); \
  } while (0)
#define GTRY(x)                      \
  do {                               \
    int rc_ = (x);                   \
    if (rc_ != PSTEP_OK) return rc_; \
  } while (0)

inline unsigned nblk(int64_t n) { return (unsigned)((n + kT - 1) / kT); }

struct Ops {
  pgas_ctx *g;
  cudaStream_t s;
  int64_t S;
  Dim d;
  dim3 grid, block;
  explicit Ops(pgas_ctx *g_)
      : g(g_), s(g_->stream), S(g_->size), d(g_->d), grid((d.n + 31) / 32, (d.n + 7) / 8, d.n), block(32, 8) {}
  double *F(int q) const { return g->f[q]; }
  V3 v3(int q) const { return {{g->f[q], g->f[q + 1], g->f[q + 2]}}; }
  CV3 c3(int q) const { return {{g->f[q], g->f[q + 1], g->f[q + 2]}}; }
  void copy(double *dst, const double *src) const {
    cudaMemcpyAsync(dst, src, sizeof(double) * S, cudaMemcpyDeviceToDevice, s);
  }
  // interior means of nf fields into sc[slot ..], then Update_P0 where q.on
  void means(CV3 f, int nf, int slot, P0Const q = P0Const{}) const {
    const int64_t nr = (int64_t)d.n * d.n;
    k_rows<<<dim3(nblk(nr * 32), (unsigned)nf), kT, 0, s>>>(d, f, g->rows);
    k_rows_total<<<(unsigned)nf, 1024, 0, s>>>(g->rows, nr, 1.0 / ((double)d.n * d.n * d.n), g->sc, slot, q);
  }
};

// lines per CTA: 32 KB of them where the line is short enough, at least 4; along y the count
// that leaves the fewest idle bins in the last tile of the half spectrum
int lines_per_cta(int n) { return n <= 256 ? 8 : 4; }
int lines_along_y(int n) {
  const int nh = n / 2 + 1, most = n <= 128 ? 16 : (n == 256 ? 8 : 4);
  int best = most;
  for (int w = most - 1; 2 * w > most; --w)
    if ((nh + w - 1) / w * w < (nh + best - 1) / best * best) best = w;
  return best;
}

int solve_poisson(pgas_ctx *g) {
  Ops o(g);
  const int n = g->c.n, W = lines_per_cta(n), Wy = lines_along_y(n), nh = n / 2 + 1;
  const size_t sx = sizeof(double2) * (size_t)W * n, sy = sizeof(double2) * (size_t)Wy * n;
  if (sx > 48 * 1024) {  // the opt-in belongs to the current device: set per solve
    GCUDA(g, cudaFuncSetAttribute(k_res_fft_x, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx));
    GCUDA(g, cudaFuncSetAttribute(k_fft_z, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx));
    GCUDA(g, cudaFuncSetAttribute(k_fft_x_back, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx));
  }
  if (sy > 48 * 1024) GCUDA(g, cudaFuncSetAttribute(k_fft_y, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sy));
  const unsigned bx = (unsigned)((int64_t)n * n / (2 * W)), bz = (unsigned)((int64_t)n * nh / W);
  const dim3 by((nh + Wy - 1) / Wy, n);
  const double scale = -0.5 / ((double)n * n * n);  // a power of two
  int it = 0;
  double error = 100;
  while (it < g->c.iterations && error > g->c.epsilon) {
    k_res_fft_x<<<bx, kT, sx, o.s>>>(o.d, g->logn, W, g->tw, o.F(F_P), o.c3(F_IRF), o.F(F_RHS_POIS), o.F(F_CENTER),
                                     g->sc, g->z);
    k_fft_y<<<by, kT, sy, o.s>>>(n, g->logn, Wy, g->tw, 0, g->z);
    k_fft_z<<<bz, kT, sx, o.s>>>(n, g->logn, W, g->tw, g->kmod, g->z);
    k_fft_y<<<by, kT, sy, o.s>>>(n, g->logn, Wy, g->tw, 1, g->z);
    k_fft_x_back<<<bx, kT, sx, o.s>>>(o.d, g->logn, W, g->tw, g->z, scale, o.F(F_P), g->sc);
    GCUDA(g, cudaMemcpyAsync(&error, g->sc + S_ERR, sizeof(double), cudaMemcpyDeviceToHost, o.s));
    GCUDA(g, cudaStreamSynchronize(o.s));
    it++;
  }
  g->last_iterations = it;
  return PSTEP_OK;
}

int update_particle(pgas_ctx *g, pstep_handle h, int k) {
  Ops o(g);
  k_velocity<<<o.grid, o.block, 0, o.s>>>(o.d, o.c3(F_RU_INT), o.c3(F_IRF), o.F(F_RHO_INT), o.F(F_RHO_NEW),
                                          o.F(F_IRHO), g->sc, o.v3(F_U), o.F(F_T), o.F(F_DIV));
  if (!h) {
    k_fill<<<nblk(o.S), kT, 0, o.s>>>(o.F(F_C), 0.0, o.S);
    for (int a = 0; a < 3; ++a) k_fill<<<nblk(o.S), kT, 0, o.s>>>(o.F(F_RHS_RU + a), 0.0, o.S);
    k_fill<<<nblk(o.S), kT, 0, o.s>>>(o.F(F_RHS_PT), 0.0, o.S);
    return PSTEP_OK;
  }
  GTRY(pstep_bind_velocity(h, o.F(F_U), o.F(F_U + 1), o.F(F_U + 2), 1));
  GTRY(pstep_bind_temperature(h, o.F(F_T), 1));
  GTRY(pstep_stage(h, k, kPre[k], kPost[k]));
  GTRY(pstep_get_field(h, PSTEP_FIELD_C, o.F(F_C), 1));
  if (g->c.twc) {
    for (int a = 0; a < 3; ++a) GTRY(pstep_get_field(h, PSTEP_FIELD_RU_X + a, o.F(F_RHS_RU + a), 1));
  } else {
    for (int a = 0; a < 3; ++a) k_fill<<<nblk(o.S), kT, 0, o.s>>>(o.F(F_RHS_RU + a), 0.0, o.S);  // grid.cpp:671
  }
  GTRY(pstep_get_field(h, PSTEP_FIELD_PART_TEMP, o.F(F_RHS_PT), 1));
  return PSTEP_OK;
}

int stage(pgas_ctx *g, pstep_handle h, int k) {
  Ops o(g);
  const pgas_config &c = g->c;
  const double dt = c.dt;
  const int last = k == 3;
  const CV3 pt = {{o.F(F_RHS_PT), o.F(F_RHS_PT), o.F(F_RHS_PT)}};
  // Update_Rho (grid.cpp:327-333), Update_P0 (:539-554), Update_Particle (:659-680)
  k_update_rho<<<o.grid, o.block, 0, o.s>>>(o.d, o.c3(F_RU_INT), o.F(F_RHO), o.F(F_RHO_NP1), o.F(F_RHO_NEW),
                                            o.F(F_IRHO), -(dt * kPost[k]), -dt * kPre[k], last);
  o.means(pt, 1, S_MEAN_E, P0Const{1, last, c.cooling, dt * kPost[k], dt * kPre[k], g->r, c.cv, c.cp, g->vcell});
  GTRY(update_particle(g, h, k));
  // Update_RU_WOP (grid.cpp:387-425)
  RuConst q;
  q.part = -c.mp / g->vcell;
  q.mu3_idx = c.mu0 / 3. * o.d.idx;
  q.mu_idx2 = c.mu0 * o.d.idx2;
  q.quarter = 0.25 * o.d.idx;
  q.a_force = c.a_force;
  q.a_const = -(c.a_force * c.rho0 * c.u0);
  q.rho0 = c.rho0;
  q.g[0] = c.gx; q.g[1] = c.gy; q.g[2] = c.gz;
  q.post = dt * kPost[k];
  q.pre = dt * kPre[k];
  q.force = c.a_force != 0.0;
  q.gravity = c.gx != 0.0 || c.gy != 0.0 || c.gz != 0.0;
  q.last = last;
  k_update_ru<<<o.grid, o.block, 0, o.s>>>(o.d, q, o.c3(F_U), o.c3(F_RU_INT), o.c3(F_RU), o.F(F_DIV), o.F(F_RHO_INT),
                                           o.F(F_RHO_NEW), o.v3(F_RHS_RU), o.v3(F_RU_NP1), o.v3(F_RU_NEW),
                                           o.v3(F_IRF));
  // Compute_Div_U_new (grid.cpp:556-563), Compute_RHS_Pois (:629-637)
  if (c.cooling) o.means(pt, 1, S_MEAN);
  k_rhs_pois<<<o.grid, o.block, 0, o.s>>>(o.d, o.c3(F_RU_NEW), o.c3(F_IRF), o.F(F_RHO_NEW), o.F(F_IRHO),
                                          o.F(F_RHS_PT), g->sc, c.k / c.cp, 1. / (dt * kPre[k]), c.cooling, o.v3(F_U),
                                          o.F(F_DIV), o.F(F_RHS_POIS), o.F(F_CENTER));
  o.means(CV3{{o.F(F_RHS_POIS), nullptr, nullptr}}, 1, S_MEAN);
  GCUDA(g, cudaGetLastError());
  // Solve_Poisson (grid.cpp:639-643)
  GTRY(solve_poisson(g));
  // Update_RU_WP (grid.cpp:651-657), TimeAdvance_RK4 (grid.cpp:705-712)
  k_pressure_step<<<o.grid, o.block, 0, o.s>>>(o.d, o.F(F_P), o.c3(F_RU_NEW), o.v3(F_RU_NP1), o.v3(F_RU_INT),
                                               o.F(F_RHO_NEW), o.F(F_RHO_INT), -(dt * kPost[k]), -(dt * kPre[k]), last);
  k_scalar_copy<<<1, 1, 0, o.s>>>(g->sc, S_P0_INT, S_P0_NEW);
  if (h) GTRY(pstep_end_stage(h));
  GCUDA(g, cudaGetLastError());
  return PSTEP_OK;
}

}  // namespace

extern "C" {

int pgas_create(const pgas_config *cfg, pgas_handle *out) {
  if (!cfg || !out) return PSTEP_ERR_ARG;
  *out = nullptr;
  const int n = cfg->n;
  int logn = 0;
  while ((1 << logn) < n) ++logn;
  if (n < 8 || n > 1024 || (1 << logn) != n) return PSTEP_ERR_CONFIG;
  if (!(cfg->l > 0) || !(cfg->dt > 0) || cfg->iterations < 1) return PSTEP_ERR_CONFIG;
  pgas_ctx *g = new pgas_ctx();
  memset((void *)g, 0, sizeof(pgas_ctx));
  g->c = *cfg;
  g->logn = logn;
  g->d.n = n;
  g->d.G = n + 2;
  const double dx = cfg->l / (double)n;
  g->d.idx = 1. / dx;
  g->d.idx2 = 1. / (dx * dx);
  g->vcell = dx * dx * dx;
  g->r = cfg->cp - cfg->cv;
  g->size = (int64_t)(n + 2) * (n + 2) * (n + 2);
  cudaGetDevice(&g->device);
  auto alloc = [&](void **p, size_t bytes) {
    if (cudaMalloc(p, bytes) != cudaSuccess) {
      cudaGetLastError();
      *p = nullptr;
      return false;
    }
    return true;
  };
  bool ok = true;
  for (int q = 0; q < F_NF && ok; ++q) {
    ok = alloc((void **)&g->f[q], sizeof(double) * g->size);
    if (ok) cudaMemset(g->f[q], 0, sizeof(double) * g->size);
  }
  ok = ok && alloc((void **)&g->sc, sizeof(double) * S_N) && alloc((void **)&g->rows, sizeof(double) * 3 * n * n) &&
       alloc((void **)&g->z, sizeof(double2) * (size_t)n * n * (n / 2 + 1)) &&
       alloc((void **)&g->tw, sizeof(double2) * n) && alloc((void **)&g->kmod, sizeof(double) * n);
  if (!ok) {
    pgas_destroy(g);
    return PSTEP_ERR_NOMEM;
  }
  // twiddles (cos, -sin of 2 pi m / n) and modified wavenumbers (poisson.cpp:428-448)
  const double two_pi = 2 * 3.141592653589793;
  double2 *tw = (double2 *)malloc(sizeof(double2) * n);
  for (int m = 0; m < n / 2; ++m) {
    const double a = two_pi * (double)m / (double)n;
    tw[m] = make_double2(cos(a), -sin(a));
  }
  cudaMemcpy(g->tw, tw, sizeof(double2) * (n / 2), cudaMemcpyHostToDevice);
  free(tw);
  double *km = (double *)malloc(sizeof(double) * n);
  {
    const double two_pi_over_l = two_pi / cfg->l;
    const double d2 = 2. / (dx * dx);
    for (int i = 0; i < n; ++i) {
      const double kk = ((i < n / 2) ? i : i - n) * two_pi_over_l;
      km[i] = (d2) * (1 - cos(kk * dx));
    }
  }
  cudaMemcpy(g->kmod, km, sizeof(double) * n, cudaMemcpyHostToDevice);
  free(km);
  if (cudaGetLastError() != cudaSuccess) {
    pgas_destroy(g);
    return PSTEP_ERR_CUDA;
  }
  *out = g;
  return PSTEP_OK;
}

int pgas_destroy(pgas_handle g) {
  if (!g) return PSTEP_ERR_ARG;
  if (g->stream) cudaStreamSynchronize(g->stream);
  else cudaDeviceSynchronize();
  for (int q = 0; q < F_NF; ++q)
    if (g->f[q]) cudaFree(g->f[q]);
  void *ps[5] = {g->sc, g->rows, g->z, g->tw, g->kmod};
  for (void *p : ps)
    if (p) cudaFree(p);
  delete g;
  return PSTEP_OK;
}

int pgas_set_stream(pgas_handle g, void *stream) {
  if (!g) return PSTEP_ERR_ARG;
  g->stream = (cudaStream_t)stream;
  return PSTEP_OK;
}

int pgas_init(pgas_handle g, pstep_handle h, const double *ru_x, const double *ru_y, const double *ru_z, const double *rho,
              double p0, int on_device) {
  if (!g || !ru_x || !ru_y || !ru_z || !rho) return PSTEP_ERR_ARG;
  Ops o(g);
  const int n = g->c.n;
  const int64_t n3 = (int64_t)n * n * n;
  const double *src[4] = {ru_x, ru_y, ru_z, rho};
  const int dst[4] = {F_RU, F_RU + 1, F_RU + 2, F_RHO};
  // interior n^3 (i fastest) -> ghosted, staged through the FFT buffer
  for (int q = 0; q < 4; ++q) {
    GCUDA(g, cudaMemcpyAsync(g->z, src[q], sizeof(double) * n3,
                             on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, o.s));
    k_scatter<<<o.grid, o.block, 0, o.s>>>(o.d, o.F(dst[q]), (const double *)g->z);
    GCUDA(g, cudaStreamSynchronize(o.s));  // the buffer is reused for the next field
  }
  k_fill<<<nblk(o.S), kT, 0, o.s>>>(o.F(F_P), 0.0, o.S);
  double sc[S_N] = {0};
  sc[S_P0] = sc[S_P0_INT] = sc[S_P0_NP1] = sc[S_P0_NEW] = p0;
  sc[S_T] = p0 / g->r;
  GCUDA(g, cudaMemcpyAsync(g->sc, sc, sizeof sc, cudaMemcpyHostToDevice, o.s));
  for (int a = 0; a < 3; ++a) {
    o.copy(o.F(F_RU_INT + a), o.F(F_RU + a));
    o.copy(o.F(F_RU_NP1 + a), o.F(F_RU + a));
  }
  o.copy(o.F(F_RHO_INT), o.F(F_RHO));
  o.copy(o.F(F_RHO_NP1), o.F(F_RHO));
  k_init_fields<<<o.grid, o.block, 0, o.s>>>(o.d, o.c3(F_RU), o.F(F_RHO_INT), g->sc, o.v3(F_IRF), o.v3(F_U), o.F(F_T));
  if (h) {
    GTRY(pstep_set_stream(h, g->stream));
    GTRY(pstep_bind_velocity(h, o.F(F_U), o.F(F_U + 1), o.F(F_U + 2), 1));
    GTRY(pstep_bind_temperature(h, o.F(F_T), 1));
    GTRY(pstep_prime(h));
    GTRY(pstep_get_field(h, PSTEP_FIELD_PART_TEMP, o.F(F_RHS_PT), 1));
  } else {
    k_fill<<<nblk(o.S), kT, 0, o.s>>>(o.F(F_RHS_PT), 0.0, o.S);
  }
  GCUDA(g, cudaGetLastError());
  GCUDA(g, cudaStreamSynchronize(o.s));
  return PSTEP_OK;
}

int pgas_stage(pgas_handle g, pstep_handle h, int k) {
  if (!g || k < 0 || k > 3) return PSTEP_ERR_ARG;
  if (h) GTRY(pstep_set_stream(h, g->stream));
  return stage(g, h, k);
}

int pgas_end_step(pgas_handle g, pstep_handle h) {
  if (!g) return PSTEP_ERR_ARG;
  Ops o(g);
  // Correct_mean_RU (grid.cpp:566-572, box) and TimeAdvance (grid.cpp:315-325)
  o.means(o.c3(F_RU_NP1), 3, S_MEAN);
  k_end_step<<<o.grid, o.block, 0, o.s>>>(o.d, o.v3(F_RU_NP1), o.v3(F_RU), o.F(F_RHO_NP1), o.F(F_RHO), g->sc,
                                          g->c.rho0 * g->c.u0);
  k_scalar_copy<<<1, 1, 0, o.s>>>(g->sc, S_P0, S_P0_NP1);
  if (h) GTRY(pstep_end_step(h));
  GCUDA(g, cudaGetLastError());
  return PSTEP_OK;
}

int pgas_step(pgas_handle g, pstep_handle h) {
  if (!g) return PSTEP_ERR_ARG;
  for (int k = 0; k < 4; ++k) GTRY(pgas_stage(g, h, k));
  return pgas_end_step(g, h);
}

int pgas_get_field(pgas_handle g, int id, double *dst, int on_device) {
  if (!g || !dst || id < 0 || id >= PGAS_NUM_FIELDS) return PSTEP_ERR_ARG;
  static const int map[PGAS_NUM_FIELDS] = {F_RU, F_RU + 1, F_RU + 2, F_RHO, F_P, F_T, F_U, F_U + 1, F_U + 2, F_C,
                                           F_RHS_RU, F_RHS_RU + 1, F_RHS_RU + 2, F_RHS_PT, F_DIV, F_RHO_NEW};
  GCUDA(g, cudaMemcpyAsync(dst, g->f[map[id]], sizeof(double) * g->size,
                           on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, g->stream));
  if (!on_device) GCUDA(g, cudaStreamSynchronize(g->stream));
  return PSTEP_OK;
}

int pgas_p0(pgas_handle g, double *p0) {
  if (!g || !p0) return PSTEP_ERR_ARG;
  GCUDA(g, cudaMemcpyAsync(p0, g->sc + S_P0, sizeof(double), cudaMemcpyDeviceToHost, g->stream));
  GCUDA(g, cudaStreamSynchronize(g->stream));
  return PSTEP_OK;
}

int pgas_last_iterations(pgas_handle g) { return g ? g->last_iterations : -1; }
const char *pgas_last_error(pgas_handle g) { return g ? g->msg : "null handle"; }

}  // extern "C"
