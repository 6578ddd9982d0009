// FP32 mixed form of the particle step (PSTEP_FP32).
//
// Storage (structure of arrays, 32 B per particle and set):
//   cell   uint32  trunc cell, 10 bits per dimension (i | j << 10 | k << 20)
//   ox,oy,oz float offset inside the cell in cell units, [0, 1)
//   u,v,w,T  float
// for the sets base, *_int, *_new and *_np1, plus RHS_T, 1/tau_p and the id.
// A position is x = (i + ox) * dx; the reference's trunc cell is i and its
// fractional part ox, its round() node is i + (ox >= 0.5). The periodic wrap is
// the cell index modulo n, so positions never leave [0, L).
//
// Temperatures (particle and gas) are stored as offsets from a reference
// temperature t_ref taken from the first data the handle sees (the first
// particle's T at upload, or the first interior cell of the first bound T
// field). The heat-transfer RHS is a difference of two nearly equal
// temperatures, (Tg - T_p); with offsets of size |T - t_ref| the fp32 rounding
// of that difference shrinks by the same factor (the trilinear weights sum to
// one, so interpolating the offset is exact algebra).
//
// Arithmetic: fields, offsets and the ODE in fp32. Deposits are summed exactly
// in 64-bit fixed point (each fp32 contribution scaled by a power of two chosen
// from device-side bounds, so no sum can overflow) and converted to fp64 with
// integer operations; integer addition is associative, so the result does not
// depend on the order of the adds and is the same on every run. Every brick of
// 8^3 cells is one work item: its particles (sorted by cell once per step, moving
// less than a cell per stage) are added into 32-bit sums in shared memory over the
// brick and the cells around it, and a second kernel sums the tiles that reach a
// cell. What a 32-bit sum cannot hold goes into 64-bit sums in memory. (Thin populations
// on large grids add to one 32-bit sum per cell in memory instead.) No per-stage sort.
//
// FP64 on GB300 runs at a small fraction of the fp32 rate, so this form keeps
// fp64 out of every per-particle operation: the only fp64 arithmetic left is
// the balance reduction over the grid.
#include <cuda_bf16.h>
#include <stdlib.h>
#include "scan.cuh"
#include "tc05.cuh"

namespace pstep {
}  // namespace pstep

namespace pstep {

enum { SBASE = 0, SINT = 1, SNEW = 2, SNP1 = 3 };
constexpr int kBr = 8;            // brick edge (cells) of the sort order
constexpr int kMaxN = 1024;       // 10 bits per cell coordinate
constexpr int kBoundSlots = 1024;

struct Set32 {
  uint32_t *cell;
  float *o[3];
  float *v[4];  // u v w T
};

// The deposit's work (see k_dep_tile): the sort's 8^3 bricks, or slices of those with more than
// kItemMax particles.
constexpr int kItemMax = 8192;
// Thin populations have no tiles: the tiles' way through memory, 41 B a cell each way, is then most of
// the deposit. A step at 512^3 with 4, 8, 16, 64, 512 cells a particle, tiles: 27.0, 23.3, 21.4, 19.5, 16.2 ms, a word
// a cell: 31.0, 21.7, 16.7, 12.3, 8.5; at 256^3 3.33, 2.89, 2.66, 2.44, 2.01 and 3.95, 2.83, 2.22, 1.64, 1.20. At 64^3,
// where all of it stays in L2, tiles are faster throughout (0.157 against 0.168 ms).
inline bool thin_population(int64_t particles, int64_t cells) {
  return cells >= (1 << 21) && particles * (cells >= (1 << 26) ? 6 : 8) <= cells;
}
constexpr int kBrickCells = kBr * kBr * kBr;
// A brick's tile: the int32 sums of its particles' contributions to the cells and faces they
// reach, one cell around the brick (momentum faces two above it along their own axis), as rows
// along x: RHS_Part_Temp and C (y, z in [-1, 8]), RHS_RU x (the same), y (y in [-1, 9]), z
// (z in [-1, 9]); a row is x in [-1, 8], [-1, 9] for RHS_RU x.
constexpr int kTE = kBr + 2;
constexpr int kRowsTri = kTE * kTE, kRowsFace = kTE * (kTE + 1);
constexpr int kRowC = kRowsTri, kRowX = 2 * kRowsTri, kRowY = 3 * kRowsTri, kRowZ = kRowY + kRowsFace,
              kRows = kRowZ + kRowsFace;
// In shared memory a row takes 12 words, x at 4 + x: cells 0 .. 7 aligned for 16-byte accesses, x =
// -1 before them, x = 8 and 9 in the next row's first words.
constexpr int kRowWords = 12;
// In memory the cells 0 .. 7 of all bricks of a brick row lie side by side (Work::mid), and a brick's
// words at x = -1, x = 8 and x = 9 by themselves (Work::side).
constexpr int kSideWords = 2 * kRows + kRowsTri;
struct Work {
  int4 *items;           // brick, first particle, end, 1 if a slice: slices from 0, whole bricks from slice_cap
  int32_t *counts;       // [0] slices, [1] whole bricks, [2] the running launch's next item
  uint8_t *dirty;        // per brick: 2 its tile in memory holds sums, 1 it is listed to be cleared, 0 zeros
  int32_t *extra_epoch;  // per brick: the last deposit launch that added to its cells in `extra`
  int32_t *word_epoch;   // thin populations, per brick: the last launch that added to its cells' words
  uint32_t *mid;         // [brick row (z, y)][kRows][cells along x]; thin: [5][cells in brick order]
  uint32_t *side;        // [brick][kSideWords]: x = -1, x = 8 (kRows each), x = 9 (RHS_RU x's rows)
  long long *extra;      // [5][cells in brick order]: what does not fit a tile's 32-bit words, exact
  int nb;                // bricks
  int64_t ncell;
  int64_t slice_cap;     // most slices
};

struct F32Form {
  Set32 set[4];
  float *rhs_t;
  float *itp;      // per-particle 1/tau_p or nullptr
  float *pp[7];    // per-particle mass ratio, itth, 1/(m Cvp), alpha, body acceleration x y z (or nullptr)
  float *gas[4];   // ug vg wg at x_int and Tg - t_ref at x_new of the last stage (PSTEP_KEEP_GAS)
  uint2 *drive;    // learned correction: the slip (3) and T_new - Tg the last stage's drag and heat transfer
                   // used, bf16 x 4 (a lagged estimate: bf16's 3 significant digits serve it)
  uint2 *corr_y;   // learned correction: the network output of the step's stage 0 (bf16 x 4)
  float *rhs_u[3];
  float *uf[3], *tf;  // fp32 ghosted copies of the bound fields
  int32_t *cell_start;  // n^3 + 1, brick-major order (per step)
  uint32_t *slots;    // kBoundSlots x 4 partial maxima (spread so blocks do not contend on one word)
  uint32_t *pslots;   // kBoundSlots x 2: the last stage's max u and max ug (order-preserving keys)
  int pmax_state;     // 0: none; 1: filled by this step's last stage; 2: valid for the base state
  int32_t *unsorted;  // sort_step's storage-order test word
  int32_t *se;        // fixed-point scale exponents per field
  unsigned long long *totals;  // exact integer sums, maxima, minima of the five fields (last deposit)
  double *fstat;               // per field: max, min, interior sum as fp64 (k_totals)
  int ext_ok[5];               // per field: its last deposit gathered the extrema too
  Work work;
  int32_t epoch;      // deposit launches so far
  int whole_since;    // a launch has written C's and RHS_Part_Temp's tiles since the work lists were made
  int thin;           // this step's deposits have no tiles (add_words)
  int mom_stale;      // a launch has written those alone: momentum rows of other bricks may hold sums
  int32_t *done;      // blocks of the running k_dep_gather that have finished
  void *corr_mem;     // learned correction: packed weight image + biases (device), or nullptr
  int sorted;
  int tref_set;
  double tref;        // temperature reference (see above)
  // host transfers: two staging slots of kStageArrays x kStageChunk doubles, filled and
  // drained on a copy stream of their own so that the copy of one chunk overlaps the
  // conversion of the other (created at the first host upload or download)
  double *stage[2];
  cudaStream_t copy_stream;
  cudaEvent_t ev_copied[2], ev_used[2];
};
constexpr int64_t kStageChunk = 1 << 22;  // particles per staged chunk
constexpr int kStageArrays = 7;

namespace {

__host__ __device__ inline uint32_t pack(int i, int j, int k) { return (uint32_t)i | ((uint32_t)j << 10) | ((uint32_t)k << 20); }
__host__ __device__ inline int ci_(uint32_t c) { return (int)(c & 1023u); }
__host__ __device__ inline int cj_(uint32_t c) { return (int)((c >> 10) & 1023u); }
__host__ __device__ inline int ck_(uint32_t c) { return (int)(c >> 20); }

// brick-major id of interior cell (i,j,k)
__host__ __device__ inline uint32_t brick_id(const Geom &G, int i, int j, int k) {
  const int nbx = G.n[0] / kBr, nby = G.n[1] / kBr;
  const int bx = i / kBr, by = j / kBr, bz = k / kBr;
  const int lx = i % kBr, ly = j % kBr, lz = k % kBr;
  return ((uint32_t)((bz * nby + by) * nbx + bx) * (kBr * kBr * kBr)) + (uint32_t)((lz * kBr + ly) * kBr + lx);
}

__device__ inline int wrapi(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

// offset o in cell units on top of cell index i: renormalise to [0, 1) and wrap
__device__ inline void renorm(int &i, float &o, int n) {
  float f = floorf(o);
  o -= f;
  i += (int)f;
  if (o >= 1.0f) { o -= 1.0f; i += 1; }
  i = wrapi(i, n);
}

__device__ inline long long glin3(const Geom &G, int i, int j, int k) { return glin(G, i, j, k); }

// the warp's maxima of 4 non-negative values, which order like their bit patterns (and are numbers: a
// maximum with 0 has dropped what is not), into one of the kBoundSlots (whole warps call; a block's
// maximum behind a barrier took 5% of the advance kernels)
__device__ __forceinline__ uint32_t warp_slot() {
  return (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) % kBoundSlots;
}
__device__ __forceinline__ void warp_max4(uint32_t *slots, float a0, float a1, float a2, float a3) {
  const uint32_t m0 = __reduce_max_sync(0xffffffffu, __float_as_uint(a0)),
                 m1 = __reduce_max_sync(0xffffffffu, __float_as_uint(a1)),
                 m2 = __reduce_max_sync(0xffffffffu, __float_as_uint(a2)),
                 m3 = __reduce_max_sync(0xffffffffu, __float_as_uint(a3));
  const int lane = threadIdx.x & 31;
  const uint32_t m = lane == 0 ? m0 : (lane == 1 ? m1 : (lane == 2 ? m2 : m3));
  if (lane < 4 && m) atomicMax(&slots[warp_slot() * 4 + lane], m);
}

// order-preserving 32-bit key of a float (larger float, larger key; 0 is below every key)
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// the same of 2 signed values as order keys (-infinity, or not a number: none)
__device__ __forceinline__ void warp_max2_signed(uint32_t *slots, float a0, float a1) {
  const uint32_t m0 = __reduce_max_sync(0xffffffffu, a0 > -INFINITY ? order_key(a0) : 0u),
                 m1 = __reduce_max_sync(0xffffffffu, a1 > -INFINITY ? order_key(a1) : 0u);
  const int lane = threadIdx.x & 31;
  const uint32_t m = lane == 0 ? m0 : m1;
  if (lane < 2 && m) atomicMax(&slots[warp_slot() * 2 + lane], m);
}

struct C32 {
  float dt_pre, dt_post, dt_pre_is, dt_post_is;
  float dpre_idx[3], dpost_idx[3];  // dt*pre/dx, dt*post/dx per dimension
  float itp, g[3], alpha, itth;
  float is;  // 1/(mp*Cvp) (particle.cpp:485)
};

enum { PP_MASS = 0, PP_ITTH, PP_HEAT_IS, PP_ALPHA, PP_ACC };  // F32Form::pp slots (PP_ACC + d)

// learned correction: the drive slip / temperature difference at most 10x the plain one
constexpr float kDriveCap = 10.f;

// One particle's stage: everything the advance kernels read, and the gas velocity
// interpolated at x_int (particle.cpp:340-360).
struct Adv {
  uint32_t cb, cint, cacc;
  float ob[3], oin[3], oac[3], vb[4], vin[4], vac[4];
  float rhs_t_old, itp, itth, alpha, dpre_is, dpost_is, gacc[3];
  float gas[3];
};

// the particle's x_int cell, offsets and velocity and the gas velocity there (particle.cpp:340-360)
template <int K>
__device__ __forceinline__ void adv_load_gas(const Geom &G, const F32Form &f, int64_t p, Adv &a) {
  const Set32 &I = (K == 0) ? f.set[SBASE] : f.set[SINT];
  a.cint = I.cell[p];
#pragma unroll
  for (int d = 0; d < 3; ++d) { a.oin[d] = I.o[d][p]; a.vin[d] = I.v[d][p]; }
  const int ii = ci_(a.cint) + 1, jj = cj_(a.cint) + 1, kk = ck_(a.cint) + 1;
  const float xl = a.oin[0], yl = a.oin[1], zl = a.oin[2];
  a.gas[0] = xl * f.uf[0][glin3(G, ii + 1, jj, kk)] + (1.f - xl) * f.uf[0][glin3(G, ii, jj, kk)];
  a.gas[1] = yl * f.uf[1][glin3(G, ii, jj + 1, kk)] + (1.f - yl) * f.uf[1][glin3(G, ii, jj, kk)];
  a.gas[2] = zl * f.uf[2][glin3(G, ii, jj, kk + 1)] + (1.f - zl) * f.uf[2][glin3(G, ii, jj, kk)];
}

// everything else the stage reads
template <int K>
__device__ __forceinline__ void adv_load_rest(const Geom &G, const F32Form &f, const C32 &c, int64_t p, Adv &a) {
  const Set32 &B = f.set[SBASE];
  const Set32 &I = (K == 0) ? f.set[SBASE] : f.set[SINT];
  const Set32 &A = (K == 0) ? f.set[SBASE] : f.set[SNP1];
  a.cb = B.cell[p];
  a.cacc = A.cell[p];
#pragma unroll
  for (int d = 0; d < 3; ++d) { a.ob[d] = B.o[d][p]; a.oac[d] = A.o[d][p]; }
#pragma unroll
  for (int q = 0; q < 4; ++q) { a.vb[q] = B.v[q][p]; a.vac[q] = A.v[q][p]; }
  a.vin[3] = I.v[3][p];
  a.rhs_t_old = f.rhs_t[p];
  a.itp = f.itp ? f.itp[p] : c.itp;
  a.itth = f.pp[PP_ITTH] ? f.pp[PP_ITTH][p] : c.itth;
  a.alpha = f.pp[PP_ALPHA] ? f.pp[PP_ALPHA][p] : c.alpha;
  a.dpre_is = f.pp[PP_HEAT_IS] ? c.dt_pre * f.pp[PP_HEAT_IS][p] : c.dt_pre_is;
  a.dpost_is = f.pp[PP_HEAT_IS] ? c.dt_post * f.pp[PP_HEAT_IS][p] : c.dt_post_is;
#pragma unroll
  for (int d = 0; d < 3; ++d) a.gacc[d] = f.pp[PP_ACC + d] ? f.pp[PP_ACC + d][p] : c.g[d];
}

template <int K>
__device__ __forceinline__ void adv_load(const Geom &G, const F32Form &f, const C32 &c, int64_t p, Adv &a) {
  adv_load_gas<K>(G, f, p, a);
  adv_load_rest<K>(G, f, c, p, a);
}

// The rest of the stage for one particle, with a.gas the gas velocity to use; with
// ty != 0 the interpolated gas temperature Tg is replaced by Tg - ty * dT, dT the
// previous stage's T_new - Tg (td_prev, or the current T_new - Tg when there is
// none): the learned correction of the particle's own heating. Returns the
// T_new - Tg the heat transfer used.
template <int K>
__device__ __forceinline__ float adv_finish_t(const Geom &G, const F32Form &f, const C32 &c, int twc, int64_t p, Adv &a,
                                              float ty, float td_prev, int32_t *__restrict__ err, float &mu0, float &mu1,
                                              float &mu2, float &mt) {
  // positions (particle.cpp:314-338) in cell units
  int ia[3] = {ci_(a.cacc), cj_(a.cacc), ck_(a.cacc)};
  int ib[3] = {ci_(a.cb), cj_(a.cb), ck_(a.cb)};
  int in_[3];
  float on[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    a.oac[d] += c.dpost_idx[d] * a.vin[d];
    renorm(ia[d], a.oac[d], G.n[d]);
    if (K != 3) {
      on[d] = a.ob[d] + c.dpre_idx[d] * a.vin[d];
      in_[d] = ib[d];
      renorm(in_[d], on[d], G.n[d]);
    } else {
      on[d] = a.oac[d];
      in_[d] = ia[d];
    }
  }
  // x_new more than one cell from the step-start cell along some axis is reported: the step is meant for
  // moves of at most one cell (the deposit takes any: what leaves a brick's tile goes into the 64-bit sums)
  {
    bool far = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      int r = in_[d] - ib[d];
      r += (r < -(G.n[d] >> 1)) ? G.n[d] : 0;
      r -= (r > (G.n[d] >> 1)) ? G.n[d] : 0;
      far |= (r < -1 || r > 1);
    }
    if (far) atomicOr(err, kErrMove);
  }
  // velocity and temperature (particle.cpp:362-399, 480-496)
  float rhs[3], vn[4];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    rhs[d] = (a.gas[d] - a.vin[d]) * a.itp;
    a.vac[d] += c.dt_post * (rhs[d] + a.gacc[d]);
    vn[d] = (K != 3) ? a.vb[d] + c.dt_pre * (rhs[d] + a.gacc[d]) : a.vac[d];
  }
  a.vac[3] += a.dpost_is * (a.rhs_t_old + a.alpha);
  vn[3] = (K != 3) ? a.vb[3] + a.dpre_is * (a.rhs_t_old + a.alpha) : a.vac[3];

  // trilinear T at x_new (particle.cpp:430-456): node = cell + h, x_l = o - h + 1/2
  const int hx = on[0] >= 0.5f, hy = on[1] >= 0.5f, hz = on[2] >= 0.5f;
  const int ni = in_[0] + hx + 1, nj = in_[1] + hy + 1, nk = in_[2] + hz + 1;  // ghosted node
  const float *T = f.tf;
  const float wx = on[0] - hx + 0.5f, wy = on[1] - hy + 0.5f, wz = on[2] - hz + 0.5f;
  float tg = wx * wy * wz * T[glin3(G, ni, nj, nk)] + (1.f - wx) * wy * wz * T[glin3(G, ni - 1, nj, nk)] +
             wx * (1.f - wy) * wz * T[glin3(G, ni, nj - 1, nk)] + wx * wy * (1.f - wz) * T[glin3(G, ni, nj, nk - 1)] +
             (1.f - wx) * (1.f - wy) * wz * T[glin3(G, ni - 1, nj - 1, nk)] +
             (1.f - wx) * wy * (1.f - wz) * T[glin3(G, ni - 1, nj, nk - 1)] +
             wx * (1.f - wy) * (1.f - wz) * T[glin3(G, ni, nj - 1, nk - 1)] +
             (1.f - wx) * (1.f - wy) * (1.f - wz) * T[glin3(G, ni - 1, nj - 1, nk - 1)];
  if (ty != 0.f) {
    const float dtn = vn[3] - tg;
    const float cap = kDriveCap * fabsf(dtn);
    const float td = td_prev != 0.f ? (fabsf(td_prev) <= cap ? td_prev : copysignf(cap, td_prev)) : dtn;
    tg -= ty * td;
  }
  const float rhs_t_new = (tg - vn[3]) * a.itth;
  if (!isfinite(rhs_t_new) || !isfinite(vn[0]) || !isfinite(vn[1]) || !isfinite(vn[2]) || !isfinite(on[0]) ||
      !isfinite(on[1]) || !isfinite(on[2]))
    atomicOr(err, kErrNonFinite);

  // stores
  const Set32 &N = f.set[SNEW];
  const Set32 &P = f.set[SNP1];
  N.cell[p] = pack(in_[0], in_[1], in_[2]);
  P.cell[p] = pack(ia[0], ia[1], ia[2]);
#pragma unroll
  for (int d = 0; d < 3; ++d) { N.o[d][p] = on[d]; P.o[d][p] = a.oac[d]; }
#pragma unroll
  for (int q = 0; q < 4; ++q) { N.v[q][p] = vn[q]; P.v[q][p] = a.vac[q]; }
  // the momentum deposit carries the particle's mass relative to cfg.mp
  const float mrel = f.pp[PP_MASS] ? f.pp[PP_MASS][p] : 1.f;
  if (twc) {
#pragma unroll
    for (int d = 0; d < 3; ++d) f.rhs_u[d][p] = rhs[d] * mrel;
  }
  f.rhs_t[p] = rhs_t_new;
  if (f.gas[0]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) f.gas[d][p] = a.gas[d];
    f.gas[3][p] = tg;
  }
  mu0 = fmaxf(mu0, fabsf(rhs[0] * mrel));
  mu1 = fmaxf(mu1, fabsf(rhs[1] * mrel));
  mu2 = fmaxf(mu2, fabsf(rhs[2] * mrel));
  mt = fmaxf(mt, fabsf(rhs_t_new));
  return vn[3] - tg;
}

template <int K>
__device__ __forceinline__ void adv_finish(const Geom &G, const F32Form &f, const C32 &c, int twc, int64_t p, Adv &a,
                                           int32_t *__restrict__ err, float &mu0, float &mu1, float &mu2, float &mt) {
  (void)adv_finish_t<K>(G, f, c, twc, p, a, 0.f, 0.f, err, mu0, mu1, mu2, mt);
}

template <int K>
__device__ __forceinline__ float adv_finish_mlp(const Geom &G, const F32Form &f, const C32 &c, int twc, int64_t p,
                                                Adv &a, float ty, float td_prev, int32_t *__restrict__ err, float &mu0,
                                                float &mu1, float &mu2, float &mt) {
  return adv_finish_t<K>(G, f, c, twc, p, a, ty, td_prev, err, mu0, mu1, mu2, mt);
}

// Bound by memory latency: a particle's 180 bytes a stage and the field values behind its cell are two
// trips, so what counts is the warps in flight. 256 threads a block at 78 and 105 registers (stages
// 0, 3 and 1, 2) and a block's maxima behind a barrier: 495, 704, 704, 586 us at 256^3 x 2^24; blocks of
// 128, nine on an SM (56 registers; stage 3, which reads less, six), maxima by warp:
// 440, 625, 625, 526 us (eight an SM 453, 625, 623, 568; six 517, 677, 676, 535).
constexpr int kAdvThreads = 128;
template <int K>
__global__ void __launch_bounds__(kAdvThreads, K == 3 ? 6 : 9) k_advance32(Geom G, F32Form f, C32 c, int twc, int64_t n,
                                                   int32_t *__restrict__ err) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  float mu0 = 0.f, mu1 = 0.f, mu2 = 0.f, mt = 0.f, umax = -INFINITY, gmax = -INFINITY;
  if (p < n) {
    Adv a;
    adv_load<K>(G, f, c, p, a);
    adv_finish<K>(G, f, c, twc, p, a, err, mu0, mu1, mu2, mt);
    umax = a.vac[0];
    gmax = a.gas[0];
  }
  // bounds for the fixed-point scales (order-independent maxima)
  warp_max4(f.slots, mu0, mu1, mu2, mt);
  // the last stage: max u of the step's result and max ug (grid.cpp:726-727)
  if (K == 3) warp_max2_signed(f.pslots, umax, gmax);
}

// ----------------------------------------------------------------------------
// The learned correction (pstep_set_correction).
//
// The network runs in its own kernel, k_corr_net, at stage 0 of every step (or at
// every stage, pstep_correction.every_stage): persistent CTAs of two warpgroups;
// each warpgroup owns tiles of 128 particles, one particle per thread, and thread
// t's network row is tensor-memory lane t of the warpgroup's 64 columns. Per tile:
// the plain interpolation at x_int and the features in registers, the feature row
// as bf16 to shared memory, three tcgen05 MMAs (16 -> 64 -> 64 -> 16 columns; each
// layer's accumulator reuses the columns of the one before, which has been read),
// bias and SiLU between them on 16-column chunks, and the network output (bf16 x 4,
// zero for particles outside the training ranges) to memory. The two warpgroups
// synchronise with named barriers only, so one's MMAs overlap the other's loads and
// epilogues; four CTAs per SM keep eight warpgroups in flight. The advance of every
// stage (k_advance32_corr) applies the kept output with that stage's own drive slip
// and prior: within a step a particle moves a few hundredths of a cell and its slip
// hardly changes, so one inference per step serves the step's four stages.
// Particles outside the training ranges keep the plain interpolation.
namespace corr {
constexpr int kRows = 128, kInP = 16, kHid = 64, kOutP = 16, kGroups = 2, kThreads = kRows * kGroups;
// shared memory: weight image W1 | W2 | W3 (bf16 tiles), biases, then per warpgroup
// X [128 x 16], H [128 x 64] (layer 1, then layer 2 output), its MMA mbarrier and an
// idle mbarrier that nothing signals (the wait-timeout test, pstep_set_wait_limit)
constexpr uint32_t W1 = 0, W2 = W1 + kHid * kInP * 2, W3 = W2 + kHid * kHid * 2, kImage = W3 + kOutP * kHid * 2;
constexpr uint32_t BIAS = kImage, GROUPS = 13 * 1024;
constexpr uint32_t G_XA = 0, G_H = G_XA + kRows * kInP * 2, G_BAR = G_H + kRows * kHid * 2, G_IDLE = G_BAR + 8,
                   kGroupStride = 21 * 1024;
constexpr uint32_t TSLOT = GROUPS + kGroups * kGroupStride, kBytes = TSLOT + 16;
static_assert(BIAS + (kHid + kHid + kOutP) * 4 <= GROUPS, "correction smem");
static_assert(G_IDLE + 8 <= kGroupStride, "correction group smem");
// with this much shared memory at most 4 CTAs fit on an SM (228 KB), so their
// 4 x 128 tensor-memory columns never exceed the 512 an SM has and no allocation waits
constexpr uint32_t kAlloc = kBytes;
static_assert(5 * (kAlloc + 1024) > 228 * 1024, "more than 4 correction CTAs per SM");
constexpr uint32_t kWaitLimit = 1u << 22;
}  // namespace corr

struct CorrDev {
  const uint4 *image;  // kImage bytes
  const float *bias;   // b1[64] b2[64] b3[16]
  float shift[10], scale[10], lo[4], hi[4];
  float inv_nu;        // 1 / kinematic viscosity of the gas
  float inv_prior_re;  // 1 / prior_re (0: outputs not scaled by the prior)
  float dp_per_itth;   // d_p = itth * dp_per_itth (1 / (Nu PI k)), per-particle diameters
  float dp;            // scalar diameter (no per-particle itth)
  float idx;           // 1 / dx
  uint32_t wait_limit; // polls of each MMA completion wait (the drain before freeing tensor memory
                       // always allows corr::kWaitLimit)
  uint32_t idle_first; // 1: each warpgroup's first completion wait polls the idle barrier (test)
  float drive_cap;     // the drive slip at most this many times the plain slip
};

static_assert(sizeof(CorrDev) <= sizeof(((pstep_ctx *)nullptr)->corr_dev), "correction constants");

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// warpgroup-local barrier (named barrier 1 + group, 128 threads; immediate ids)
__device__ __forceinline__ void group_bar(int wg) {
  if (wg == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
  else asm volatile("bar.sync 2, 128;" ::: "memory");
}
__device__ __forceinline__ bool group_and(int wg, bool v) {
  uint32_t out;
  if (wg == 0)
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(out)
        : "r"(v ? 1u : 0u)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(out)
        : "r"(v ? 1u : 0u)
        : "memory");
  return out != 0;
}
__device__ __forceinline__ void group_sync_mma(int wg) {
  tc05::fence_smem_async();
  tc05::fence_before();
  group_bar(wg);
  tc05::fence_after();
}
__device__ __forceinline__ bool group_wait(int wg, uint64_t *mbar, uint32_t &phase, uint32_t limit) {
  const bool ok = tc05::mbar_wait(mbar, phase, limit);
  tc05::fence_after();
  const bool all = group_and(wg, ok);
  if (all) phase ^= 1u;
  return all;
}

// 16 accumulator columns + bias -> SiLU -> bf16, into row r, columns [c0, c0+16) of a 64-column tile
// SiLU z * sigmoid(z) = u (1 + tanh u) = u tanh(u) + u with u = z/2 and the hardware
// tanh approximation; with the halved bias hb, u = v/2 + hb is one fma
__device__ __forceinline__ float silu_half(float v, float hb) {
  const float u = fmaf(v, 0.5f, hb);
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
  return fmaf(u, t, u);
}

// bias: the layer's bias halved
__device__ __forceinline__ void silu_chunk_to_tile(uint8_t *tile, int r, int c0, const float (&v)[16],
                                                   const float *bias) {
  float h[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) h[q] = silu_half(v[q], bias[c0 + q]);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint4 w;
    w.x = pack_bf16x2(h[half * 8 + 0], h[half * 8 + 1]);
    w.y = pack_bf16x2(h[half * 8 + 2], h[half * 8 + 3]);
    w.z = pack_bf16x2(h[half * 8 + 4], h[half * 8 + 5]);
    w.w = pack_bf16x2(h[half * 8 + 6], h[half * 8 + 7]);
    *reinterpret_cast<uint4 *>(tile + tc05::tile_off(r, c0 + half * 8, corr::kHid)) = w;
  }
}

// the drive slip: the previous stage's (at most `cap` x the plain one), or the plain slip
__device__ __forceinline__ void drive_slip(const uint2 dw, const float (&s)[3], float smag, float cap, float &sdrv,
                                           float (&dir)[3], float &dmag_used) {
  const float d0 = bf16_lo(dw.x), d1 = bf16_hi(dw.x), d2 = bf16_lo(dw.y);
  const float dmag = sqrtf(d0 * d0 + d1 * d1 + d2 * d2);
  if (dmag > 0.f) {
    sdrv = fminf(dmag, cap * smag);
    dir[0] = d0; dir[1] = d1; dir[2] = d2;
    dmag_used = dmag;
  } else {
    sdrv = smag;
    dir[0] = s[0]; dir[1] = s[1]; dir[2] = s[2];
    dmag_used = smag;
  }
}

__device__ __forceinline__ float prior_of(const CorrDev &cd, float dpdx, float rep) {
  return cd.inv_prior_re > 0.f ? dpdx / (1.f + rep / dpdx * cd.inv_prior_re) : 1.f;
}

__device__ __forceinline__ float particle_dp(const F32Form &f, const CorrDev &cd, int64_t p, float itth) {
  return f.pp[PP_ITTH] ? itth * cd.dp_per_itth : cd.dp;
}

// A particle's network inputs as loaded from memory (x_int cell, offsets and velocity,
// the drive state), fetched one tile ahead so that their memory round trip overlaps the
// current tile's tensor-core work
struct NetRaw {
  uint32_t cell;
  float o[3], v[3];
  uint2 drive;
};
template <int K>
__device__ __forceinline__ void net_raw_load(const F32Form &f, int64_t p, int64_t n, NetRaw &r) {
  if (p >= n) return;
  const Set32 &I = (K == 0) ? f.set[SBASE] : f.set[SINT];
  r.cell = I.cell[p];
#pragma unroll
  for (int d = 0; d < 3; ++d) { r.o[d] = I.o[d][p]; r.v[d] = I.v[d][p]; }
  r.drive = f.drive[p];
}

// The network of every particle at its x_int position: features from the plain
// interpolation and the drive state of the previous stage, three tcgen05 layers,
// the output (bf16 x 4) to f.corr_y (zero outside the training ranges).
template <int K>
__global__ void __launch_bounds__(corr::kThreads, 4) k_corr_net(Geom G, F32Form f, C32 c, int64_t n,
                                                                int32_t *__restrict__ err, CorrDev cd) {
  extern __shared__ __align__(1024) uint8_t sm[];
  using namespace tc05;
  const int tid = threadIdx.x, wg = tid >> 7, lt = tid & (corr::kRows - 1), warp = tid >> 5;
  uint8_t *W1 = sm + corr::W1, *W2 = sm + corr::W2, *W3 = sm + corr::W3;
  float *b1 = reinterpret_cast<float *>(sm + corr::BIAS), *b2 = b1 + corr::kHid, *b3 = b2 + corr::kHid;
  uint8_t *gbase = sm + corr::GROUPS + wg * corr::kGroupStride;
  uint8_t *XA = gbase + corr::G_XA, *H = gbase + corr::G_H;
  uint64_t *mbar = reinterpret_cast<uint64_t *>(gbase + corr::G_BAR);
  uint64_t *idle = reinterpret_cast<uint64_t *>(gbase + corr::G_IDLE);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + corr::TSLOT);
  const uint32_t limit = cd.wait_limit ? cd.wait_limit : corr::kWaitLimit;
  for (uint32_t q = tid; q < corr::kImage / 16; q += corr::kThreads) reinterpret_cast<uint4 *>(sm)[q] = cd.image[q];
  // hidden-layer biases halved for silu_half (exact: a power-of-two scale)
  for (int q = tid; q < corr::kHid + corr::kHid + corr::kOutP; q += corr::kThreads)
    b1[q] = q < 2 * corr::kHid ? 0.5f * cd.bias[q] : cd.bias[q];
  if (lt == 0) {
    mbar_init(mbar, 1);
    mbar_init(idle, 1);
  }
  if (warp == 0) tmem_alloc(tslot, 128);
  tc05::fence_smem_async();
  tc05::fence_before();
  __syncthreads();
  tc05::fence_after();
  const uint32_t tcol = *tslot + (uint32_t)(wg * 64);
  const uint32_t tl = tcol + ((uint32_t)((warp & 3) * 32) << 16);  // this warp's lane quadrant
  const uint32_t id64 = idesc_bf16(128, 64), id16 = idesc_bf16(128, 16);
  const uint32_t sX = smem_u32(XA), sH = smem_u32(H), sW1 = smem_u32(W1), sW2 = smem_u32(W2), sW3 = smem_u32(W3);
  uint32_t phase = 0;
  bool ok = true;
  bool first = cd.idle_first != 0;
  const int64_t ntiles = (n + corr::kRows - 1) / corr::kRows;
  const int64_t tstride = (int64_t)gridDim.x * corr::kGroups;
  NetRaw raw{};
  net_raw_load<K>(f, ((int64_t)blockIdx.x * corr::kGroups + wg) * corr::kRows + lt, n, raw);
  for (int64_t tile = (int64_t)blockIdx.x * corr::kGroups + wg; tile < ntiles && ok; tile += tstride) {
    const int64_t p = tile * corr::kRows + lt;
    const bool live = p < n;
    bool use = false;
    {
      float x[corr::kInP];
#pragma unroll
      for (int j = 0; j < corr::kInP; ++j) x[j] = 0.f;
      if (live) {
        // the plain interpolation at x_int (particle.cpp:340-360) from the prefetched inputs
        const int ii = ci_(raw.cell) + 1, jj = cj_(raw.cell) + 1, kk = ck_(raw.cell) + 1;
        const float gas[3] = {
            raw.o[0] * f.uf[0][glin3(G, ii + 1, jj, kk)] + (1.f - raw.o[0]) * f.uf[0][glin3(G, ii, jj, kk)],
            raw.o[1] * f.uf[1][glin3(G, ii, jj + 1, kk)] + (1.f - raw.o[1]) * f.uf[1][glin3(G, ii, jj, kk)],
            raw.o[2] * f.uf[2][glin3(G, ii, jj, kk + 1)] + (1.f - raw.o[2]) * f.uf[2][glin3(G, ii, jj, kk)]};
        const float s[3] = {raw.v[0] - gas[0], raw.v[1] - gas[1], raw.v[2] - gas[2]};
        const float smag = sqrtf(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
        float sdrv, dir[3], dmag;
        drive_slip(raw.drive, s, smag, cd.drive_cap, sdrv, dir, dmag);
        const float itth = f.pp[PP_ITTH] ? f.pp[PP_ITTH][p] : c.itth;
        const float itp = f.itp ? f.itp[p] : c.itp;
        const float alpha = f.pp[PP_ALPHA] ? f.pp[PP_ALPHA][p] : c.alpha;
        const float his = f.pp[PP_HEAT_IS] ? f.pp[PP_HEAT_IS][p] : c.is;
        const float dpdx = particle_dp(f, cd, p, itth) * cd.idx;
        const float rep = sdrv * particle_dp(f, cd, p, itth) * cd.inv_nu;
        const float q = alpha * his;
        const float taup = 1.f / itp;
        use = smag > 0.f && dmag > 0.f && dpdx >= cd.lo[0] && dpdx <= cd.hi[0] && rep >= cd.lo[1] &&
              rep <= cd.hi[1] && q >= cd.lo[2] && q <= cd.hi[2] && taup >= cd.lo[3] && taup <= cd.hi[3];
        if (use) {
          const float inv = 1.f / dmag;
          const float fin[10] = {raw.o[0], raw.o[1], raw.o[2], dir[0] * inv, dir[1] * inv, dir[2] * inv, dpdx,
                                 logf(rep), q, logf(taup)};
#pragma unroll
          for (int j = 0; j < 10; ++j) x[j] = (fin[j] - cd.shift[j]) * cd.scale[j];
        }
      }
#pragma unroll
      for (int cb = 0; cb < 2; ++cb) {
        uint4 w;
        w.x = pack_bf16x2(x[cb * 8 + 0], x[cb * 8 + 1]);
        w.y = pack_bf16x2(x[cb * 8 + 2], x[cb * 8 + 3]);
        w.z = pack_bf16x2(x[cb * 8 + 4], x[cb * 8 + 5]);
        w.w = pack_bf16x2(x[cb * 8 + 6], x[cb * 8 + 7]);
        *reinterpret_cast<uint4 *>(XA + tile_off(lt, cb * 8, corr::kInP)) = w;
      }
    }
    group_sync_mma(wg);
    if (lt == 0) {
      mma_bf16(tcol, tile_desc(sX, corr::kInP, 0, 0), tile_desc(sW1, corr::kInP, 0, 0), id64, 0);
      commit(mbar);
    }
    net_raw_load<K>(f, (tile + tstride) * corr::kRows + lt, n, raw);  // the next tile's inputs, in flight
    // (the timeout test polls the idle barrier here, as a completion that never arrives;
    // the MMA's own completion is then drained below before the tensor memory is freed)
    ok = group_wait(wg, first ? idle : mbar, phase, limit);
    first = false;
    if (!ok) break;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      float v[16];
      tmem_ld16(tl + cc * 16, v);
      silu_chunk_to_tile(H, lt, cc * 16, v, b1);
    }
    group_sync_mma(wg);
    if (lt == 0) {  // layer 2 into the same columns (layer 1 has been read)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        mma_bf16(tcol, tile_desc(sH, corr::kHid, 0, ks), tile_desc(sW2, corr::kHid, 0, ks), id64, ks);
      commit(mbar);
    }
    ok = group_wait(wg, mbar, phase, limit);
    if (!ok) break;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {  // layer 2 output overwrites layer 1's in H (its MMA is done)
      float v[16];
      tmem_ld16(tl + cc * 16, v);
      silu_chunk_to_tile(H, lt, cc * 16, v, b2);
    }
    group_sync_mma(wg);
    if (lt == 0) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        mma_bf16(tcol, tile_desc(sH, corr::kHid, 0, ks), tile_desc(sW3, corr::kHid, 0, ks), id16, ks);
      commit(mbar);
    }
    ok = group_wait(wg, mbar, phase, limit);
    if (!ok) break;
    float y[16];
    tmem_ld16(tl, y);
    tc05::fence_before();  // the accumulator reads before the warpgroup's next MMA
    if (live) {
      float yo[4] = {0.f, 0.f, 0.f, 0.f};
      if (use) {
#pragma unroll
        for (int d = 0; d < 4; ++d) yo[d] = y[d] + b3[d];
      }
      f.corr_y[p] = make_uint2(pack_bf16x2(yo[0], yo[1]), pack_bf16x2(yo[2], yo[3]));
    }
  }
  if (!ok) {
    if (lt == 0) atomicOr(err, kErrTimeout);
    tc05::mbar_wait(mbar, phase, corr::kWaitLimit);  // the MMA issued before the wait ran out
  }
  tc05::fence_before();
  __syncthreads();
  tc05::fence_after();
  if (warp == 0) tmem_dealloc(*tslot, 128);
}

// every stage with the correction: the kept network output, applied with this stage's
// drive slip and prior
constexpr int kCorrThreads = 128;  // (256^3 x 2^24, a stage: 256 x 5 an SM 664 us, 128 x 8, 9, 10: 676, 616, 656)
template <int K>
__global__ void __launch_bounds__(kCorrThreads, 9) k_advance32_corr(Geom G, F32Form f, C32 c, int twc, int64_t n,
                                                        int32_t *__restrict__ err, CorrDev cd) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  float mu0 = 0.f, mu1 = 0.f, mu2 = 0.f, mt = 0.f, umax = -INFINITY, gmax = -INFINITY;
  if (p < n) {
    Adv a;
    adv_load<K>(G, f, c, p, a);
    const uint2 yw = f.corr_y[p];
    const float yo[4] = {bf16_lo(yw.x), bf16_hi(yw.x), bf16_lo(yw.y), bf16_hi(yw.y)};
    float ty = 0.f, td = 0.f;
    if (yo[0] != 0.f || yo[1] != 0.f || yo[2] != 0.f || yo[3] != 0.f) {
      const float s[3] = {a.vin[0] - a.gas[0], a.vin[1] - a.gas[1], a.vin[2] - a.gas[2]};
      const float smag = sqrtf(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
      float sdrv, dir[3], dmag;
      const uint2 dw = f.drive[p];
      drive_slip(dw, s, smag, cd.drive_cap, sdrv, dir, dmag);
      const float dp = particle_dp(f, cd, p, a.itth);
      const float prior = prior_of(cd, dp * cd.idx, sdrv * dp * cd.inv_nu);
#pragma unroll
      for (int d = 0; d < 3; ++d) a.gas[d] -= sdrv * prior * yo[d];
      ty = prior * yo[3];
      td = bf16_hi(dw.y);
    }
    const float dv[3] = {a.vin[0] - a.gas[0], a.vin[1] - a.gas[1], a.vin[2] - a.gas[2]};
    const float dt_drive = adv_finish_mlp<K>(G, f, c, twc, p, a, ty, td, err, mu0, mu1, mu2, mt);
    f.drive[p] = make_uint2(pack_bf16x2(dv[0], dv[1]), pack_bf16x2(dv[2], dt_drive));
    umax = a.vac[0];
    gmax = a.gas[0];
  }
  warp_max4(f.slots, mu0, mu1, mu2, mt);
  if (K == 3) warp_max2_signed(f.pslots, umax, gmax);
}

// the prime (grid.cpp:223-226) at the base positions: Tg, RHS_T
__global__ void k_prime32(Geom G, F32Form f, float itth, int64_t n) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  float mt = 0.f;
  if (p < n) {
    const Set32 &B = f.set[SBASE];
    const uint32_t cb = B.cell[p];
    const float o0 = B.o[0][p], o1 = B.o[1][p], o2 = B.o[2][p];
    const int hx = o0 >= 0.5f, hy = o1 >= 0.5f, hz = o2 >= 0.5f;
    const float tx = o0 - hx + 0.5f, ty = o1 - hy + 0.5f, tz = o2 - hz + 0.5f;
    const int ni = ci_(cb) + hx + 1, nj = cj_(cb) + hy + 1, nk = ck_(cb) + hz + 1;
    const float *T = f.tf;
    const float tg = tx * ty * tz * T[glin3(G, ni, nj, nk)] + (1.f - tx) * ty * tz * T[glin3(G, ni - 1, nj, nk)] +
                     tx * (1.f - ty) * tz * T[glin3(G, ni, nj - 1, nk)] + tx * ty * (1.f - tz) * T[glin3(G, ni, nj, nk - 1)] +
                     (1.f - tx) * (1.f - ty) * tz * T[glin3(G, ni - 1, nj - 1, nk)] +
                     (1.f - tx) * ty * (1.f - tz) * T[glin3(G, ni - 1, nj, nk - 1)] +
                     tx * (1.f - ty) * (1.f - tz) * T[glin3(G, ni, nj - 1, nk - 1)] +
                     (1.f - tx) * (1.f - ty) * (1.f - tz) * T[glin3(G, ni - 1, nj - 1, nk - 1)];
    mt = (tg - B.v[3][p]) * (f.pp[PP_ITTH] ? f.pp[PP_ITTH][p] : itth);
    f.rhs_t[p] = mt;
  }
  warp_max4(f.slots, 0.f, 0.f, 0.f, fmaxf(0.f, fabsf(mt)));
}

// q * 2^-se, exact: 2^52 + 2^31 + q from its digits, times 2^-se less the offset in one operation
__device__ __forceinline__ double small_to_f64(int32_t q, int se) {
  const int scale = (1023 - se) << 20;  // 2^-se's high word
  const double x = __hiloint2double(0x43300000, (int)((uint32_t)q ^ 0x80000000u));
  return fma(x, __hiloint2double(scale, 0),
             __hiloint2double((int)((uint32_t)(scale + (52 << 20)) | 0x80000000u), (int)0x80000000u));
}

// exact conversion of a scaled 64-bit integer sum q * 2^-se to fp64 with integer operations
__device__ inline double fixed_to_f64(long long q, int se) {
  if (q == 0) return 0.0;
  if (q == (long long)(int)q) {  // |q| < 2^31: the same steps in 32-bit operations, exact (no rounding)
    const unsigned sgn = q < 0 ? 1u : 0u;
    unsigned m = (unsigned)(sgn ? -q : q);
    const int lz = __clz(m);
    m <<= lz;  // leading one at bit 31: value = (m / 2^31) * 2^(31 - lz - se)
    const int ex = 31 - lz - se + 1023;
    if (ex <= 0) return 0.0;
    return __hiloint2double((int)((sgn << 31) | ((unsigned)ex << 20) | ((m >> 11) & 0xfffffu)), (int)(m << 21));
  }
  unsigned long long sgn = q < 0 ? 1ull : 0ull;
  unsigned long long m = sgn ? (unsigned long long)(-q) : (unsigned long long)q;
  int lz = __clzll(m);
  m <<= lz;  // leading one at bit 63: value = (m / 2^63) * 2^(63 - lz - se)
  long long ex = (long long)(63 - lz - se) + 1023;
  unsigned long long man = (m >> 11) & ((1ull << 52) - 1ull);
  unsigned long long rb = m & 0x7ffull;
  if (rb > 0x400ull || (rb == 0x400ull && (man & 1ull))) {
    man += 1ull;
    if (man == (1ull << 52)) { man = 0; ex += 1; }
  }
  if (ex <= 0) return 0.0;  // below the normal range (not reached for physical scales)
  return __longlong_as_double((long long)((sgn << 63) | ((unsigned long long)ex << 52) | man));
}

// The deposit's work lists: whole bricks in (about) storage order, and the slices of bricks with
// more than kItemMax particles, which come first (no brick holds up the end). A brick whose
// tile in memory holds an earlier population's words is an item with no particles: it then
// writes a tile of zeros, so that the gather reads every tile without asking. keep: no launch has
// written the tiles of C and RHS_Part_Temp since the last lists were made; what they were to clear is
// listed again. (A run without TWC leaves the momentum rows as they are: dep_launch.)
// thin: there are no tiles, so nothing is listed but the slices.
__global__ void __launch_bounds__(256) k_work(const int32_t *__restrict__ cs, Work w, int keep, int thin) {
  __shared__ int32_t warp_n[8], base;
  const int b = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t p0 = 0, p1 = 0;
  bool was = false;
  if (b < w.nb) {
    p0 = cs[(int64_t)b * kBrickCells];
    p1 = cs[((int64_t)b + 1) * kBrickCells];
    const int st = w.dirty[b];
    was = !thin && (st == 2 || (st == 1 && keep));
  }
  const int cnt = p1 - p0;
  const bool sums = !thin && cnt > 0 && cnt <= kItemMax, whole = sums || was;
  if (b < w.nb) w.dirty[b] = sums ? 2 : (was ? 1 : 0);
  const unsigned votes = __ballot_sync(0xffffffffu, whole);
  if (lane == 0) warp_n[wid] = __popc(votes);
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int q = 0; q < 8; ++q) {
      const int v = warp_n[q];
      warp_n[q] = n;
      n += v;
    }
    base = n ? atomicAdd(&w.counts[1], n) : 0;
  }
  __syncthreads();
  if (whole)
    w.items[w.slice_cap + base + warp_n[wid] + __popc(votes & ((1u << lane) - 1u))] =
        make_int4(b, p0, sums ? p1 : p0, 0);
  if (cnt > kItemMax) {
    const int c = (cnt + kItemMax - 1) / kItemMax;  // at most 2 cnt / kItemMax: slice_cap bounds their sum
    const int at = atomicAdd(&w.counts[0], c);
    for (int q = 0; q < c; ++q)
      w.items[at + q] = make_int4(b, p0 + (int)((int64_t)cnt * q / c), p0 + (int)((int64_t)cnt * (q + 1) / c), 1);
  }
}

// v into the exact 64-bit sum of field fld (0 C, 1-3 RHS_RU, 4 RHS_Part_Temp) at cell (x, y, z),
// taken periodically
__device__ __noinline__ void extra_add(const Geom &G, const Work &w, int32_t epoch, int fld, int x, int y, int z,
                                       long long v) {
  const uint32_t id = brick_id(G, wrapi(x, G.n[0]), wrapi(y, G.n[1]), wrapi(z, G.n[2]));
  atomicAdd((unsigned long long *)&w.extra[fld * w.ncell + id], (unsigned long long)v);
  w.extra_epoch[id / kBrickCells] = epoch;  // every writer of a launch writes the same value
}

// cell c relative to b, of its periodic copies the one in [-1, 8] where there is one
__device__ __forceinline__ int rel_tile(int c, int b, int n) {
  int r = c - b;
  r += r < -1 ? n : 0;
  r -= r > kBr ? n : 0;
  return r;
}

// Exact sums. Every contribution is scaled so that the largest magnitude is 2^24 (the fp32 values
// carry 24 significant bits, so nothing beyond their own rounding is lost) and rounded to an
// integer v. A tile's word is their sum modulo 2^32; an add whose signed result overflows shows in
// the returned old value (the sign bit of the result's carry-out test below) and puts +-2^32
// into the cell's 64-bit sum, so word + extra is the exact sum whatever the order of the adds.
__device__ __forceinline__ uint32_t add_word(uint32_t *a, int32_t v) {
  const uint32_t old = atomicAdd(a, (uint32_t)v), sum = old + (uint32_t)v;
  return (old ^ sum) & ((uint32_t)v ^ sum);  // top bit: overflow
}

// trilinear deposit (particle.cpp:526-559, :586-658) of a particle with in-cell offsets o3 and
// value val (already times the field's fixed-point scale) on the 8 cells around its round()
// node; acc: the tile word of the node's cell minus one in every dimension
template <typename Over>
__device__ __forceinline__ void deposit_trilinear(uint32_t *acc, const float o3[3], float val, Over over) {
  float w[3][2];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float xl = o3[d] - (o3[d] >= 0.5f ? 1.f : 0.f) + 0.5f;
    w[d][0] = 1.f - xl;  // cell node - 1
    w[d][1] = xl;        // cell node
  }
  int32_t v[8];
  uint32_t ov[8];
#pragma unroll
  for (int oz = 0; oz < 2; ++oz)
#pragma unroll
    for (int oy = 0; oy < 2; ++oy) {
      const float wyz = w[2][oz] * w[1][oy] * val;
#pragma unroll
      for (int ox = 0; ox < 2; ++ox) {
        const int q = (oz * 2 + oy) * 2 + ox;
        v[q] = __float2int_rn(w[0][ox] * wyz);
        ov[q] = add_word(acc + (oz * kTE + oy) * kRowWords + ox, v[q]);
      }
    }
  const uint32_t any = (ov[0] | ov[1] | ov[2]) | (ov[3] | ov[4] | ov[5]) | (ov[6] | ov[7]);
  if ((int32_t)any < 0) {
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if ((int32_t)ov[q] < 0) over(q & 1, (q >> 1) & 1, q >> 2, v[q] > 0 ? 1ll << 32 : -(1ll << 32));
  }
}

// the same, for a particle that reaches past its brick's tile: every contribution straight into the
// 64-bit sums (node: the round() node's cell)
__device__ __noinline__ void deposit_trilinear_far(const Geom &G, const Work &w, int32_t epoch, int fld, int nx, int ny,
                                                   int nz, float o0, float o1, float o2, float val) {
  const float o3[3] = {o0, o1, o2};
  float wt[3][2];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float xl = o3[d] - (o3[d] >= 0.5f ? 1.f : 0.f) + 0.5f;
    wt[d][0] = 1.f - xl;
    wt[d][1] = xl;
  }
  for (int q = 0; q < 8; ++q) {
    const int ox = q & 1, oy = (q >> 1) & 1, oz = q >> 2;
    const float wyz = wt[2][oz] * wt[1][oy] * val;
    const int32_t v = __float2int_rn(wt[0][ox] * wyz);
    if (v) extra_add(G, w, epoch, fld, nx - 1 + ox, ny - 1 + oy, nz - 1 + oz, v);
  }
}

// warp sum of an int64 with 32-bit warp reductions: three pieces of the two's-complement value (bits
// 0-20 and 21-41 unsigned, 42-63 signed), whose 32-lane sums cannot overflow, recombined exactly
__device__ __forceinline__ long long warp_sum_i64(long long v) {
  const unsigned lo = (unsigned)(v & 0x1fffffll), mid = (unsigned)((v >> 21) & 0x1fffffll);
  const int hi = (int)(v >> 42);
  const unsigned slo = __reduce_add_sync(0xffffffffu, lo), smid = __reduce_add_sync(0xffffffffu, mid);
  const int shi = __reduce_add_sync(0xffffffffu, hi);
  return (long long)shi * (1ll << 42) + (long long)smid * (1ll << 21) + (long long)slo;
}

// Thin populations have no tiles: a particle's contributions go straight to a word per cell and field
// (Work::mid as [5][cells in brick order]), with the tiles' own handling of overflows. A cell's place
// is a sum over the dimensions. at[d][.], brick[d][.]: that of the particle's cell less one, its cell and
// its cell plus one (periodic), and of their bricks.
struct Places {
  uint32_t at[3][3], brick[3][3];
};
__device__ __forceinline__ Places places_of(const Geom &G, uint32_t cell) {
  const int c[3] = {ci_(cell), cj_(cell), ck_(cell)};
  const uint32_t across[3] = {1u, (uint32_t)(G.n[0] / kBr), (uint32_t)(G.n[0] / kBr) * (uint32_t)(G.n[1] / kBr)};
  Places r;
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int q = s == 0 ? (c[d] == 0 ? G.n[d] - 1 : c[d] - 1) : (s == 1 ? c[d] : (c[d] == G.n[d] - 1 ? 0 : c[d] + 1));
      r.brick[d][s] = (uint32_t)(q / kBr) * across[d];
      r.at[d][s] = r.brick[d][s] * kBrickCells + ((uint32_t)(q % kBr) << (3 * d));
    }
  return r;
}
__device__ __forceinline__ void mark_bricks(const Work &w, int32_t epoch, const Places &r) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int x = q & 1 ? 2 : 0, y = q & 2 ? 2 : 0, z = q & 4 ? 2 : 0;
    if ((!x || r.brick[0][2] != r.brick[0][0]) && (!y || r.brick[1][2] != r.brick[1][0]) &&
        (!z || r.brick[2][2] != r.brick[2][0]))
      w.word_epoch[r.brick[0][x] + r.brick[1][y] + r.brick[2][z]] = epoch;
  }
}
__device__ __noinline__ void word_overflow(const Work &w, int32_t epoch, int64_t at, uint32_t brick, int32_t v) {
  atomicAdd((unsigned long long *)&w.extra[at], v > 0 ? 1ull << 32 : (unsigned long long)-(1ll << 32));
  w.extra_epoch[brick] = epoch;
}
// contributions v[0 .. N) of field fld at the cells id[.]
template <int N>
__device__ __forceinline__ void add_words(const Work &w, int32_t epoch, int fld, const uint32_t (&id)[N], const int32_t (&v)[N]) {
  uint32_t *words = w.mid + fld * w.ncell, over[N], any = 0u;
#pragma unroll
  for (int q = 0; q < N; ++q) over[q] = v[q] ? add_word(words + id[q], v[q]) : 0u;
#pragma unroll
  for (int q = 0; q < N; ++q) any |= over[q];
  if ((int32_t)any < 0) {
#pragma unroll
    for (int q = 0; q < N; ++q)
      if ((int32_t)over[q] < 0) word_overflow(w, epoch, fld * w.ncell + id[q], id[q] / kBrickCells, v[q]);
  }
}
__device__ __forceinline__ void add_trilinear(const Work &w, int32_t epoch, int fld, const Places &r, const float o3[3],
                                              float val) {
  float wt[3][2];
  bool h[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    h[d] = o3[d] >= 0.5f;
    const float xl = o3[d] - (o3[d] >= 0.5f ? 1.f : 0.f) + 0.5f;
    wt[d][0] = 1.f - xl;
    wt[d][1] = xl;
  }
  uint32_t id[8];
  int32_t v[8];
#pragma unroll
  for (int oz = 0; oz < 2; ++oz)
#pragma unroll
    for (int oy = 0; oy < 2; ++oy) {
      const float wyz = wt[2][oz] * wt[1][oy] * val;
      const uint32_t yz = (h[1] ? r.at[1][oy + 1] : r.at[1][oy]) + (h[2] ? r.at[2][oz + 1] : r.at[2][oz]);
#pragma unroll
      for (int ox = 0; ox < 2; ++ox) {
        id[(oz * 2 + oy) * 2 + ox] = yz + (h[0] ? r.at[0][ox + 1] : r.at[0][ox]);
        v[(oz * 2 + oy) * 2 + ox] = __float2int_rn(wt[0][ox] * wyz);
      }
    }
  add_words(w, epoch, fld, id, v);
}

constexpr int kDepThreads = 256;

// The deposit, first half. One CTA per item (a brick, or a slice of a crowded one): the item's
// particles, which the step's sort left together, add
//   FIELDS >= 1: the concentration, FIELDS == 2: also the face momentum, at the *_int position,
//   RHS_T at the *_new position
// into the brick's tile in shared memory, which then goes to memory as it is; k_dep_gather sums
// the tiles that reach a cell. Particles move less than a cell from the brick between sorts and
// the tile reaches one cell past it: a position more than half a cell outside the brick goes into
// the 64-bit sums instead (as does everything of a slice, word by word).
//
// THIN: the particles of all bricks but the sliced ones by themselves, a thread each, into a word per
// cell and field (add_words).
//
// Every particle is visited once. (Before, a CTA owned 16^3 cells and visited the particles of all
// cells that could reach them, two cells around: 1.95 visits a particle, each with a test per
// target, and two 32-bit adds per contribution so that sums of any size fitted: 840 warp
// instructions a visit.) Bound: the shared-memory adds (22 a particle) and instruction issue;
// four CTAs per SM let one's flush overlap the others' particles, and the 25 KB tile leaves them
// an L1 (with blocks of 32 x 8 x 8 cells, 71 KB, it ran half as fast). 512^3 cells x 2^27 particles,
// half of them in 64 blobs: 3.8 ms, and 3.0 ms for the gather, against 10.4 ms; 256^3 x 2^24: 0.51 +
// 0.33 against 1.57 ms.
template <int FIELDS, bool THIN>
__global__ void __launch_bounds__(kDepThreads, 4)
    k_dep_tile(Geom G, F32Form f, Set32 SI, Set32 SN, int32_t epoch, int64_t n) {
  constexpr int ROWS = FIELDS == 0 ? kRowsTri : (FIELDS == 1 ? 2 * kRowsTri : kRows);
  constexpr int WORDS = ROWS * kRowWords + 4;
  __shared__ __align__(16) uint32_t acc[WORDS];
  __shared__ int4 next_item;
  const Work &w = f.work;
  const int32_t n_slices = w.counts[0], n_items = n_slices + w.counts[1];
  // Every CTA works out the fields' scales from the stage's partial maxima (16 KB of L2 reads a CTA; a
  // launch of their own cost 5 us with its gap), the first one leaves them to the gather and
  // readies the statistics. The gather clears the maxima and the item counter.
  __shared__ uint32_t part[4][kDepThreads / 32];
  __shared__ int exponent[5];
  {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t m[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int q = 0; q < kBoundSlots / kDepThreads; ++q) {
      const uint4 v = reinterpret_cast<const uint4 *>(f.slots)[q * kDepThreads + threadIdx.x];
      m[0] = max(m[0], v.x);
      m[1] = max(m[1], v.y);
      m[2] = max(m[2], v.z);
      m[3] = max(m[3], v.w);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = __reduce_max_sync(0xffffffffu, m[q]);
    if (lane < 4) part[lane][wid] = lane == 0 ? m[0] : (lane == 1 ? m[1] : (lane == 2 ? m[2] : m[3]));
    __syncthreads();
    if (threadIdx.x < 5) {
      // largest contribution of each field: concentration weights <= 1, momentum |RHS_u|,
      // energy |RHS_T| (weights <= 1); its magnitude maps to at most 2^24
      uint32_t top = 0u;
      if (threadIdx.x)
        for (int q = 0; q < kDepThreads / 32; ++q) top = max(top, part[threadIdx.x - 1][q]);
      const float b = threadIdx.x ? __uint_as_float(top) : 1.f;
      int e = 0;
      if (b > 0.f && isfinite(b)) frexpf(b, &e);  // b < 2^e
      const int se = 24 - e > 100 ? 100 : 24 - e;
      exponent[threadIdx.x] = se;
      if (blockIdx.x == 0) f.se[threadIdx.x] = se;
    }
    if (blockIdx.x == 0 && threadIdx.x < 15 && (FIELDS || threadIdx.x % 5 == 4))
      f.totals[threadIdx.x] =
          threadIdx.x < 5 ? 0ull : (threadIdx.x < 10 ? (unsigned long long)LLONG_MIN : (unsigned long long)LLONG_MAX);
    __syncthreads();
  }
  float scale[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) scale[q] = ldexpf(1.0f, exponent[q]);  // exact powers of two
  if (THIN) {
    for (int64_t p = (int64_t)blockIdx.x * kDepThreads + threadIdx.x; p < n; p += (int64_t)gridDim.x * kDepThreads) {
      const uint32_t cb = f.set[SBASE].cell[p], cn = SN.cell[p];
      uint32_t ci = 0;
      float oi[3] = {0.f, 0.f, 0.f}, on[3], ru[3] = {0.f, 0.f, 0.f};
      if (FIELDS) ci = SI.cell[p];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        on[d] = SN.o[d][p];
        if (FIELDS) oi[d] = SI.o[d][p];
        if (FIELDS == 2) ru[d] = f.rhs_u[d][p];
      }
      const float rt = f.rhs_t[p];
      const int32_t *first = f.cell_start + (brick_id(G, ci_(cb), cj_(cb), ck_(cb)) & ~(uint32_t)(kBrickCells - 1));
      if (first[kBrickCells] - first[0] > kItemMax) continue;  // in a slice
      if (FIELDS) {
        const Places r = places_of(G, ci);
        mark_bricks(w, epoch, r);
        add_trilinear(w, epoch, 0, r, oi, scale[0]);
        if (FIELDS == 2) {
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const float u = ru[d] * scale[1 + d];
            const uint32_t across = d == 0 ? r.at[1][1] + r.at[2][1] : (d == 1 ? r.at[0][1] + r.at[2][1] : r.at[0][1] + r.at[1][1]);
            const uint32_t id[2] = {across + r.at[d][1], across + r.at[d][2]};
            const int32_t v[2] = {__float2int_rn((1.f - oi[d]) * u), __float2int_rn(oi[d] * u)};
            add_words(w, epoch, 1 + d, id, v);
          }
        }
      }
      const Places r = places_of(G, cn);
      mark_bricks(w, epoch, r);
      add_trilinear(w, epoch, 4, r, on, rt * scale[4]);
    }
  }
  auto fetch = [&](int idx) {
    return idx >= n_items ? make_int4(-1, 0, 0, 0)
                          : (idx < n_slices ? w.items[idx] : w.items[w.slice_cap + idx - n_slices]);
  };
  for (int q = threadIdx.x; q < WORDS / 4; q += kDepThreads)
    reinterpret_cast<uint4 *>(acc)[q] = make_uint4(0u, 0u, 0u, 0u);
  if (threadIdx.x == 0) next_item = fetch(atomicAdd(&w.counts[2], 1));
  __syncthreads();
  while (true) {
    const int4 item = next_item;
    if (item.x < 0) break;
    int idx = 0;
    if (threadIdx.x == 0) idx = atomicAdd(&w.counts[2], 1);  // the next item, while this one runs
    const int nbx = G.n[0] / kBr, nby = G.n[1] / kBr;
    const int tx = item.x % nbx, row0 = item.x / nbx;  // brick row (z, y)
    const int bx = tx * kBr, by = (row0 % nby) * kBr, bz = (row0 / nby) * kBr;
    // Lane groups of 8 walk their own sub-range, 8 consecutive particles per pass (one aligned
    // 32-byte sector of each 4-byte array), and the 4 groups of a warp take sub-ranges a quarter
    // of the item apart: the lanes of a warp in a crowded cell would otherwise all add to the
    // same words.
    const int len = item.z - item.y;
    const int grp = (int)(threadIdx.x >> 5) + (kDepThreads / 32) * (int)((threadIdx.x >> 3) & 3);
    const int g0 = grp ? (item.y + len * grp / (kDepThreads / 8)) & ~7 : item.y & ~7;
    const int g1 = grp == kDepThreads / 8 - 1 ? item.z : (item.y + len * (grp + 1) / (kDepThreads / 8)) & ~7;
    for (int p = g0 + (int)(threadIdx.x & 7); p < g1; p += 8) {
      if (p < item.y) continue;
      // all loads first: one memory round trip per particle
      uint32_t ci = 0;
      float oi[3] = {0.f, 0.f, 0.f}, on[3], ru[3] = {0.f, 0.f, 0.f};
      if (FIELDS) {
        ci = SI.cell[p];
#pragma unroll
        for (int d = 0; d < 3; ++d) oi[d] = SI.o[d][p];
        if (FIELDS == 2) {
#pragma unroll
          for (int d = 0; d < 3; ++d) ru[d] = f.rhs_u[d][p];
        }
      }
      const uint32_t cn = SN.cell[p];
#pragma unroll
      for (int d = 0; d < 3; ++d) on[d] = SN.o[d][p];
      const float rt = f.rhs_t[p];
      if (FIELDS) {
        const int r0 = rel_tile(ci_(ci), bx, G.n[0]), r1 = rel_tile(cj_(ci), by, G.n[1]),
                  r2 = rel_tile(ck_(ci), bz, G.n[2]);
        const int n0 = r0 + (oi[0] >= 0.5f), n1 = r1 + (oi[1] >= 0.5f), n2 = r2 + (oi[2] >= 0.5f);
        // nodes 0 .. 8: the targets node - 1 and node and the cell's faces lie in the tile
        if ((unsigned)n0 <= (unsigned)kBr && (unsigned)n1 <= (unsigned)kBr && (unsigned)n2 <= (unsigned)kBr) {
          deposit_trilinear(acc + (kRowC + n2 * kTE + n1) * kRowWords + 3 + n0, oi, scale[0],
                            [&](int x, int y, int z, long long v) {
                              extra_add(G, w, epoch, 0, bx + n0 - 1 + x, by + n1 - 1 + y, bz + n2 - 1 + z, v);
                            });
          if (FIELDS == 2) {
            // face-normal deposits (particle.cpp:498-524): along d, face r[d] gets (1 - x_l) R_d
            // and face r[d] + 1 gets x_l R_d, at the particle's cell across
            uint32_t *fx = acc + (kRowX + (r2 + 1) * kTE + r1 + 1) * kRowWords + 4 + r0;
            uint32_t *fy = acc + (kRowY + (r2 + 1) * (kTE + 1) + r1 + 1) * kRowWords + 4 + r0;
            uint32_t *fz = acc + (kRowZ + (r2 + 1) * kTE + r1 + 1) * kRowWords + 4 + r0;
            int32_t v[6];
            uint32_t ov[6];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const float r = ru[d] * scale[1 + d];
              v[2 * d] = __float2int_rn((1.f - oi[d]) * r);
              v[2 * d + 1] = __float2int_rn(oi[d] * r);
            }
            ov[0] = add_word(fx, v[0]);
            ov[1] = add_word(fx + 1, v[1]);
            ov[2] = add_word(fy, v[2]);
            ov[3] = add_word(fy + kRowWords, v[3]);
            ov[4] = add_word(fz, v[4]);
            ov[5] = add_word(fz + kTE * kRowWords, v[5]);
            if ((int32_t)((ov[0] | ov[1] | ov[2]) | (ov[3] | ov[4] | ov[5])) < 0) {
#pragma unroll
              for (int q = 0; q < 6; ++q)
                if ((int32_t)ov[q] < 0)
                  extra_add(G, w, epoch, 1 + q / 2, bx + r0 + (q == 1), by + r1 + (q == 3), bz + r2 + (q == 5),
                            v[q] > 0 ? 1ll << 32 : -(1ll << 32));
            }
          }
        } else {
          deposit_trilinear_far(G, w, epoch, 0, bx + n0, by + n1, bz + n2, oi[0], oi[1], oi[2], scale[0]);
          if (FIELDS == 2) {
#pragma unroll 1
            for (int d = 0; d < 3; ++d) {
              const float r = ru[d] * scale[1 + d];
              const int32_t v0 = __float2int_rn((1.f - oi[d]) * r), v1 = __float2int_rn(oi[d] * r);
              if (v0) extra_add(G, w, epoch, 1 + d, bx + r0, by + r1, bz + r2, v0);
              if (v1) extra_add(G, w, epoch, 1 + d, bx + r0 + (d == 0), by + r1 + (d == 1), bz + r2 + (d == 2), v1);
            }
          }
        }
      }
      {
        const int n0 = rel_tile(ci_(cn), bx, G.n[0]) + (on[0] >= 0.5f),
                  n1 = rel_tile(cj_(cn), by, G.n[1]) + (on[1] >= 0.5f),
                  n2 = rel_tile(ck_(cn), bz, G.n[2]) + (on[2] >= 0.5f);
        if ((unsigned)n0 <= (unsigned)kBr && (unsigned)n1 <= (unsigned)kBr && (unsigned)n2 <= (unsigned)kBr)
          deposit_trilinear(acc + (n2 * kTE + n1) * kRowWords + 3 + n0, on, rt * scale[4],
                            [&](int x, int y, int z, long long v) {
                              extra_add(G, w, epoch, 4, bx + n0 - 1 + x, by + n1 - 1 + y, bz + n2 - 1 + z, v);
                            });
        else
          deposit_trilinear_far(G, w, epoch, 4, bx + n0, by + n1, bz + n2, on[0], on[1], on[2], rt * scale[4]);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) next_item = fetch(idx);  // (the running item's was read before the barrier)
    if (!item.w) {
      uint32_t *mid = w.mid + (int64_t)row0 * kRows * G.n[0] + bx;
      for (int q = threadIdx.x; q < 2 * ROWS; q += kDepThreads) {
        const int row = q >> 1, half = q & 1;
        uint4 *t = reinterpret_cast<uint4 *>(acc + row * kRowWords + 4 + 4 * half);
        *reinterpret_cast<uint4 *>(mid + row * G.n[0] + 4 * half) = *t;
        *t = make_uint4(0u, 0u, 0u, 0u);
      }
      uint32_t *side = w.side + (int64_t)item.x * kSideWords;
      for (int row = threadIdx.x; row < ROWS; row += kDepThreads) {
        uint32_t *t = acc + row * kRowWords;
        side[row] = t[3];
        side[kRows + row] = t[kRowWords];
        t[3] = 0u;
        t[kRowWords] = 0u;
      }
      if (FIELDS == 2) {
        for (int row = threadIdx.x; row < kRowsTri; row += kDepThreads) {
          uint32_t *t = acc + (kRowX + row) * kRowWords + kRowWords + 1;
          side[2 * kRows + row] = *t;
          *t = 0u;
        }
      }
    } else {
      for (int q = threadIdx.x; q < WORDS; q += kDepThreads) {
        const int32_t v = (int32_t)acc[q];
        acc[q] = 0u;
        if (!v) continue;
        int row = q / kRowWords, x = q % kRowWords - 4;
        if (x < -1) {  // x = 8 and 9 of the row before
          x += kRowWords;
          row -= 1;
        }
        int fld = 4, ey = kTE;
        if (row >= kRowZ) { fld = 3; row -= kRowZ; }
        else if (row >= kRowY) { fld = 2; row -= kRowY; ey = kTE + 1; }
        else if (row >= kRowX) { fld = 1; row -= kRowX; }
        else if (row >= kRowC) { fld = 0; row -= kRowC; }
        extra_add(G, w, epoch, fld, bx + x, by - 1 + row % ey, bz - 1 + row / ey, v);
      }
    }
    __syncthreads();
  }
}

// The deposit, second half: every cell's exact sums from the tiles that reach it -- its own brick's
// and, on a brick's boundary layers, its neighbours' -- and the 64-bit extras where the brick
// has any this launch, converted to fp64 and written to the cell and its periodic ghost images.
// THIN: the cell's own word instead of the tiles.
// A block takes one field (blockIdx.y: RHS_Part_Temp, C, RHS_RU x, y, z; the ones from `sums` on are
// zero, RHS_RU without TWC, grid.cpp:671); a warp takes 32 cells along x of a layer's eight rows in
// a brick row: of every tile that reaches them ten rows (eleven of RHS_RU y) lie one behind the other, so
// their words are in flight together, as 128-byte lines, and the x neighbours' words from the end lanes of
// each brick. The launch's exact field statistics are gathered on the way; the last block to finish
// turns them into the balance sums (momentum components, interior mean of RHS_Part_Temp,
// grid.cpp:541) and, with EXT, the fields' maxima and minima. Bound: latency of the loads and memory
// (12 GB at 512^3). A warp with one row of all fields at a time had ten words in flight and decided
// about the neighbours row by row: 512^3 4.2 ms (6.1 with the extremes), 256^3 0.47 (0.70); this
// way 3.0 and 0.33, with or without.
template <bool EXT, bool THIN>
__global__ void __launch_bounds__(256, 4) k_dep_gather(Geom G, F32Form f, int32_t epoch, int sums, double inv_cells,
                                                       double *__restrict__ outC, double *__restrict__ outX,
                                                       double *__restrict__ outY, double *__restrict__ outZ,
                                                       double *__restrict__ outE, double *__restrict__ mom,
                                                       double *__restrict__ emean) {
  const Work &w = f.work;
  const int fq = blockIdx.y, fld = fq == 0 ? 4 : fq - 1;
  double *__restrict__ out = fq == 0 ? outE : (fq == 1 ? outC : (fq == 2 ? outX : (fq == 3 ? outY : outZ)));
  const int nbx = G.n[0] / kBr, nby = G.n[1] / kBr, nbz = G.n[2] / kBr;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n0 = G.n[0], nx = (n0 + 31) / 32;
  // the running sum, maximum and minimum; the extremes in 32 bits (INT_MIN, INT_MAX: none yet) while
  // a warp's sums are inside them, else in shared memory
  __shared__ long long wide[2];
  long long tot = 0;
  int32_t vmax = INT_MIN, vmin = INT_MAX;
  if (EXT) {
    if (threadIdx.x == 0) {
      wide[0] = LLONG_MIN;
      wide[1] = LLONG_MAX;
    }
    __syncthreads();
  }
  if (blockIdx.x == 0 && fq == 0) {  // ready for the next stage's maxima and the next launch's items
    for (int q = threadIdx.x; q < kBoundSlots; q += blockDim.x) reinterpret_cast<uint4 *>(f.slots)[q] = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x == 0) w.counts[2] = 0;
  }
  if (fq >= sums) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < G.gsize; t += (int64_t)gridDim.x * blockDim.x)
      out[t] = 0.0;
  } else {
    const int se = f.se[fld];
    const int first = fq < 2 ? fq * kRowC : (fq == 2 ? kRowX : (fq == 3 ? kRowY : kRowZ));
    const int layer_rows = fq == 3 ? kTE + 1 : kTE;
    const int32_t *__restrict__ mid = reinterpret_cast<const int32_t *>(w.mid);
    const int32_t *__restrict__ side = reinterpret_cast<const int32_t *>(w.side);
    const int tasks = nx * nby * nbz;
    for (int task = blockIdx.x; task < tasks; task += gridDim.x) {
      const int xb = task % nx, row = task / nx, by = row % nby, bz = row / nby;
      const int lz = (wid + task) % kBr;  // (the layers turn over the warps: the outer ones take longer)
      const bool live = xb * 32 + lane < n0;
      const int i = live ? xb * 32 + lane : n0 - 1;
      const int bx = i / kBr, lx = i % kBr;
      // Besides the cell's own brick, in each dimension, the neighbour whose tile reaches it: cell 0
      // takes the lower brick's coordinate 8, cell 1 its 9 (the faces along that dimension alone),
      // cell 7 the upper brick's -1. Along x: words of the side array
      const bool end = lx == 0 || lx == kBr - 1 || (lx == 1 && fq == 2);
      const int ox = lx <= 1 ? (bx == 0 ? nbx - 1 : bx - 1) : (bx == nbx - 1 ? 0 : bx + 1);
      const int at = lx == 0 ? kRows : (lx == 1 ? 2 * kRows - kRowX : 0);
      const int yl = by == 0 ? nby - 1 : by - 1, yh = by == nby - 1 ? 0 : by + 1;
      long long v[kBr];
#pragma unroll
      for (int r = 0; r < kBr; ++r) v[r] = 0;
      // adds layer cz (z + 1) of the tiles of brick row (., tz) and its y neighbours
      auto layer = [&](int tz, int cz) {
        const int at_row = first + cz * layer_rows;
        auto words = [&](int ty, int cy, const int32_t *&m, const int32_t *&sd) {
          const int64_t brow = (int64_t)tz * nby + ty;
          m = mid + (brow * kRows + at_row + cy) * n0 + i;
          sd = side + (brow * nbx + ox) * kSideWords + at + at_row + cy;
        };
        const int32_t *m, *sd, *ml, *sl, *mh, *sh;
        words(by, 1, m, sd);
        words(yl, kBr + 1, ml, sl);
        words(yh, 0, mh, sh);
        // of each row a word, and the end lanes' side word: the eight rows, y = 8 and 9 of the lower
        // brick's tile, y = -1 of the upper's
        constexpr int R = kBr + 3;
        int32_t p[R], q[R];
#pragma unroll
        for (int r = 0; r < kBr; ++r) p[r] = m[(int64_t)r * n0];
        p[kBr] = ml[0];
        p[kBr + 1] = fq == 3 ? ml[n0] : 0;
        p[kBr + 2] = mh[0];
#pragma unroll
        for (int r = 0; r < R; ++r) q[r] = 0;
        if (end) {
#pragma unroll
          for (int r = 0; r < kBr; ++r) q[r] = sd[r];
          q[kBr] = sl[0];
          if (fq == 3) q[kBr + 1] = sl[1];
          q[kBr + 2] = sh[0];
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
          v[r < kBr ? r : (r == kBr + 2 ? kBr - 1 : r - kBr)] += (long long)p[r] + (long long)q[r];
      };
      const int own = (bz * nby + by) * nbx + bx;
      if (!THIN) {
        layer(bz, lz + 1);
        if (lz == 0 || (lz == 1 && fq == 4)) layer(bz == 0 ? nbz - 1 : bz - 1, kBr + 1 + lz);
        if (lz == kBr - 1) layer(bz == nbz - 1 ? 0 : bz + 1, 0);
      } else if (live && w.word_epoch[own] == epoch) {
        uint32_t *x = w.mid + fld * w.ncell + (int64_t)own * kBrickCells + lz * kBr * kBr + lx;
        int32_t e[kBr];
#pragma unroll
        for (int r = 0; r < kBr; ++r) e[r] = (int32_t)x[r * kBr];
#pragma unroll
        for (int r = 0; r < kBr; ++r) {
          v[r] = e[r];
          if (e[r]) x[r * kBr] = 0u;  // ready for the next launch
        }
      }
      if (live && w.extra_epoch[own] == epoch) {
        long long *x = w.extra + fld * w.ncell + (int64_t)own * kBrickCells + lz * kBr * kBr + lx;
        long long e[kBr];
#pragma unroll
        for (int r = 0; r < kBr; ++r) e[r] = x[r * kBr];
#pragma unroll
        for (int r = 0; r < kBr; ++r) {
          v[r] += e[r];
          if (e[r]) x[r * kBr] = 0;  // ready for the next launch
        }
      }
      if (!live) continue;
      // the cell and its periodic images: along x the end cells of a row have one, along y and z whole
      // rows do
      const int j = by * kBr, k = bz * kBr + lz;
      double *to = out + glin3(G, i + 1, j + 1, k + 1);
      const int img_x = i == 0 ? n0 : (i == n0 - 1 ? -n0 : 0);
      const long long plane = (long long)G.g[0] * G.g[1],
                      img_z = k == 0 ? G.n[2] * plane : (k == G.n[2] - 1 ? -G.n[2] * plane : 0);
      auto put = [&](int r, double o) {
        double *c = to + (long long)r * G.g[0];
        auto along_x = [&](double *a) {
          *a = o;
          if (img_x) a[img_x] = o;
        };
        along_x(c);
        if (img_z) along_x(c + img_z);
        if (j + r == 0 || j + r == G.n[1] - 1) {
          double *y = c + (j + r == 0 ? G.n[1] : -G.n[1]) * (long long)G.g[0];
          along_x(y);
          if (img_z) along_x(y + img_z);
        }
        tot += v[r];
      };
      bool small = true;
#pragma unroll
      for (int r = 0; r < kBr; ++r) small &= v[r] == (long long)(int)v[r] && (!EXT || (v[r] != INT_MIN && v[r] != INT_MAX));
      if (small) {
#pragma unroll
        for (int r = 0; r < kBr; ++r) {
          put(r, small_to_f64((int)v[r], se));
          if (EXT) {
            vmax = max(vmax, (int)v[r]);
            vmin = min(vmin, (int)v[r]);
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < kBr; ++r) {
          put(r, fixed_to_f64(v[r], se));
          if (EXT) {
            atomicMax(&wide[0], v[r]);
            atomicMin(&wide[1], v[r]);
          }
        }
      }
    }
  }
  __shared__ long long red[8][3];
  __shared__ int last;
  const long long sm = warp_sum_i64(tot);
  const int32_t mx = __reduce_max_sync(0xffffffffu, vmax), mn = __reduce_min_sync(0xffffffffu, vmin);
  if (lane == 0) {
    red[wid][0] = sm;
    red[wid][1] = mx;
    red[wid][2] = mn;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long all = 0, high = fq < sums ? LLONG_MIN : 0, low = fq < sums ? LLONG_MAX : 0;
    for (int u = 0; u < 8; ++u) {
      all += red[u][0];
      if (EXT) {
        if (red[u][1] > (long long)INT_MIN) high = max(high, red[u][1]);
        if (red[u][2] < (long long)INT_MAX) low = min(low, red[u][2]);
      }
    }
    if (all) atomicAdd(&f.totals[fld], (unsigned long long)all);
    if (EXT) {
      if (fq < sums) {
        high = max(high, wide[0]);
        low = min(low, wide[1]);
      }
      atomicMax(reinterpret_cast<long long *>(&f.totals[5 + fld]), high);
      atomicMin(reinterpret_cast<long long *>(&f.totals[10 + fld]), low);
    }
    __threadfence();
    last = atomicAdd(f.done, 1) == (int)(gridDim.x * gridDim.y) - 1;
  }
  __syncthreads();
  if (!last) return;
  if (threadIdx.x == 0) *f.done = 0;
  __threadfence();
  if (threadIdx.x < gridDim.y) {
    const int fld = threadIdx.x == 0 ? 4 : threadIdx.x - 1, e = f.se[fld];
    const long long sm = (long long)__ldcg(&f.totals[fld]);
    if (EXT) {  // integer order is the fp64 order at one scale
      f.fstat[3 * fld + 0] = fixed_to_f64((long long)__ldcg(&f.totals[5 + fld]), e);
      f.fstat[3 * fld + 1] = fixed_to_f64((long long)__ldcg(&f.totals[10 + fld]), e);
    }
    const double sum = fixed_to_f64(sm, e);
    f.fstat[3 * fld + 2] = sum;
    if (fld >= 1 && fld <= 3) mom[fld - 1] = sum;
    if (fld == 4) *emean = sum * inv_cells;
  }
}

// fp32 <-> fp64 conversions in integer operations, the values the hardware conversions give:
// GB300 converts between the two at its FP64 rate (two lanes per SM and clock), which bounded
// every kernel that hands particles or fields across (2^27 particles down: 10.9 ms, 1.1 TB/s).
// Zeros, subnormals, infinities and NaNs (and results outside the normal fp32 range) take the
// hardware conversion.
__device__ __forceinline__ double widen(float v) {
  const uint32_t u = __float_as_uint(v), a = u & 0x7fffffffu;
  if (a - 0x00800000u >= 0x7f000000u) return (double)v;  // not a normal number
  return __hiloint2double((int)((u & 0x80000000u) | ((a >> 3) + 0x38000000u)), (int)(u << 29));
}
__device__ __forceinline__ float narrow(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const uint32_t hi = (uint32_t)(b >> 32), a = hi & 0x7fffffffu;
  // biased exponents 897 .. 1149: normal in fp32 also after rounding up
  if (a - 0x38100000u >= 0x47e00000u - 0x38100000u) return (float)v;
  // round to nearest even at bit 29, then rebias: exponent and fraction move as one number
  const unsigned long long m = (b & 0x7fffffffffffffffull) + 0x0fffffffull + ((b >> 29) & 1ull);
  return __uint_as_float((hi & 0x80000000u) | ((uint32_t)(m >> 29) - (896u << 23)));
}
// a cell index 0 .. 1023 as fp64
__device__ __forceinline__ double widen_index(int i) {
  const uint32_t u = __float_as_uint((float)i);
  return i ? __hiloint2double((int)((u >> 3) + 0x38000000u), (int)(u << 29)) : 0.0;
}

// up to three fields at once; every thread keeps four independent loads in flight. shift
// must be 0 for a plain conversion (it is then not subtracted).
struct ToF32 {
  const double *src[3];
  float *dst[3];
};
__global__ void __launch_bounds__(256) k_to_f32(ToF32 a, int64_t n, double shift) {
  const double *__restrict__ src = a.src[blockIdx.y];
  float *__restrict__ dst = a.dst[blockIdx.y];
  const int64_t i0 = (int64_t)blockIdx.x * (blockDim.x * 4) + threadIdx.x;
  double v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = i0 + q * 256 < n ? __ldcs(src + i0 + q * 256) : 0.0;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (i0 + q * 256 < n) dst[i0 + q * 256] = shift != 0.0 ? narrow(v[q] - shift) : narrow(v[q]);
}

// upload: absolute fp64 positions -> cell + fp32 offset (the reference's trunc cell)
// particles p0 .. p0 + n - 1 from fp64 arrays holding them from index 0
// The FP64 pipe is the bound, so a position below 2^20 cells takes two FP64 operations: its whole part is
// read out of the high word, and the same digits alone are subtracted (4,000,001 particles 163 us by
// conversions and floor, 153 with four operations, this way 108).
__global__ void k_from_f64(Geom G, F32Form f, const double *__restrict__ x, const double *__restrict__ y,
                           const double *__restrict__ z, const double *__restrict__ u, const double *__restrict__ v,
                           const double *__restrict__ w, const double *__restrict__ t, double tref, int64_t p0,
                           int64_t n, int32_t *__restrict__ err) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t p = p0 + i;
  const double X[3] = {x[i], y[i], z[i]};
  const double V[4] = {u[i], v[i], w[i], t[i]};
  int c[3];
  float o[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double xi = X[d] * G.idx[d];
    int i;
    float of;
    const uint32_t hi = (uint32_t)__double2hiint(xi);
    if (hi < 0x41300000u) {  // 0 <= xi < 2^20: the whole part is in the high word
      const int e = (int)(hi >> 20) - 1023;
      const uint32_t whole = e < 0 ? 0u : hi & ~((1u << (20 - e)) - 1u);  // its digits alone
      i = e < 0 ? 0 : (int)(((hi & 0xfffffu) | 0x100000u) >> (20 - e));
      of = narrow(xi - __hiloint2double((int)whole, 0));  // exact
    } else {
      if (!isfinite(xi)) { atomicOr(err, kErrNonFinite); xi = 0.0; }
      const double fl = floor(xi);
      i = (int)fl;
      of = (float)(xi - fl);
    }
    if (of >= 1.0f) { of = 0.0f; i += 1; }
    c[d] = wrapi(i, G.n[d]);
    o[d] = of;
  }
  const Set32 &B = f.set[SBASE];
  B.cell[p] = pack(c[0], c[1], c[2]);
#pragma unroll
  for (int d = 0; d < 3; ++d) B.o[d][p] = o[d];
  B.v[0][p] = narrow(V[0]);
  B.v[1][p] = narrow(V[1]);
  B.v[2][p] = narrow(V[2]);
  B.v[3][p] = narrow(V[3] - tref);
}

// the position conversions' cell sizes l/n (a double division each, made on the host) and -1024 times them
struct Dx {
  double d[3], off[3];
};
Dx cell_size(const Geom &G) {
  Dx r;
  for (int d = 0; d < 3; ++d) {
    r.d[d] = G.l[d] / G.n[d];
    r.off[d] = -1024.0 * r.d[d];
  }
  return r;
}
// (i + o) dx for a cell index below 1024 and an offset in [0, 1), rounded as written. From 2^-19 on
// i + o is exact and 1024 + i + o is put together from its digits, so that one fused operation gives
// the product: an FP64 instruction takes 16 cycles of an SM (with an addition and a product, the
// download of 2^24 particles took 438 us, this way 254).
__device__ __forceinline__ double position(int i, float o, const Dx &dx, int d) {
  const uint32_t u = __float_as_uint(o);
  if (u - 0x36000000u >= 0x3f800000u - 0x36000000u) return (widen_index(i) + widen(o)) * dx.d[d];
  const uint32_t m = (u & 0x007fffffu) | 0x00800000u;
  const int shift = (int)(u >> 23) - 108;  // 0 .. 18: o = (m << shift) 2^-42
  const uint32_t hi = (__funnelshift_l(m, 0u, shift) + ((uint32_t)i << 10)) | 0x40900000u;
  return fma(__hiloint2double((int)hi, (int)(m << shift)), dx.d[d], dx.off[d]);
}

// download: one array of a set as fp64 (positions back to absolute coordinates)
// particles p0 .. p0 + n - 1 into dst[0 .. n)
__global__ void k_to_f64_arr(Dx dx, Set32 S, int comp, double tref, int64_t p0, int64_t n,
                             double *__restrict__ dst) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int64_t p = p0 + q;
  if (comp < 3) {
    const uint32_t c = S.cell[p];
    const int i = comp == 0 ? ci_(c) : (comp == 1 ? cj_(c) : ck_(c));
    dst[q] = position(i, S.o[comp][p], dx, comp);
  } else if (comp < 6) {
    dst[q] = widen(S.v[comp - 3][p]);
  } else {
    dst[q] = widen(S.v[3][p]) + tref;
  }
}

// the particles' cells in brick order, and how many each cell holds (whole warps; 2^24 particles: 44 us
// and the count by itself 55, together 66)
__global__ void k_keys32(Geom G, Set32 S, int64_t n, uint32_t *__restrict__ key, int32_t *__restrict__ counts) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t id = 0xffffffffu;
  if (p < n) {
    const uint32_t c = S.cell[p];
    id = brick_id(G, ci_(c), cj_(c), ck_(c));
    key[p] = id;
  }
  const Run run = run_of(id);
  if (p < n && run.place == 0) atomicAdd(&counts[id], run.len);
}

// any key above its successor: the storage is not in key order
__global__ void k_keys_unsorted(const uint32_t *__restrict__ key, int64_t n, int32_t *__restrict__ flag) {
  int unsorted = 0;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p + 1 < n; p += (int64_t)gridDim.x * blockDim.x)
    unsorted |= key[p] > key[p + 1];
  if (__syncthreads_or(unsorted) && threadIdx.x == 0) atomicOr(flag, 1);
}

// Per-particle arrays gathered through the sort permutation, up to kPermBatch
// arrays of one element type per launch: the permutation is read once per batch
// and every thread keeps one independent load per array in flight (a gather of
// one array per launch is bound by load latency, not bandwidth).
// (2^24 particles, 11 arrays: eight and three 282 us, in one launch 249.)
constexpr int kPermBatch = 12;
template <typename T> struct PermBatch {
  const T *src[kPermBatch];
  T *dst[kPermBatch];
};
template <typename T, int K>
__global__ void __launch_bounds__(256) k_perm_batch(PermBatch<T> b, const int32_t *__restrict__ idx, int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t j = __ldcs(idx + i);
    T v[K];
#pragma unroll
    for (int a = 0; a < K; ++a) v[a] = __ldcs(b.src[a] + j);
#pragma unroll
    for (int a = 0; a < K; ++a) __stcs(b.dst[a] + i, v[a]);
  }
}

__global__ void k_f32_to_f64(const float *__restrict__ src, int64_t n, double *__restrict__ dst) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = widen(src[i]);
}

__global__ void k_to_f32_shift(const float *__restrict__ src, int64_t n, double shift, double *__restrict__ dst) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = widen(src[i]) + shift;
}

__global__ void k_recip32(const double *__restrict__ tau, int64_t n, float *__restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (float)(1. / tau[i]);
}

inline int nb(int64_t n) { return (int)((n + kThreads - 1) / kThreads); }

C32 make_c32(const pstep_ctx *h, int k, double pre, double post) {
  const pstep_config &cfg = h->cfg;
  C32 c;
  const double dt = cfg.dt;
  const double iS = 1. / (cfg.mp * cfg.cvp);
  c.dt_pre = (float)(dt * pre);
  c.dt_post = (float)(dt * post);
  c.dt_pre_is = (float)(dt * pre * iS);
  c.dt_post_is = (float)(dt * post * iS);
  for (int d = 0; d < 3; ++d) {
    c.dpre_idx[d] = (float)(dt * pre * h->geom.idx[d]);
    c.dpost_idx[d] = (float)(dt * post * h->geom.idx[d]);
  }
  c.itp = cfg.tp != 0 ? (float)(1. / cfg.tp) : 0.f;
  c.g[0] = (float)(cfg.particle_gravity * cfg.gx);
  c.g[1] = (float)(cfg.particle_gravity * cfg.gy);
  c.g[2] = (float)(cfg.particle_gravity * cfg.gz);
  c.alpha = (float)(0.25 * cfg.epsilonp * kPi * cfg.dp * cfg.dp * cfg.i0);
  c.itth = (float)(cfg.nu * kPi * cfg.dp * cfg.k);
  c.is = (float)iS;
  (void)k;
  return c;
}

template <typename T>
int dalloc32(pstep_ctx *h, T *&p, size_t count) {
  p = nullptr;
  cudaError_t e = cudaMalloc((void **)&p, sizeof(T) * (count ? count : 1));
  if (e != cudaSuccess) {
    p = nullptr;
    snprintf(h->err, sizeof h->err, "cudaMalloc: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return PSTEP_ERR_NOMEM;
  }
  return PSTEP_OK;
}
template <typename T>
void dfree32(T *&p) {
  if (p) cudaFree((void *)p);
  p = nullptr;
}

#define TRY32(x)                       \
  do {                                 \
    int rc_ = (x);                     \
    if (rc_ != PSTEP_OK) return rc_;   \
  } while (0)

int dep_launch(pstep_ctx *h, bool do_int, Set32 SI, Set32 SN, bool ext);

// check_sorted: first test whether the storage is in key order already (a population
// uploaded as an earlier step left it, e.g. a host round trip), and then only build the
// cell-start table; one 4-byte read-back
int sort_step(pstep_ctx *h, bool check_sorted = false) {
  // particles by brick-major cell of the base position; storage reordered; per-cell CSR kept
  F32Form &f = *h->f32;
  const Geom &G = h->geom;
  const int64_t n = h->np;
  const int64_t ncell = (int64_t)G.n[0] * G.n[1] * G.n[2];
  // the brick-major cells and the permutation: RHS_u holds nothing between stages
  uint32_t *key = reinterpret_cast<uint32_t *>(f.rhs_u[0]);
  int32_t *sidx = reinterpret_cast<int32_t *>(f.rhs_u[1]);
  PSTEP_CUDA(cudaMemsetAsync(h->counts, 0, sizeof(int32_t) * ncell, h->stream));
  if (n > 0) {
    k_keys32<<<nb(n), kThreads, 0, h->stream>>>(G, f.set[SBASE], n, key, h->counts);
    PSTEP_LAUNCHED(h);
  }
  bool in_order = false;
  if (check_sorted && n > 1) {
    PSTEP_CUDA(cudaMemsetAsync(f.unsorted, 0, sizeof(int32_t), h->stream));
    k_keys_unsorted<<<h->num_sms * 8, kThreads, 0, h->stream>>>(key, n, f.unsorted);
    PSTEP_LAUNCHED(h);
    int32_t u = 1;
    PSTEP_CUDA(cudaMemcpyAsync(&u, f.unsorted, sizeof u, cudaMemcpyDeviceToHost, h->stream));
    PSTEP_CUDA(cudaStreamSynchronize(h->stream));
    in_order = u == 0;
  }
  // The order inside a cell is left as the scatter makes it: every result of this form
  // (integer deposit sums, per-particle states by id) is independent of storage order.
  if (in_order)
    TRY32(exclusive_scan(h, h->counts, ncell, f.cell_start, nullptr));
  else
    TRY32(csr_sort(h, key, 0, ncell, h->s.flag, f.cell_start, sidx, nullptr, 0, true));
  if (n > 0 && !in_order) {
    Set32 &B = f.set[SBASE];
    // every 4-byte per-particle array that lives across steps; the addresses of their
    // pointer fields (float *, uint32_t *, int32_t *), swapped through memcpy
    void *arrs[32];
    int na = 0;
    for (int d = 0; d < 3; ++d) arrs[na++] = &B.o[d];
    for (int q = 0; q < 4; ++q) arrs[na++] = &B.v[q];
    arrs[na++] = &B.cell;
    arrs[na++] = &h->s.flag;
    arrs[na++] = &f.rhs_t;
    if (f.itp) arrs[na++] = &f.itp;
    for (int q = 0; q < 7; ++q)
      if (f.pp[q]) arrs[na++] = &f.pp[q];
    for (int q = 0; q < 4; ++q)
      if (f.gas[q]) arrs[na++] = &f.gas[q];
    // Scratch: the *_np1 set's 8 arrays and four of the *_new set's. After the step's last stage
    // the base set holds the new positions and every *_int, *_new and *_np1 query reads the base
    // set, so the stage sets carry nothing across the step boundary.
    Set32 &S = f.set[SNP1], &S2 = f.set[SNEW];
    void *scr[kPermBatch] = {&S.cell, &S.o[0], &S.o[1], &S.o[2], &S.v[0], &S.v[1],
                             &S.v[2], &S.v[3], &S2.v[0], &S2.v[1], &S2.v[2], &S2.v[3]};
    auto get = [](void *field) { void *p; memcpy(&p, field, sizeof p); return p; };
    auto put = [](void *field, void *p) { memcpy(field, &p, sizeof p); };
    const int pgrid = h->num_sms * 8;
    for (int a0 = 0; a0 < na; a0 += kPermBatch) {
      const int k = na - a0 < kPermBatch ? na - a0 : kPermBatch;
      PermBatch<uint32_t> pb{};
      for (int a = 0; a < k; ++a) {
        pb.src[a] = (const uint32_t *)get(arrs[a0 + a]);
        pb.dst[a] = (uint32_t *)get(scr[a]);
      }
      switch (k) {
        case 1: k_perm_batch<uint32_t, 1><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 2: k_perm_batch<uint32_t, 2><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 3: k_perm_batch<uint32_t, 3><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 4: k_perm_batch<uint32_t, 4><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 5: k_perm_batch<uint32_t, 5><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 6: k_perm_batch<uint32_t, 6><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 7: k_perm_batch<uint32_t, 7><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 8: k_perm_batch<uint32_t, 8><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 9: k_perm_batch<uint32_t, 9><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 10: k_perm_batch<uint32_t, 10><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        case 11: k_perm_batch<uint32_t, 11><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
        default: k_perm_batch<uint32_t, 12><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n); break;
      }
      PSTEP_LAUNCHED(h);
      for (int a = 0; a < k; ++a) {  // the gathered copy takes the array's place; the old one is scratch
        void *old = get(arrs[a0 + a]);
        put(arrs[a0 + a], pb.dst[a]);
        put(scr[a], old);
      }
    }
    // f.corr_y (the network output) is not carried: stage 0 rewrites it for every
    // particle before stages 1-3 read it, so it is the drive state's scratch here
    if (f.drive) {
      PermBatch<uint2> pb{};
      pb.src[0] = f.drive;
      pb.dst[0] = f.corr_y;
      k_perm_batch<uint2, 1><<<pgrid, 256, 0, h->stream>>>(pb, sidx, n);
      PSTEP_LAUNCHED(h);
      uint2 *t = f.drive;
      f.drive = f.corr_y;
      f.corr_y = t;
    }
  }
  // deposit work lists for this step's particle distribution
  PSTEP_CUDA(cudaMemsetAsync(f.work.counts, 0, 2 * sizeof(int32_t), h->stream));
  const int thin = thin_population(n, ncell);
  if (thin && !f.thin) {  // no tiles from here on: every word 0, as the gather leaves them
    PSTEP_CUDA(cudaMemsetAsync(f.work.mid, 0, sizeof(uint32_t) * f.work.nb * kRows * kBr, h->stream));
    PSTEP_CUDA(cudaMemsetAsync(f.work.side, 0, sizeof(uint32_t) * f.work.nb * kSideWords, h->stream));
    f.mom_stale = 0;
  }
  f.thin = thin;
  k_work<<<nb(f.work.nb), 256, 0, h->stream>>>(f.cell_start, f.work, f.whole_since ? 0 : 1, thin);
  PSTEP_LAUNCHED(h);
  f.whole_since = 0;
  f.sorted = 1;
  return PSTEP_OK;
}

}  // namespace

int f32_create(pstep_ctx *h) {
  const Geom &G = h->geom;
  for (int d = 0; d < 3; ++d) {
    if (G.n[d] > kMaxN || G.n[d] % kBr != 0 || G.n[d] < 2 * kBr) {
      snprintf(h->err, sizeof h->err, "FP32 form needs cells per side a multiple of %d in [%d, %d]", kBr, 2 * kBr,
               kMaxN);
      return PSTEP_ERR_CONFIG;
    }
  }
  F32Form *f = new F32Form();
  memset((void *)f, 0, sizeof(F32Form));
  h->f32 = f;
  const size_t cap = (size_t)h->cap;
  for (int s = 0; s < 4; ++s) {
    TRY32(dalloc32(h, f->set[s].cell, cap));
    for (int d = 0; d < 3; ++d) TRY32(dalloc32(h, f->set[s].o[d], cap));
    for (int q = 0; q < 4; ++q) TRY32(dalloc32(h, f->set[s].v[q], cap));
    // zeros (cell 0, offset 0) until a stage writes them: a stage that stopped early
    // (a device-side error) leaves nothing unwritten behind it
    PSTEP_CUDA(cudaMemsetAsync(f->set[s].cell, 0, sizeof(uint32_t) * cap, h->stream));
    for (int d = 0; d < 3; ++d) PSTEP_CUDA(cudaMemsetAsync(f->set[s].o[d], 0, sizeof(float) * cap, h->stream));
    for (int q = 0; q < 4; ++q) PSTEP_CUDA(cudaMemsetAsync(f->set[s].v[q], 0, sizeof(float) * cap, h->stream));
  }
  TRY32(dalloc32(h, f->rhs_t, cap));
  PSTEP_CUDA(cudaMemsetAsync(f->rhs_t, 0, sizeof(float) * cap, h->stream));
  for (int d = 0; d < 3; ++d) {
    TRY32(dalloc32(h, f->rhs_u[d], cap));
    PSTEP_CUDA(cudaMemsetAsync(f->rhs_u[d], 0, sizeof(float) * cap, h->stream));
  }
  if (h->cfg.flags & PSTEP_KEEP_GAS)
    for (int q = 0; q < 4; ++q) {
      TRY32(dalloc32(h, f->gas[q], cap));
      PSTEP_CUDA(cudaMemsetAsync(f->gas[q], 0, sizeof(float) * cap, h->stream));
    }
  const size_t gs = (size_t)G.gsize;
  for (int d = 0; d < 3; ++d) TRY32(dalloc32(h, f->uf[d], gs));
  TRY32(dalloc32(h, f->tf, gs));
  const size_t ncell = (size_t)G.n[0] * G.n[1] * G.n[2];
  TRY32(dalloc32(h, f->cell_start, ncell + 1));
  {  // deposit work lists, tiles and 64-bit sums
    Work &w = f->work;
    w.nb = (G.n[0] / kBr) * (G.n[1] / kBr) * (G.n[2] / kBr);
    w.ncell = (int64_t)ncell;
    // a brick of c > kItemMax particles makes ceil(c / kItemMax) <= 2 c / kItemMax slices
    w.slice_cap = 2 * (int64_t)h->cap / kItemMax + 1;
    TRY32(dalloc32(h, w.items, (size_t)(w.slice_cap + w.nb)));
    TRY32(dalloc32(h, w.counts, 4));
    TRY32(dalloc32(h, w.dirty, (size_t)w.nb));
    TRY32(dalloc32(h, w.extra_epoch, (size_t)w.nb));
    TRY32(dalloc32(h, w.word_epoch, (size_t)w.nb));
    PSTEP_CUDA(cudaMemsetAsync(w.word_epoch, 0, sizeof(int32_t) * w.nb, h->stream));
    const size_t mid = (size_t)w.nb * kRows * kBr, sides = (size_t)w.nb * kSideWords;
    TRY32(dalloc32(h, w.mid, mid));
    TRY32(dalloc32(h, w.side, sides));
    TRY32(dalloc32(h, w.extra, 5 * ncell));
    PSTEP_CUDA(cudaMemsetAsync(w.counts, 0, 4 * sizeof(int32_t), h->stream));
    PSTEP_CUDA(cudaMemsetAsync(w.extra_epoch, 0, sizeof(int32_t) * w.nb, h->stream));
    PSTEP_CUDA(cudaMemsetAsync(w.dirty, 0, w.nb, h->stream));
    PSTEP_CUDA(cudaMemsetAsync(w.mid, 0, sizeof(uint32_t) * mid, h->stream));
    PSTEP_CUDA(cudaMemsetAsync(w.side, 0, sizeof(uint32_t) * sides, h->stream));
    PSTEP_CUDA(cudaMemsetAsync(w.extra, 0, sizeof(long long) * 5 * ncell, h->stream));
  }
  TRY32(dalloc32(h, f->slots, kBoundSlots * 4));
  PSTEP_CUDA(cudaMemsetAsync(f->slots, 0, kBoundSlots * 4 * sizeof(uint32_t), h->stream));
  TRY32(dalloc32(h, f->pslots, kBoundSlots * 2));
  TRY32(dalloc32(h, f->unsorted, 1));
  f->pmax_state = 0;
  TRY32(dalloc32(h, f->se, 8));
  TRY32(dalloc32(h, f->totals, 16));
  TRY32(dalloc32(h, f->fstat, 16));
  PSTEP_CUDA(cudaMemsetAsync(f->fstat, 0, 16 * sizeof(double), h->stream));
  TRY32(dalloc32(h, h->s.flag, cap));
  TRY32(dalloc32(h, f->done, 1));
  PSTEP_CUDA(cudaMemsetAsync(f->done, 0, sizeof(int32_t), h->stream));
  return PSTEP_OK;
}

int f32_destroy(pstep_ctx *h) {
  F32Form *f = h->f32;
  if (!f) return PSTEP_OK;
  for (int s = 0; s < 4; ++s) {
    dfree32(f->set[s].cell);
    for (int d = 0; d < 3; ++d) dfree32(f->set[s].o[d]);
    for (int q = 0; q < 4; ++q) dfree32(f->set[s].v[q]);
  }
  dfree32(f->rhs_t); dfree32(f->itp);
  if (f->corr_mem) cudaFree(f->corr_mem);
  for (int q = 0; q < 7; ++q) dfree32(f->pp[q]);
  for (int q = 0; q < 4; ++q) dfree32(f->gas[q]);
  dfree32(f->drive);
  dfree32(f->corr_y);
  for (int d = 0; d < 3; ++d) { dfree32(f->rhs_u[d]); dfree32(f->uf[d]); }
  dfree32(f->tf); dfree32(f->cell_start);
  dfree32(f->done); dfree32(f->se); dfree32(f->slots); dfree32(f->pslots); dfree32(f->unsorted); dfree32(f->totals); dfree32(f->fstat);
  {
    Work &w = f->work;
    dfree32(w.items); dfree32(w.counts); dfree32(w.dirty); dfree32(w.extra_epoch); dfree32(w.word_epoch);
    dfree32(w.mid); dfree32(w.side); dfree32(w.extra);
  }
  if (f->stage[0]) {
    cudaStreamSynchronize(f->copy_stream);
    for (int sl = 0; sl < 2; ++sl) {
      dfree32(f->stage[sl]);
      cudaEventDestroy(f->ev_copied[sl]);
      cudaEventDestroy(f->ev_used[sl]);
    }
    cudaStreamDestroy(f->copy_stream);
  }
  delete f;
  h->f32 = nullptr;
  return PSTEP_OK;
}

// the host-transfer staging of the FP32 form (first use)
static int stage_init(pstep_ctx *h) {
  F32Form &f = *h->f32;
  if (f.stage[0]) return PSTEP_OK;
  for (int sl = 0; sl < 2; ++sl) TRY32(dalloc32(h, f.stage[sl], (size_t)(kStageArrays * kStageChunk)));
  PSTEP_CUDA(cudaStreamCreateWithFlags(&f.copy_stream, cudaStreamNonBlocking));
  for (int sl = 0; sl < 2; ++sl) {
    PSTEP_CUDA(cudaEventCreateWithFlags(&f.ev_copied[sl], cudaEventDisableTiming));
    PSTEP_CUDA(cudaEventCreateWithFlags(&f.ev_used[sl], cudaEventDisableTiming));
  }
  return PSTEP_OK;
}

int f32_upload(pstep_ctx *h, const double *x, const double *y, const double *z, const double *u, const double *v,
               const double *w, const double *t, int on_device) {
  F32Form &f = *h->f32;
  const int64_t n = h->np;
  dfree32(f.itp);
  for (int q = 0; q < 7; ++q) dfree32(f.pp[q]);
  if (f.drive) PSTEP_CUDA(cudaMemsetAsync(f.drive, 0, sizeof(uint2) * (size_t)h->cap, h->stream));
  if (f.corr_y) PSTEP_CUDA(cudaMemsetAsync(f.corr_y, 0, sizeof(uint2) * (size_t)h->cap, h->stream));
  f.sorted = 0;
  f.pmax_state = 0;
  if (n == 0) return PSTEP_OK;
  if (!f.tref_set) {
    double t0 = 0.0;
    if (on_device) PSTEP_CUDA(cudaMemcpy(&t0, t, sizeof(double), cudaMemcpyDeviceToHost));
    else t0 = t[0];
    f.tref = (double)(float)t0;
    f.tref_set = 1;
  }
  const double *src[7] = {x, y, z, u, v, w, t};
  if (on_device) {
    k_from_f64<<<nb(n), kThreads, 0, h->stream>>>(h->geom, f, src[0], src[1], src[2], src[3], src[4], src[5],
                                                  src[6], f.tref, 0, n, h->err_word);
    PSTEP_LAUNCHED(h);
    return PSTEP_OK;
  }
  // host arrays: chunks of kStageChunk particles copied into the two staging slots in
  // turn on the copy stream, each converted on the handle's stream once it has landed
  TRY32(stage_init(h));
  for (int64_t c = 0, p0 = 0; p0 < n; ++c, p0 += kStageChunk) {
    const int sl = (int)(c & 1);
    const int64_t len = n - p0 < kStageChunk ? n - p0 : kStageChunk;
    // the slot's last conversion (of this upload, or of an earlier upload or read-back
    // still running on the handle's stream) is done; an event never recorded is complete
    PSTEP_CUDA(cudaStreamWaitEvent(f.copy_stream, f.ev_used[sl], 0));
    double *b = f.stage[sl];
    for (int q = 0; q < 7; ++q)
      PSTEP_CUDA(cudaMemcpyAsync(b + q * kStageChunk, src[q] + p0, sizeof(double) * len, cudaMemcpyHostToDevice,
                                 f.copy_stream));
    PSTEP_CUDA(cudaEventRecord(f.ev_copied[sl], f.copy_stream));
    PSTEP_CUDA(cudaStreamWaitEvent(h->stream, f.ev_copied[sl], 0));
    k_from_f64<<<nb(len), kThreads, 0, h->stream>>>(h->geom, f, b, b + kStageChunk, b + 2 * kStageChunk,
                                                    b + 3 * kStageChunk, b + 4 * kStageChunk, b + 5 * kStageChunk,
                                                    b + 6 * kStageChunk, f.tref, p0, len, h->err_word);
    PSTEP_LAUNCHED(h);
    PSTEP_CUDA(cudaEventRecord(f.ev_used[sl], h->stream));
  }
  // the host arrays may be reused when this returns: every copy has been read
  PSTEP_CUDA(cudaStreamSynchronize(f.copy_stream));
  return PSTEP_OK;
}

int f32_set_tau(pstep_ctx *h, const double *tau, int on_device) {
  F32Form &f = *h->f32;
  if (!tau) {
    dfree32(f.itp);
    return PSTEP_OK;
  }
  if (f.sorted) {
    snprintf(h->err, sizeof h->err, "tau_p must be set before pstep_prime");
    return PSTEP_ERR_STATE;
  }
  if (!f.itp) TRY32(dalloc32(h, f.itp, (size_t)h->cap));
  const int64_t n = h->np;
  if (n == 0) return PSTEP_OK;
  const double *src = tau;
  double *tmp = nullptr;
  if (!on_device) {
    TRY32(dalloc32(h, tmp, (size_t)n));
    PSTEP_CUDA(cudaMemcpyAsync(tmp, tau, sizeof(double) * n, cudaMemcpyHostToDevice, h->stream));
    src = tmp;
  }
  k_recip32<<<nb(n), kThreads, 0, h->stream>>>(src, n, f.itp);
  PSTEP_LAUNCHED(h);
  if (tmp) {
    PSTEP_CUDA(cudaStreamSynchronize(h->stream));
    dfree32(tmp);
  }
  return PSTEP_OK;
}

__global__ void k_d2f(const double *__restrict__ src, int64_t n, float *__restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (float)src[i];
}

int f32_set_props(pstep_ctx *h, const pstep_particle_props *pr, int on_device) {
  F32Form &f = *h->f32;
  if (f.sorted) {
    snprintf(h->err, sizeof h->err, "particle properties must be set before pstep_prime");
    return PSTEP_ERR_STATE;
  }
  TRY32(f32_set_tau(h, pr->tau_p, on_device));
  const double *src[7] = {pr->mass_ratio, pr->itth, pr->heat_is, pr->alpha, pr->accel[0], pr->accel[1], pr->accel[2]};
  const int64_t n = h->np;
  double *tmp = nullptr;
  if (!on_device && n > 0) TRY32(dalloc32(h, tmp, (size_t)n));
  for (int q = 0; q < 7; ++q) {
    if (!src[q]) {
      dfree32(f.pp[q]);
      continue;
    }
    if (!f.pp[q]) TRY32(dalloc32(h, f.pp[q], (size_t)h->cap));
    if (n == 0) continue;
    const double *s = src[q];
    if (!on_device) {
      PSTEP_CUDA(cudaMemcpyAsync(tmp, src[q], sizeof(double) * n, cudaMemcpyHostToDevice, h->stream));
      s = tmp;
    }
    k_d2f<<<nb(n), kThreads, 0, h->stream>>>(s, n, f.pp[q]);
    PSTEP_LAUNCHED(h);
  }
  if (tmp) {
    PSTEP_CUDA(cudaStreamSynchronize(h->stream));
    dfree32(tmp);
  }
  return PSTEP_OK;
}

// host round-to-nearest-even fp32 -> bf16 bits (finite values)
static uint16_t bf16_bits(float v) {
  uint32_t u;
  memcpy(&u, &v, 4);
  u += 0x7FFFu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}

int f32_set_correction(pstep_ctx *h, const pstep_correction *pc) {
  F32Form &f = *h->f32;
  if (f.corr_mem) {
    PSTEP_CUDA(cudaStreamSynchronize(h->stream));
    cudaFree(f.corr_mem);
    f.corr_mem = nullptr;
  }
  h->corr_on = 0;
  if (!pc) return PSTEP_OK;
  if (!pc->params || !(pc->nu_gas > 0)) {
    snprintf(h->err, sizeof h->err, "correction needs parameters and a positive gas viscosity");
    return PSTEP_ERR_ARG;
  }
  const Geom &G = h->geom;
  if (G.n[0] != G.n[1] || G.n[0] != G.n[2] || G.l[0] != G.l[1] || G.l[0] != G.l[2]) {
    snprintf(h->err, sizeof h->err, "the correction's d_p/dx needs a cubic grid");
    return PSTEP_ERR_CONFIG;
  }
  // weight tiles in the canonical K-major layout (tc05.cuh), then fp32 biases
  const size_t bias_off = corr::kImage;
  const size_t bytes = bias_off + sizeof(float) * (corr::kHid + corr::kHid + corr::kOutP);
  uint8_t *img = (uint8_t *)calloc(1, bytes);
  const float *P = pc->params;
  for (int o = 0; o < corr::kHid; ++o)
    for (int j = 0; j < corr::kInP; ++j)
      *(uint16_t *)(img + corr::W1 + tc05::tile_off(o, j, corr::kInP)) = bf16_bits(P[o * corr::kInP + j]);
  for (int o = 0; o < corr::kHid; ++o)
    for (int i = 0; i < corr::kHid; ++i)
      *(uint16_t *)(img + corr::W2 + tc05::tile_off(o, i, corr::kHid)) = bf16_bits(P[1088 + o * corr::kHid + i]);
  for (int o = 0; o < corr::kOutP; ++o)
    for (int i = 0; i < corr::kHid; ++i)
      *(uint16_t *)(img + corr::W3 + tc05::tile_off(o, i, corr::kHid)) = bf16_bits(P[5248 + o * corr::kHid + i]);
  float *bias = (float *)(img + bias_off);
  for (int q = 0; q < corr::kHid; ++q) bias[q] = P[1024 + q];
  for (int q = 0; q < corr::kHid; ++q) bias[corr::kHid + q] = P[5184 + q];
  for (int q = 0; q < corr::kOutP; ++q) bias[2 * corr::kHid + q] = P[6272 + q];
  cudaError_t e = cudaMalloc(&f.corr_mem, bytes);
  if (e == cudaSuccess) e = cudaMemcpy(f.corr_mem, img, bytes, cudaMemcpyHostToDevice);
  free(img);
  if (e != cudaSuccess) {
    cudaGetLastError();
    f.corr_mem = nullptr;
    snprintf(h->err, sizeof h->err, "correction upload: %s", cudaGetErrorString(e));
    return PSTEP_ERR_CUDA;
  }
  CorrDev &cd = *reinterpret_cast<CorrDev *>(h->corr_dev);
  cd.image = (const uint4 *)f.corr_mem;
  cd.bias = (const float *)((const uint8_t *)f.corr_mem + bias_off);
  for (int q = 0; q < 10; ++q) { cd.shift[q] = pc->shift[q]; cd.scale[q] = pc->scale[q]; }
  for (int q = 0; q < 4; ++q) { cd.lo[q] = pc->lo[q]; cd.hi[q] = pc->hi[q]; }
  cd.inv_nu = (float)(1.0 / pc->nu_gas);
  cd.inv_prior_re = pc->prior_re > 0.f ? 1.f / pc->prior_re : 0.f;
  const pstep_config &cfg = h->cfg;
  cd.dp_per_itth = (cfg.nu > 0 && cfg.k > 0) ? (float)(1.0 / (cfg.nu * kPi * cfg.k)) : 0.f;
  cd.dp = (float)cfg.dp;
  cd.idx = (float)G.idx[0];
  h->corr_every_stage = pc->every_stage ? 1 : 0;
  cd.drive_cap = pc->drive_cap > 0.f ? pc->drive_cap : kDriveCap;
  if (!f.drive) TRY32(dalloc32(h, f.drive, (size_t)h->cap));
  PSTEP_CUDA(cudaMemsetAsync(f.drive, 0, sizeof(uint2) * (size_t)h->cap, h->stream));
  if (!f.corr_y) TRY32(dalloc32(h, f.corr_y, (size_t)h->cap));
  PSTEP_CUDA(cudaMemsetAsync(f.corr_y, 0, sizeof(uint2) * (size_t)h->cap, h->stream));
  h->corr_on = 1;
  return PSTEP_OK;
}

// fp32 copies of the fields just bound: which = 1 the velocity (3 fields), 2 the temperature
int f32_bind_fields(pstep_ctx *h, int which) {
  F32Form &f = *h->f32;
  const int64_t gs = h->geom.gsize;
  if (h->tf && !f.tref_set) {
    double t0 = 0.0;  // first interior cell
    PSTEP_CUDA(cudaMemcpyAsync(&t0, h->tf + glin(h->geom, 1, 1, 1), sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    PSTEP_CUDA(cudaStreamSynchronize(h->stream));
    f.tref = (double)(float)t0;
    f.tref_set = 1;
  }
  const double *src[4] = {h->ux, h->uy, h->uz, h->tf};
  float *dst[4] = {f.uf[0], f.uf[1], f.uf[2], f.tf};
  ToF32 a{};
  int nf = 0;
  for (int q = 0; q < 3; ++q)
    if (src[q] && (which & 1)) {
      a.src[nf] = src[q];
      a.dst[nf++] = dst[q];
    }
  const unsigned blocks = (unsigned)((gs + 1023) / 1024);
  if (nf) {
    k_to_f32<<<dim3(blocks, (unsigned)nf), 256, 0, h->stream>>>(a, gs, 0.0);
    PSTEP_LAUNCHED(h);
  }
  if (src[3] && (which & 2)) {
    a.src[0] = src[3];
    a.dst[0] = dst[3];
    k_to_f32<<<blocks, 256, 0, h->stream>>>(a, gs, f.tref);
    PSTEP_LAUNCHED(h);
  }
  return PSTEP_OK;
}

int f32_prime(pstep_ctx *h) {
  F32Form &f = *h->f32;
  TRY32(sort_step(h, true));
  const C32 c = make_c32(h, 0, 0.5, 1. / 6.);
  if (h->np > 0) {
    k_prime32<<<nb(h->np), kThreads, 0, h->stream>>>(h->geom, f, c.itth, h->np);
    PSTEP_LAUNCHED(h);
  }
  // part2gas_Temp_int at the base positions
  return dep_launch(h, false, f.set[SBASE], f.set[SBASE], true);
}

int f32_stage(pstep_ctx *h, int k, double pre, double post) {
  F32Form &f = *h->f32;
  const C32 c = make_c32(h, k, pre, post);
  const int64_t n = h->np;
  const int nb_adv = (int)((n + kAdvThreads - 1) / kAdvThreads), nb_corr = (int)((n + kCorrThreads - 1) / kCorrThreads);
  CorrDev cd = *reinterpret_cast<const CorrDev *>(h->corr_dev);
  cd.wait_limit = h->wait_limit;
  cd.idle_first = h->wait_idle ? 1u : 0u;
  if (n > 0 && h->corr_on && (k == 0 || h->corr_every_stage)) {
    // the network at this stage's x_int: persistent CTAs of two warpgroups, 4 per SM,
    // tiles of 128 particles
    prof_begin(h, PSTEP_PHASE_NETWORK);
    const int64_t pairs = (n + 2 * corr::kRows - 1) / (2 * corr::kRows);
    const unsigned grid = (unsigned)(pairs < 4 * (int64_t)h->num_sms ? pairs : 4 * (int64_t)h->num_sms);
    auto net = k == 0 ? k_corr_net<0> : (k == 1 ? k_corr_net<1> : (k == 2 ? k_corr_net<2> : k_corr_net<3>));
    // the shared-memory opt-in belongs to the current (launch) device: set it per launch
    PSTEP_CUDA(cudaFuncSetAttribute(net, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)corr::kAlloc));
    net<<<grid, corr::kThreads, corr::kAlloc, h->stream>>>(h->geom, f, c, n, h->err_word, cd);
    PSTEP_LAUNCHED(h);
    prof_end(h, PSTEP_PHASE_NETWORK);
  }
  if (k == 3) {  // the last stage gathers the step result's max u and max ug
    PSTEP_CUDA(cudaMemsetAsync(f.pslots, 0, sizeof(uint32_t) * kBoundSlots * 2, h->stream));
    f.pmax_state = 1;
  } else if (f.pmax_state == 1) {
    f.pmax_state = 0;  // a stage after the last one without the step's end
  }
  prof_begin(h, PSTEP_PHASE_ADVANCE);
  if (n > 0 && h->corr_on) {
    switch (k) {
      case 0: k_advance32_corr<0><<<nb_corr, kCorrThreads, 0, h->stream>>>(h->geom, f, c, h->cfg.twc, n, h->err_word, cd); break;
      case 1: k_advance32_corr<1><<<nb_corr, kCorrThreads, 0, h->stream>>>(h->geom, f, c, h->cfg.twc, n, h->err_word, cd); break;
      case 2: k_advance32_corr<2><<<nb_corr, kCorrThreads, 0, h->stream>>>(h->geom, f, c, h->cfg.twc, n, h->err_word, cd); break;
      default: k_advance32_corr<3><<<nb_corr, kCorrThreads, 0, h->stream>>>(h->geom, f, c, h->cfg.twc, n, h->err_word, cd); break;
    }
    PSTEP_LAUNCHED(h);
  } else if (n > 0) {
    switch (k) {
      case 0: k_advance32<0><<<nb_adv, kAdvThreads, 0, h->stream>>>(h->geom, f, c, h->cfg.twc, n, h->err_word); break;
      case 1: k_advance32<1><<<nb_adv, kAdvThreads, 0, h->stream>>>(h->geom, f, c, h->cfg.twc, n, h->err_word); break;
      case 2: k_advance32<2><<<nb_adv, kAdvThreads, 0, h->stream>>>(h->geom, f, c, h->cfg.twc, n, h->err_word); break;
      default: k_advance32<3><<<nb_adv, kAdvThreads, 0, h->stream>>>(h->geom, f, c, h->cfg.twc, n, h->err_word); break;
    }
    PSTEP_LAUNCHED(h);
  }
  prof_end(h, PSTEP_PHASE_ADVANCE);
  // one walk: concentration + momentum at *_int (the base itself at stage 0), RHS_T at *_new;
  // the field extrema (pstep_field_stats) only in the step's last stage, whose fields the
  // step leaves
  prof_begin(h, PSTEP_PHASE_DEPOSIT_INT);
  TRY32(dep_launch(h, true, f.set[h->int_is_base ? SBASE : SINT], f.set[SNEW], k == 3));
  prof_end(h, PSTEP_PHASE_DEPOSIT_INT);
  return PSTEP_OK;
}

namespace {
// The deposit at SI (concentration and momentum; do_int) and SN (RHS_T): scales and counters, the
// tiles, then the fields with their ghost layers and balance sums.
int dep_launch(pstep_ctx *h, bool do_int, Set32 SI, Set32 SN, bool ext) {
  F32Form &f = *h->f32;
  const Geom &G = h->geom;
  const int32_t epoch = ++f.epoch;
  const int twc = h->cfg.twc;
  // fields with sums: RHS_Part_Temp, and C, and (with TWC) the momentum
  const int fields = do_int ? (twc ? 2 : 1) : 0;
  const int64_t most = (int64_t)f.work.nb + f.work.slice_cap;
  const unsigned grid_t = (unsigned)(most < 4 * (int64_t)h->num_sms ? most : 4 * (int64_t)h->num_sms);
  if (fields == 2 && f.mom_stale && !f.thin) {  // TWC switched on again: this launch writes the listed bricks' tiles, the rest are zeros
    PSTEP_CUDA(cudaMemsetAsync(f.work.mid, 0, sizeof(uint32_t) * f.work.nb * kRows * kBr, h->stream));
    PSTEP_CUDA(cudaMemsetAsync(f.work.side, 0, sizeof(uint32_t) * f.work.nb * kSideWords, h->stream));
  }
  auto tile = f.thin ? (fields == 2 ? k_dep_tile<2, true> : (fields == 1 ? k_dep_tile<1, true> : k_dep_tile<0, true>))
                     : (fields == 2 ? k_dep_tile<2, false> : (fields == 1 ? k_dep_tile<1, false> : k_dep_tile<0, false>));
  tile<<<grid_t, kDepThreads, 0, h->stream>>>(G, f, SI, SN, epoch, h->np);
  PSTEP_LAUNCHED(h);
  if (fields && !f.thin) {
    f.whole_since = 1;
    f.mom_stale = fields == 1;
  }
  double *C = h->dep[PSTEP_FIELD_C], *X = h->dep[PSTEP_FIELD_RU_X], *Y = h->dep[PSTEP_FIELD_RU_Y],
         *Z = h->dep[PSTEP_FIELD_RU_Z], *E = h->dep[PSTEP_FIELD_PART_TEMP];
  const int64_t tasks = (int64_t)((G.n[0] + 31) / 32) * (G.n[1] / kBr) * (G.n[2] / kBr), fit = 4 * (int64_t)h->num_sms;
  auto gather = f.thin ? (ext ? k_dep_gather<true, true> : k_dep_gather<false, true>)
                       : (ext ? k_dep_gather<true, false> : k_dep_gather<false, false>);
  gather<<<dim3((unsigned)(tasks < fit ? tasks : fit), fields ? 5 : 1), 256, 0, h->stream>>>(
      G, f, epoch, fields == 2 ? 5 : fields + 1, 1.0 / ((double)G.n[0] * G.n[1] * G.n[2]), C, X, Y, Z, E, h->mom_dev,
      h->emean_dev);
  PSTEP_LAUNCHED(h);
  for (int q = 0; q < 5; ++q)
    if (do_int || q == 4) f.ext_ok[q] = ext ? 1 : 0;
  return PSTEP_OK;
}
}  // namespace

// particle::max of u or ug (grid.cpp:726-727) as the last stage gathered them, when they
// describe the current base state (the step's result): PSTEP_OK with *out set, or -1
// when they are not available (the caller then makes a pass over the array)
int f32_fused_max(pstep_ctx *h, int id, double *out) {
  F32Form &f = *h->f32;
  if (f.pmax_state != 2 || (id != PSTEP_U && id != PSTEP_UG)) return -1;
  uint32_t keys[kBoundSlots * 2];
  PSTEP_CUDA(cudaMemcpyAsync(keys, f.pslots, sizeof keys, cudaMemcpyDeviceToHost, h->stream));
  PSTEP_CUDA(cudaStreamSynchronize(h->stream));
  const int q = id == PSTEP_U ? 0 : 1;
  uint32_t best = 0;
  for (int s = 0; s < kBoundSlots; ++s) best = keys[2 * s + q] > best ? keys[2 * s + q] : best;
  if (best == 0) return -1;
  const uint32_t bits = (best & 0x80000000u) ? (best & 0x7fffffffu) : ~best;
  float v;
  memcpy(&v, &bits, sizeof v);
  *out = (double)v;
  return PSTEP_OK;
}

// a deposited field's max, min and interior sum as the last deposit that wrote it
// gathered them (FP32 form): PSTEP_OK with r set, or -1 when that deposit did not gather
// the extrema (a stage other than a step's last; the caller then makes a pass)
int f32_field_stats(pstep_ctx *h, int field, double r[3]) {
  F32Form &f = *h->f32;
  if (!f.ext_ok[field]) return -1;
  PSTEP_CUDA(cudaMemcpyAsync(r, f.fstat + 3 * field, 3 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  PSTEP_CUDA(cudaStreamSynchronize(h->stream));
  return PSTEP_OK;
}

int f32_end_stage(pstep_ctx *h) {
  F32Form &f = *h->f32;
  Set32 t = f.set[SINT];
  f.set[SINT] = f.set[SNEW];
  f.set[SNEW] = t;
  return PSTEP_OK;
}

int f32_end_step(pstep_ctx *h) {
  F32Form &f = *h->f32;
  f.pmax_state = f.pmax_state == 1 ? 2 : 0;  // the last stage's maxima describe the new base
  Set32 t = f.set[SBASE];
  f.set[SBASE] = f.set[SNP1];
  f.set[SNP1] = t;
  prof_begin(h, PSTEP_PHASE_REORDER);
  int rc = sort_step(h);
  prof_end(h, PSTEP_PHASE_REORDER);
  return rc;
}

namespace {
__global__ void k_positions32(Dx dx, Set32 S, const int32_t *__restrict__ idx, int32_t n, double *__restrict__ xyz) {
  const int32_t i = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n) return;
  const int32_t p = idx[i];
  if (p < 0) return;
  const uint32_t c = S.cell[p];
  const int cc[3] = {ci_(c), cj_(c), ck_(c)};
#pragma unroll
  for (int d = 0; d < 3; ++d) xyz[3 * i + d] = position(cc[d], S.o[d][p], dx, d);
}
}  // namespace

// positions (as pstep_get_particle_array returns them) of the particles at storage
// indices idx[0 .. n) (negative: skipped) into xyz (device, 3 per particle)
int f32_positions(pstep_ctx *h, const int32_t *idx, int32_t n, double *xyz) {
  F32Form &f = *h->f32;
  if (n <= 0) return PSTEP_OK;
  k_positions32<<<(n + kThreads - 1) / kThreads, kThreads, 0, h->stream>>>(cell_size(h->geom), f.set[SBASE], idx, n, xyz);
  PSTEP_LAUNCHED(h);
  return PSTEP_OK;
}

namespace {
// the base state of particles p0 .. p0 + n - 1 as fp64 (absolute positions, velocities,
// temperature) into dst[q][0 .. n): the arrays pstep_get_particle_array returns for
// PSTEP_X .. PSTEP_T, all seven from one read of each particle. HBM-bound with the integer
// conversions and the cell size divided on the host (seven FP64 operations a particle are left).
__global__ void k_to_f64_all(Dx dx, Set32 S, double tref, int64_t p0, int64_t n, double *__restrict__ x,
                             double *__restrict__ y, double *__restrict__ z, double *__restrict__ u,
                             double *__restrict__ v, double *__restrict__ w, double *__restrict__ t) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int64_t p = p0 + q;
  const uint32_t c = S.cell[p];
  const float o0 = S.o[0][p], o1 = S.o[1][p], o2 = S.o[2][p];
  const float v0 = S.v[0][p], v1 = S.v[1][p], v2 = S.v[2][p], v3 = S.v[3][p];
  __stcs(x + q, position(ci_(c), o0, dx, 0));
  __stcs(y + q, position(cj_(c), o1, dx, 1));
  __stcs(z + q, position(ck_(c), o2, dx, 2));
  __stcs(u + q, widen(v0));
  __stcs(v + q, widen(v1));
  __stcs(w + q, widen(v2));
  __stcs(t + q, widen(v3) + tref);
}
}  // namespace

// pstep_download_particles, FP32 form: the base state and the ids in storage order. Host
// destinations: chunks converted into the two staging slots in turn and copied out on the
// copy stream, all seven arrays per chunk, so one pipeline serves the whole download.
int f32_download(pstep_ctx *h, double *const dst[7], int32_t *flag, int on_device) {
  F32Form &f = *h->f32;
  const int64_t n = h->np;
  if (n == 0) return PSTEP_OK;
  const Set32 &B = f.set[SBASE];
  if (on_device) {
    k_to_f64_all<<<nb(n), kThreads, 0, h->stream>>>(cell_size(h->geom), B, f.tref, 0, n, dst[0], dst[1], dst[2], dst[3],
                                                    dst[4], dst[5], dst[6]);
    PSTEP_LAUNCHED(h);
    PSTEP_CUDA(cudaMemcpyAsync(flag, h->s.flag, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, h->stream));
    PSTEP_CUDA(cudaStreamSynchronize(h->stream));
    return PSTEP_OK;
  }
  TRY32(stage_init(h));
  for (int64_t c = 0, p0 = 0; p0 < n; ++c, p0 += kStageChunk) {
    const int sl = (int)(c & 1);
    const int64_t len = n - p0 < kStageChunk ? n - p0 : kStageChunk;
    double *b = f.stage[sl];
    PSTEP_CUDA(cudaStreamWaitEvent(h->stream, f.ev_copied[sl], 0));  // the slot's last copy (any call) is done
    k_to_f64_all<<<nb(len), kThreads, 0, h->stream>>>(cell_size(h->geom), B, f.tref, p0, len, b, b + kStageChunk,
                                                      b + 2 * kStageChunk, b + 3 * kStageChunk, b + 4 * kStageChunk,
                                                      b + 5 * kStageChunk, b + 6 * kStageChunk);
    PSTEP_LAUNCHED(h);
    PSTEP_CUDA(cudaEventRecord(f.ev_used[sl], h->stream));
    PSTEP_CUDA(cudaStreamWaitEvent(f.copy_stream, f.ev_used[sl], 0));
    for (int q = 0; q < 7; ++q)
      PSTEP_CUDA(cudaMemcpyAsync(dst[q] + p0, b + q * kStageChunk, sizeof(double) * len, cudaMemcpyDeviceToHost,
                                 f.copy_stream));
    PSTEP_CUDA(cudaEventRecord(f.ev_copied[sl], f.copy_stream));
  }
  // the ids need no conversion: one copy behind the chunks, after everything enqueued on
  // the handle's stream so far
  PSTEP_CUDA(cudaEventRecord(f.ev_used[0], h->stream));
  PSTEP_CUDA(cudaStreamWaitEvent(f.copy_stream, f.ev_used[0], 0));
  PSTEP_CUDA(cudaMemcpyAsync(flag, h->s.flag, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, f.copy_stream));
  PSTEP_CUDA(cudaStreamSynchronize(f.copy_stream));
  return PSTEP_OK;
}

int f32_get_array(pstep_ctx *h, int id, void *dst, int on_device) {
  F32Form &f = *h->f32;
  const int64_t n = h->np;
  int set = SBASE, comp = 0;
  if (id <= PSTEP_T) { set = SBASE; comp = id - PSTEP_X; }
  else if (id <= PSTEP_T_INT) { set = h->int_is_base ? SBASE : SINT; comp = id - PSTEP_X_INT; }
  else if (id <= PSTEP_T_NEW) { set = h->phase != 0 ? SNEW : (h->int_is_base ? SBASE : SINT); comp = id - PSTEP_X_NEW; }
  else if (id <= PSTEP_T_NP1) { set = h->np1_is_base ? SBASE : SNP1; comp = id - PSTEP_X_NP1; }
  else set = -1;
  if (id >= PSTEP_UG && !f.gas[0]) {
    snprintf(h->err, sizeof h->err, "gas values per particle need the PSTEP_KEEP_GAS flag");
    return PSTEP_ERR_CONFIG;
  }
  // particles p0 .. p0 + len - 1 as fp64 into out[0 .. len)
  auto convert = [&](int64_t p0, int64_t len, double *out) {
    if (set >= 0) {
      k_to_f64_arr<<<nb(len), kThreads, 0, h->stream>>>(cell_size(h->geom), f.set[set], comp, f.tref, p0, len, out);
    } else if (id >= PSTEP_UG) {
      k_to_f32_shift<<<nb(len), kThreads, 0, h->stream>>>(f.gas[id - PSTEP_UG] + p0, len,
                                                          id == PSTEP_TG ? f.tref : 0.0, out);
    } else {
      k_f32_to_f64<<<nb(len), kThreads, 0, h->stream>>>(f.rhs_t + p0, len, out);  // RHS_T
    }
  };
  if (on_device) {
    convert(0, n, (double *)dst);
    PSTEP_LAUNCHED(h);
    PSTEP_CUDA(cudaStreamSynchronize(h->stream));  // complete on return, as for host destinations
    return PSTEP_OK;
  }
  // host destination: chunks converted into the staging slots in turn and copied out on
  // the copy stream, the copy of one overlapping the conversion of the next
  TRY32(stage_init(h));
  double *out = (double *)dst;
  for (int64_t c = 0, p0 = 0; p0 < n; ++c, p0 += kStageChunk) {
    const int sl = (int)(c & 1);
    const int64_t len = n - p0 < kStageChunk ? n - p0 : kStageChunk;
    PSTEP_CUDA(cudaStreamWaitEvent(h->stream, f.ev_copied[sl], 0));  // the slot's last copy (any call) is done
    convert(p0, len, f.stage[sl]);
    PSTEP_LAUNCHED(h);
    PSTEP_CUDA(cudaEventRecord(f.ev_used[sl], h->stream));
    PSTEP_CUDA(cudaStreamWaitEvent(f.copy_stream, f.ev_used[sl], 0));
    PSTEP_CUDA(cudaMemcpyAsync(out + p0, f.stage[sl], sizeof(double) * len, cudaMemcpyDeviceToHost, f.copy_stream));
    PSTEP_CUDA(cudaEventRecord(f.ev_copied[sl], f.copy_stream));
  }
  PSTEP_CUDA(cudaStreamSynchronize(f.copy_stream));
  return PSTEP_OK;
}

}  // namespace pstep
