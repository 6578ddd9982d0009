// Two-way-coupling deposition, FP64 drop-in form. No atomics anywhere: every
// target value is a sum in a fixed order, so results are identical run to run.
//
// Fast path (k_dep_brick): one CTA per brick of B^3 target cells of the ghosted
// grid. Its threads walk the CSR segments (particles sorted by node, then h,
// then storage index) of the brick's nodes plus a one-node halo and form partial
// sums in shared memory -- the 8 trilinear offsets of every node, and the
// face-normal partials of every trunc cell from the h classes' runs that fall into
// it, lists of like length side by side -- then every target cell sums its partials
// in a fixed order. Halo nodes are walked by both neighbouring bricks; no cross-brick
// reduction.
//
// Reference-order path (PSTEP_REFERENCE_SUMS, k_dep_ordered): a warp merges the node lists
// around its targets by the particles' positions in the reference's vectors, so every cell
// receives its contributions in exactly the order the reference's scatter loop adds them
// (particle.cpp:498-658), from 0, with the reference's weight expressions.
// Either way the cumulative ghost fold and the ghost refresh then replay
// communicator.cpp's single-rank sequence.
//
// Compiled with -fmad=false (see stage_f64.cu).
#include "pstep_internal.cuh"

namespace pstep {
namespace {

struct DepIn {
  const int32_t *cell_start;  // gsize + 1
  const int32_t *sidx;        // nullptr: identity
  const int32_t *okey;        // reference order: a sorted particle's position in the reference's vectors
  const double *frac[3];
  const uint32_t *key;
  const double *val[3];       // RHS_u,v,w (int-deposit) or RHS_T in val[0] (temperature deposit)
  const double *kept;         // the int-deposit: a field to be copied beside the targets, or nullptr
  double *keep;
};

__device__ inline int32_t pidx(const DepIn &d, int32_t p) { return d.sidx ? d.sidx[p] : p; }

__device__ inline bool node_ok(const Geom &G, int i, int j, int k) {
  // particle nodes are round(x*idx)+1 in 1..n+1
  return i >= 1 && i <= G.n[0] + 1 && j >= 1 && j <= G.n[1] + 1 && k >= 1 && k <= G.n[2] + 1;
}

__device__ inline double xl_round(double f, int h) { return (h ? (f - 1.0) : f) + 0.5; }

// Reference order. A warp owns 4 x 4 x 2 targets, a lane each, and merges the segments of all nodes
// that reach them (sorted by the particles' positions in the reference's vectors) into one
// sequence in that order, so every target receives its contributions in exactly the order the
// reference's scatter loop adds them (particle.cpp:498-658), from 0, with the reference's weight
// expressions:
//   trilinear (concentration weights, or weights * RHS_T): nodes t + {0,1}^3; offset o = node - t
//     selects the factor (o ? 1 - x_l : x_l) per dimension, combined as ((fx*fy)*fz)[*val], the
//     operand order of every term in particle.cpp:548-555 and :645-652;
//   faces (particle.cpp:498-524): x-face t receives x_l RHS_u from particles whose trunc cell
//     (ghosted) is (ti-1, tj, tk) and (1-x_l) RHS_u from those in (ti, tj, tk); cell = node - h.
// 32 particles at a time: the merge (every lane holds the heads of up to five segments, a warp
// minimum picks the next), then a lane per particle forms all its contributions, then the lanes
// take theirs one particle after the other -- one FP64 addition per particle and no
// divergence, whatever the density. (A thread per target with its own merge of 8 or 12 segments,
// forming each weight where it is added, ran at the pace of the slowest lane: 90^3 cells x 400,000
// particles in 64 blobs, a stage: 2.8 ms for C and the faces, 1.03 ms for the temperature; this
// way 0.42 and 0.18 ms; with an addition per target array instead of one for all 0.70 ms.)
constexpr int kOrdWarps = 4;
struct OrdRec {
  // trilinear contributions by offset (x 1, y 2, z 4); faces, per dimension: (1 - x_l) r at the
  // cell, x_l r at the next
  double v[14];
};
template <bool FACES>
__global__ void __launch_bounds__(32 * kOrdWarps) k_dep_ordered(Geom G, DepIn d, int with_val,
                                                                double *__restrict__ out_tri,
                                                                double *__restrict__ out_x,
                                                                double *__restrict__ out_y,
                                                                double *__restrict__ out_z) {
  __shared__ OrdRec recs[kOrdWarps][32];
  __shared__ int2 meta[kOrdWarps][32];  // node and cell relative to the block's first target: x + 256 y + 65536 z
  constexpr int LO = FACES ? 1 : 0;     // nodes [b - LO, b + 4] x [b - LO, b + 4] x [b - LO, b + 2]
  constexpr int RX = 5 + LO, RZ = 3 + LO, R = RX * RX * RZ, SEG = (R + 31) / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  OrdRec *rec = recs[wid];
  int2 *mt = meta[wid];
  const int nbx = (G.g[0] + 3) / 4, nby = (G.g[1] + 3) / 4, nbz = (G.g[2] + 1) / 2;
  const int block = (int)blockIdx.x * kOrdWarps + wid;
  if (block >= nbx * nby * nbz) return;  // whole warps
  const int b0 = (block % nbx) * 4, b1 = ((block / nbx) % nby) * 4, b2 = (block / (nbx * nby)) * 2;
  const int tx = lane & 3, ty = (lane >> 2) & 3, tz = lane >> 4;
  // A particle adds to the 2 x 2 x 2 targets at its node and below, and per dimension to the cell
  // and the next face; the lane's x, y and z faces are those two columns, rows or both away, so
  // that the fourteen targets lie in different lanes and one addition serves them all.
  const int target = tx + ty * 256 + tz * 65536, target_x = target ^ 0x200, target_y = target ^ 2,
            target_z = target ^ 0x202;
  int32_t cur[SEG], end[SEG], key[SEG];
#pragma unroll
  for (int q = 0; q < SEG; ++q) {
    const int r = q * 32 + lane;
    const int ni = b0 - LO + r % RX, nj = b1 - LO + (r / RX) % RX, nk = b2 - LO + r / (RX * RX);
    cur[q] = end[q] = 0;
    if (r < R && node_ok(G, ni, nj, nk)) {
      const long long n = glin(G, ni, nj, nk);
      cur[q] = d.cell_start[n];
      end[q] = d.cell_start[n + 1];
    }
    key[q] = cur[q] < end[q] ? d.okey[cur[q]] : INT32_MAX;
  }
  double acc = 0.0, ax = 0.0, ay = 0.0, az = 0.0;
  int n;
  do {
    int32_t mine = 0;
    for (n = 0; n < 32; ++n) {
      int32_t m = key[0];
#pragma unroll
      for (int q = 1; q < SEG; ++q) m = min(m, key[q]);
      const int32_t least = __reduce_min_sync(0xffffffffu, m);
      if (least == INT32_MAX) break;
      int32_t pos = 0;
      if (m == least) {  // one lane: positions are distinct
#pragma unroll
        for (int q = 0; q < SEG; ++q)
          if (key[q] == least) {
            pos = cur[q]++;
            key[q] = cur[q] < end[q] ? d.okey[cur[q]] : INT32_MAX;
          }
      }
      pos = __shfl_sync(0xffffffffu, pos, __ffs(__ballot_sync(0xffffffffu, m == least)) - 1);
      if (lane == n) mine = pos;
    }
    if (lane < n) {
      const int32_t p = pidx(d, mine);
      const uint32_t k = d.key[p];
      const uint32_t lin = k >> 3, row = lin / (uint32_t)G.g[0], lev = row / (uint32_t)G.g[1];
      const int hx = (int)((k >> 2) & 1u), hy = (int)((k >> 1) & 1u), hz = (int)(k & 1u);
      const int nx = (int)(lin - row * (uint32_t)G.g[0]) - b0, ny = (int)(row - lev * (uint32_t)G.g[1]) - b1,
                nz = (int)lev - b2;
      const double f0 = d.frac[0][p], f1 = d.frac[1][p], f2 = d.frac[2][p];
      const double xl = xl_round(f0, hx), yl = xl_round(f1, hy), zl = xl_round(f2, hz);
      const double fx[2] = {xl, 1 - xl}, fy[2] = {yl, 1 - yl}, fz[2] = {zl, 1 - zl};
      const double v = with_val ? d.val[0][p] : 0.0;
      OrdRec &r = rec[lane];
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        const double w = fx[o & 1] * fy[(o >> 1) & 1] * fz[o >> 2];
        r.v[o] = with_val ? w * v : w;
      }
      if (FACES) {
        const double fr[3] = {f0, f1, f2};
#pragma unroll
        for (int D = 0; D < 3; ++D) {
          const double u = d.val[D][p];
          r.v[8 + 2 * D] = (1 - fr[D]) * u;
          r.v[9 + 2 * D] = fr[D] * u;
        }
      }
      mt[lane] = make_int2(nx + ny * 256 + nz * 65536, nx - hx + (ny - hy) * 256 + (nz - hz) * 65536);
    }
    __syncwarp();
    for (int i = 0; i < n; ++i) {
      const int2 mm = mt[i];
      const int qt = mm.x - target;  // offsets 0 or 1, or a bit above them is set
      const bool it = !(qt & ~0x10101);
      if (!FACES) {
        if (it) acc += rec[i].v[(qt | qt >> 7 | qt >> 14) & 7];
      } else {
        // at most one of the lane's four targets takes from a particle
        const int qx = target_x - mm.y, qy = target_y - mm.y, qz = target_z - mm.y;  // target - cell
        const bool ix = !(qx & ~1), iy = !(qy & ~0x100), iz = !(qz & ~0x10000);
        const int at = it ? (qt | qt >> 7 | qt >> 14) & 7 : ix ? 8 + qx : iy ? 10 + (qy >> 8) : iz ? 12 + (qz >> 16) : 0;
        const double sum = (ix ? ax : iy ? ay : iz ? az : acc) + rec[i].v[at];
        if (it) acc = sum;
        if (ix) ax = sum;
        if (iy) ay = sum;
        if (iz) az = sum;
      }
    }
    __syncwarp();
  } while (n == 32);
  auto put = [&](double *__restrict__ out, int dx, int dy, double v) {
    const int ti = b0 + (tx ^ dx), tj = b1 + (ty ^ dy), tk = b2 + tz;
    if (ti < G.g[0] && tj < G.g[1] && tk < G.g[2]) out[glin(G, ti, tj, tk)] = v;
  };
  put(out_tri, 0, 0, acc);
  if (d.keep && b0 + tx < G.g[0] && b1 + ty < G.g[1] && b2 + tz < G.g[2]) {
    const long long t = glin(G, b0 + tx, b1 + ty, b2 + tz);
    d.keep[t] = d.kept[t];
  }
  if (FACES) {
    put(out_x, 0, 2, ax);
    put(out_y, 2, 0, ay);
    put(out_z, 2, 2, az);
  }
}

// ---- fast path ----------------------------------------------------------------
constexpr int kB = 8;                 // brick edge (target cells)
constexpr int kB1 = kB + 1;           // trilinear node region edge [b, b+B]; trunc cells [b-1, b+B-1]
constexpr int kB2 = kB + 2;           // face node region edge [b-1, b+B]
constexpr int kNodes = kB1 * kB1 * kB1, kRegion = kB2 * kB2 * kB2;
constexpr int kBrickThreads = 384;
// Lists longer than this are summed by a warp: lanes stride the particles in order and a
// fixed shuffle tree adds the lane sums. The order is fixed by the list alone, so the result
// is the same from run to run; one thread walking a blob-centre node (~1000 particles) would
// hold up its whole brick.
// The line: a warp pays ceil(n / 32) rounds and a reduction, 32 threads with lists alike n rounds
// for 32 lists; beside each other at 2^24 particles in 64 blobs: node lists up to 24, 32, 64, 128
// by threads 2.06, 2.05, 1.86, 1.83 ms (temperature deposit), cell lists, which gather from
// eight runs, 4.28, 4.13, 4.50, 4.77 ms (with the trilinear part). Nodes stop at 32 all the same: a chain of
// 64 additions rounds more than lane sums and a tree (error of RHS_Part_Temp 6.95e-16 -> 7.25e-16).
constexpr int kDenseNode = 32, kDenseCell = 32;
constexpr int kBins = kDenseNode + 2;  // list lengths 0 .. 64, and longer

// The warp's sums of m[0..7] in a fixed order; each round a lane hands over the half of its values
// that its partner goes on with: 9 FP64 additions instead of 40. Lane l ends with the sum of
// m[(l >> 2) & 7 as bits 4, 3, 2], the same in the four lanes of a value.
__device__ __forceinline__ double warp_sums8(const double (&m)[8], int lane) {
  double a[4];
  bool up = lane & 16;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double got = __shfl_xor_sync(0xffffffffu, up ? m[i] : m[i + 4], 16);
    a[i] = (up ? m[i + 4] : m[i]) + got;
  }
  up = lane & 8;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double got = __shfl_xor_sync(0xffffffffu, up ? a[i] : a[i + 2], 8);
    a[i] = (up ? a[i + 2] : a[i]) + got;
  }
  up = lane & 4;
  const double got = __shfl_xor_sync(0xffffffffu, up ? a[0] : a[1], 4);
  double v = (up ? a[1] : a[0]) + got;
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v + __shfl_xor_sync(0xffffffffu, v, 1);
}

// The fast deposit sums moments per node instead of the 8 corner weights: with
// t = (x_l, y_l, z_l) of each particle and value v (1 for the concentration),
// M[s] = sum v * prod_{d in s} t_d for the 8 subsets s of {x (4), y (2), z (1)}.
// The corner with (1 - t_d) in the dimensions of bit set o and t_d in the others is
// sum_{A subset of o} (-1)^|A| M[A | ~o], formed once per node.
// GB300's FP64 pipe (two lanes per SM and clock) is the bound of this kernel, and per particle
// this takes 3 + 4 + 8 FP64 operations instead of 6 + 3 + 24 (+ 8). x_l = frac + 0.5 - h is formed as
// frac + (h ? -0.5 : 0.5), the same value (frac - 1 and frac - 0.5 are exact for
// frac >= 0.5).
template <int MODE> struct TriRec {
  uint32_t key;
  double f[3], v;
};
template <int MODE>
__device__ __forceinline__ TriRec<MODE> tri_load(const DepIn &d, int32_t p) {
  TriRec<MODE> r;
  r.key = d.key[p];
#pragma unroll
  for (int D = 0; D < 3; ++D) r.f[D] = d.frac[D][p];
  r.v = MODE ? d.val[0][p] : 0.0;
  return r;
}
template <int MODE>
__device__ __forceinline__ void moments_add(double (&m)[8], const TriRec<MODE> &r) {
  const uint32_t key = r.key;
  const double v = r.v;
  const double xl = r.f[0] + ((key & 4u) ? -0.5 : 0.5);
  const double yl = r.f[1] + ((key & 2u) ? -0.5 : 0.5);
  const double zl = r.f[2] + ((key & 1u) ? -0.5 : 0.5);
  const double xy = xl * yl, xz = xl * zl, yz = yl * zl, xyz = xy * zl;
  if (MODE) {
    m[0] += v;
    m[4] = fma(xl, v, m[4]);
    m[2] = fma(yl, v, m[2]);
    m[1] = fma(zl, v, m[1]);
    m[6] = fma(xy, v, m[6]);
    m[5] = fma(xz, v, m[5]);
    m[3] = fma(yz, v, m[3]);
    m[7] = fma(xyz, v, m[7]);
  } else {  // m[0], the particle count, is set by the caller
    m[4] += xl;
    m[2] += yl;
    m[1] += zl;
    m[6] += xy;
    m[5] += xz;
    m[3] += yz;
    m[7] += xyz;
  }
}

// moments -> corner partials in place (index bit 2: x takes 1 - x_l, bit 1: y, bit 0: z), the terms of the sum
// above one after the other (a dimension at a time takes 12 additions instead of 19 and rounds more: the
// error of C in a box of 64^3 cells and 2^15 particles 1.425e-16 -> 1.445e-16)
__device__ __forceinline__ void corners_of(double (&m)[8]) {
  double c[8];
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    const int rest = ~o & 7;
    c[o] = m[rest];
#pragma unroll
    for (int a = 1; a < 8; ++a)
      if ((a & o) == a) c[o] = (__popc(a) & 1) ? c[o] - m[a | rest] : c[o] + m[a | rest];
  }
#pragma unroll
  for (int o = 0; o < 8; ++o) m[o] = c[o];
}

// face sums: (sum (1 - t) r, sum t r) per dimension, t the in-cell fraction and r the RHS_u component; the first
// one's terms are rounded once each (as sum r - sum t r a cell of two particles lost a bit)
struct FaceRec {
  double f[3], r[3];
};
__device__ __forceinline__ FaceRec face_load(const DepIn &d, int32_t p) {
  FaceRec q;
#pragma unroll
  for (int D = 0; D < 3; ++D) {
    q.f[D] = d.frac[D][p];
    q.r[D] = d.val[D][p];
  }
  return q;
}
__device__ __forceinline__ void face_add(double (&f)[6], const FaceRec &q) {
#pragma unroll
  for (int D = 0; D < 3; ++D) {
    f[2 * D] += fma(-q.f[D], q.r[D], q.r[D]);
    f[2 * D + 1] = fma(q.f[D], q.r[D], f[2 * D + 1]);
  }
}

__device__ inline int32_t seg_lower_h(const DepIn &d, int32_t a, int32_t b, uint32_t hcls) {
  // first position in [a, b) whose particle has h class >= hcls (segments are sorted by h)
  while (a < b) {
    int32_t m = (a + b) >> 1;
    if ((d.key[pidx(d, m)] & 7u) < hcls) a = m + 1; else b = m;
  }
  return a;
}

// Shared memory of a brick's CTA: the partials (trilinear first, then the faces in the same
// place), slot-major so that neighbouring slots fall on neighbouring banks.
constexpr int kTabulated = 255;
template <int MODE> struct BrickSmem {
  static constexpr int kTable = MODE ? 1 : kRegion;  // the faces' tables are the int deposit's
  union {
    double tri[8][kNodes];    // corner partials of node b + l
    double face[6][kNodes];   // face partials of trunc cell b - 1 + l
  };
  uint8_t cls_end[kTable][8];  // node b - 1 + l: ends of the h classes 0..7 (at most kTabulated particles)
  int32_t start[kRegion];      // node b - 1 + l: first sorted position
  int32_t count[kRegion];      // its particles
  uint16_t length[kNodes];     // list length of an item (clamped); faces: | non-empty h classes << 8
  uint16_t order[kNodes];      // items by list length
  int32_t bin[kBins];
  int32_t n_dense, n_empty, next;
};

// Items 0 .. kNodes - 1 by their list length (sm.length's low byte), ascending, into sm.order; the
// order inside a length is left to the atomics, since every item is summed by itself. A thread
// walks one item's list and the FP64 pipe is charged per warp instruction: lists of like
// length side by side let a warp's lanes end together (in storage order a warp ran the longest
// of 32 lists with about a quarter of its lanes live).
template <int DENSE, int MODE>
__device__ __forceinline__ void order_by_length(BrickSmem<MODE> &sm) {
  const int lane = (int)(threadIdx.x & 31u);
  for (int q = threadIdx.x; q < kBins; q += blockDim.x) sm.bin[q] = 0;
  __syncthreads();
  // a few lengths hold most items: one add per distinct length of a warp
  for (int s0 = threadIdx.x - lane; s0 < kNodes; s0 += blockDim.x) {
    const int s = s0 + lane;
    const int b = s < kNodes ? sm.length[s] & 255 : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    if (b >= 0 && lane == __ffs(peers) - 1) atomicAdd(&sm.bin[b], __popc(peers));
  }
  __syncthreads();
  if (threadIdx.x < 32) {  // exclusive scan of the bins
    int carry = 0;
    for (int b0 = 0; b0 < kBins; b0 += 32) {
      const int b = b0 + lane;
      const int v = b < kBins ? sm.bin[b] : 0;
      int x = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (b < kBins) sm.bin[b] = carry + x - v;
      if (b == 0) sm.n_empty = v;
      if (b == DENSE + 1) sm.n_dense = v;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) sm.next = 0;
  }
  __syncthreads();
  for (int s0 = threadIdx.x - lane; s0 < kNodes; s0 += blockDim.x) {
    const int s = s0 + lane;
    const int b = s < kNodes ? sm.length[s] & 255 : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    const int leader = __ffs(peers) - 1;
    int at = 0;
    if (b >= 0 && lane == leader) at = atomicAdd(&sm.bin[b], __popc(peers));
    at = __shfl_sync(0xffffffffu, at, leader);
    if (b >= 0) sm.order[at + __popc(peers & ((1u << lane) - 1u))] = (uint16_t)s;
  }
  __syncthreads();
}

// The ordered items in units: one dense item for a whole warp, or up to 32 others, a lane each;
// warps take the longest lists first. dense(s) is called by all lanes, light(s) by single ones
// (every item but the empty ones).
template <int MODE, typename Dense, typename Light>
__device__ __forceinline__ void take_items(BrickSmem<MODE> &sm, Dense dense, Light light) {
  const int lane = (int)(threadIdx.x & 31u);
  const int nd = sm.n_dense, nl = kNodes - nd - sm.n_empty, units = nd + (nl + 31) / 32;
  while (true) {
    int u = 0;
    if (lane == 0) u = atomicAdd(&sm.next, 1);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= units) break;
    if (u < nd) {
      dense((int)sm.order[kNodes - 1 - u]);
    } else {
      const int w = kNodes - nd - 1 - ((u - nd) * 32 + lane);
      if (w >= sm.n_empty) light((int)sm.order[w]);
    }
    __syncwarp();
  }
}

// mode 0: concentration (weights) + face momentum partials at x_int; mode 1: weights * RHS_T.
//
// Trilinear: one item per node of [b, b+B], its moments summed over the node's segment. Faces:
// one item per trunc cell of [b-1, b+B-1]; its particles are, for each h class, that class's
// run in node c + h's segment (the runs in class order, the empty ones skipped by a mask), so
// all of a cell's particles are summed by one thread. Bound: the FP64 pipe; per particle 14 (15
// in mode 1) operations for the trilinear sums and 9 for the faces, 19 + 7 a node and target,
// 6 + 3 a cell and target. The pipe answers through a queue (short scoreboard), so a brick's
// phases stay latency-bound between barriers (three CTAs per SM). 256^3 cells x 2^24 particles in
// 64 blobs: 4.2 and 2.0 ms. (Node lists to 64, corners a dimension at a time, faces as sum r - sum x_l r:
// 4.4 and 1.7, of the first 1.9 the trilinear part, 0.8 the class table and order of the cells, 1.7 the face
// sums. A thread per node in storage order, the faces in eight h-class phases over all nodes: 15 and 5 ms.)
template <int MODE>
__global__ void __launch_bounds__(kBrickThreads, 3) k_dep_brick(Geom G, DepIn d, int twc,
                                                             double *__restrict__ out_tri,
                                                             double *__restrict__ out_x,
                                                             double *__restrict__ out_y,
                                                             double *__restrict__ out_z) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BrickSmem<MODE> &sm = *reinterpret_cast<BrickSmem<MODE> *>(smem_raw);
  const int nbx = (G.g[0] + kB - 1) / kB, nby = (G.g[1] + kB - 1) / kB;
  const int bx = (int)(blockIdx.x % nbx) * kB;
  const int by = (int)((blockIdx.x / nbx) % nby) * kB;
  const int bz = (int)(blockIdx.x / ((long long)nbx * nby)) * kB;
  const int lane = (int)(threadIdx.x & 31u);
  const bool faces = MODE == 0 && twc;

  // segment table of the region's nodes [b-1, b+B]
  for (int s = threadIdx.x; s < kRegion; s += blockDim.x) {
    const int lx = s % kB2, ly = (s / kB2) % kB2, lz = s / (kB2 * kB2);
    const int ni = bx - 1 + lx, nj = by - 1 + ly, nk = bz - 1 + lz;
    int32_t a0 = 0, cnt = 0;
    if (node_ok(G, ni, nj, nk)) {
      const long long n = glin(G, ni, nj, nk);
      a0 = d.cell_start[n];
      cnt = d.cell_start[n + 1] - a0;
    }
    if (faces) {
      uint64_t ends = 0;
      if (cnt <= 16) {
        uint64_t c = 0;  // 8 one-byte class counts, then their running sums (at most 16)
        for (int32_t q = 0; q < cnt; ++q) c += 1ull << (8u * (d.key[pidx(d, a0 + q)] & 7u));
        ends = c * 0x0101010101010101ull;
      } else if (cnt <= kTabulated) {
#pragma unroll 1
        for (int hc = 0; hc < 7; ++hc)
          ends |= (uint64_t)(seg_lower_h(d, a0, a0 + cnt, hc + 1) - a0) << (8 * hc);
        ends |= (uint64_t)cnt << 56;
      }
      *reinterpret_cast<uint64_t *>(sm.cls_end[MODE ? 0 : s]) = ends;
    }
    sm.start[s] = a0;
    sm.count[s] = cnt;
    // the trilinear item of a node in [b, b+B]
    if (lx && ly && lz)
      sm.length[((lz - 1) * kB1 + (ly - 1)) * kB1 + (lx - 1)] = (uint16_t)min(cnt, kDenseNode + 1);
  }
  for (int s = threadIdx.x; s < 8 * kNodes; s += blockDim.x) sm.tri[0][s] = 0.0;
  __syncthreads();

  // ---- trilinear: node items (slot l in [0, B]^3, region slot l + 1)
  order_by_length<kDenseNode>(sm);
  auto region_of = [](int s) {
    const int lx = s % kB1, ly = (s / kB1) % kB1, lz = s / (kB1 * kB1);
    return ((lz + 1) * kB2 + (ly + 1)) * kB2 + (lx + 1);
  };
  take_items(
      sm,
      [&](int s) {
        const int rs = region_of(s);
        const int32_t a = sm.start[rs], cnt = sm.count[rs];
        double m[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) m[o] = 0.0;
        for (int32_t q = a + lane; q < a + cnt; q += 32) moments_add<MODE>(m, tri_load<MODE>(d, pidx(d, q)));
        // the moments as they are; their corners below, a lane per node
        const double v = warp_sums8(m, lane);
        if (!(lane & 3)) sm.tri[lane >> 2][s] = !MODE && lane == 0 ? (double)cnt : v;
      },
      [&](int s) {
        const int rs = region_of(s);
        const int32_t a = sm.start[rs], cnt = sm.count[rs];
        double m[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) m[o] = 0.0;
        // a list's loads ahead of its sums: the index two particles ahead, the record one
        int32_t ahead = cnt > 1 ? pidx(d, a + 1) : 0;
        TriRec<MODE> rec = tri_load<MODE>(d, pidx(d, a));
        for (int32_t q = a + 1; q < a + cnt; ++q) {
          const TriRec<MODE> next = tri_load<MODE>(d, ahead);
          if (q + 1 < a + cnt) ahead = pidx(d, q + 1);
          moments_add<MODE>(m, rec);
          rec = next;
        }
        moments_add<MODE>(m, rec);
        if (!MODE) m[0] = (double)cnt;
        corners_of(m);
#pragma unroll
        for (int o = 0; o < 8; ++o) sm.tri[o][s] = m[o];
      });
  __syncthreads();
  for (int w = threadIdx.x; w < sm.n_dense; w += blockDim.x) {
    const int s = sm.order[kNodes - 1 - w];
    double m[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) m[o] = sm.tri[o][s];
    corners_of(m);
#pragma unroll
    for (int o = 0; o < 8; ++o) sm.tri[o][s] = m[o];
  }
  __syncthreads();
  // h classes and length of every cell item (slot l in [0, B]^3: cell b - 1 + l; its class-h run
  // is in the segment of region slot l + h)
  auto node_of = [](int base, int hc) { return base + ((hc & 1) * kB2 + ((hc >> 1) & 1)) * kB2 + ((hc >> 2) & 1); };
  auto run = [&](int rs, int hc, int32_t &a, int32_t &e) {
    const int32_t a0 = sm.start[rs], cnt = sm.count[rs];
    if (cnt <= kTabulated) {
      a = a0 + (hc ? sm.cls_end[MODE ? 0 : rs][hc - 1] : 0);
      e = a0 + sm.cls_end[MODE ? 0 : rs][hc];
    } else {  // a segment longer than the table holds
      a = hc ? seg_lower_h(d, a0, a0 + cnt, hc) : a0;
      e = hc < 7 ? seg_lower_h(d, a, a0 + cnt, hc + 1) : a0 + cnt;
    }
  };
  if (faces) {
    for (int s = threadIdx.x; s < kNodes; s += blockDim.x) {
      const int base = ((s / (kB1 * kB1)) * kB2 + (s / kB1) % kB1) * kB2 + s % kB1;
      int n = 0, classes = 0;
#pragma unroll
      for (int hc = 0; hc < 8; ++hc) {
        int32_t a, e;
        run(node_of(base, hc), hc, a, e);
        n += e - a;
        classes |= e > a ? 1 << hc : 0;
      }
      sm.length[s] = (uint16_t)(min(n, kDenseCell + 1) | classes << 8);
    }
  }
  for (int s = threadIdx.x; s < kB * kB * kB; s += blockDim.x) {
    const int lx = s % kB, ly = (s / kB) % kB, lz = s / (kB * kB);
    const int ti = bx + lx, tj = by + ly, tk = bz + lz;
    if (ti >= G.g[0] || tj >= G.g[1] || tk >= G.g[2]) continue;
    const long long t = glin(G, ti, tj, tk);
    const double kept = !MODE && d.keep ? __ldcs(d.kept + t) : 0.0;
    double acc = 0.0;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const int ox = (o >> 2) & 1, oy = (o >> 1) & 1, oz = o & 1;
      const double v = sm.tri[o][((lz + oz) * kB1 + (ly + oy)) * kB1 + (lx + ox)];
      acc = o ? acc + v : v;
    }
    out_tri[t] = acc;
    if (!MODE && d.keep) __stcs(d.keep + t, kept);
  }
  if (!faces) return;
  __syncthreads();

  // ---- faces
  for (int s = threadIdx.x; s < 6 * kNodes; s += blockDim.x) sm.face[0][s] = 0.0;
  order_by_length<kDenseCell>(sm);
  take_items(
      sm,
      [&](int s) {
        const int base = ((s / (kB1 * kB1)) * kB2 + (s / kB1) % kB1) * kB2 + s % kB1;
        double fs[6] = {0, 0, 0, 0, 0, 0};
        for (int classes = sm.length[s] >> 8; classes; classes &= classes - 1) {
          const int hc = __ffs(classes) - 1;
          int32_t a, e;
          run(node_of(base, hc), hc, a, e);
          for (int32_t q = a + lane; q < e; q += 32) face_add(fs, face_load(d, pidx(d, q)));
        }
        const double m[8] = {fs[0], fs[1], fs[2], fs[3], fs[4], fs[5], 0.0, 0.0};
        const double v = warp_sums8(m, lane);  // lanes 0, 4, .. 20: fs[0..5]
        if (!(lane & 3) && lane < 24) sm.face[lane >> 2][s] = v;
      },
      [&](int s) {
        const int base = ((s / (kB1 * kB1)) * kB2 + (s / kB1) % kB1) * kB2 + s % kB1;
        double fs[6] = {0, 0, 0, 0, 0, 0};
        // the cell's particles one after the other, run by run; the next one's loads ahead
        int classes = sm.length[s] >> 8;
        int32_t q = 0, e = 0;
        auto next = [&]() -> int32_t {  // -1 at the end
          if (q == e) {
            if (!classes) return -1;
            const int hc = __ffs(classes) - 1;
            classes &= classes - 1;
            run(node_of(base, hc), hc, q, e);
          }
          return pidx(d, q++);
        };
        double fb[6] = {0, 0, 0, 0, 0, 0};  // every other particle's
        int32_t ahead = next();
        FaceRec rec = face_load(d, ahead);
        ahead = next();
        while (ahead >= 0) {
          const FaceRec other = face_load(d, ahead);
          ahead = next();
          face_add(fs, rec);
          if (ahead < 0) {
            rec = other;
            break;
          }
          rec = face_load(d, ahead);
          ahead = next();
          face_add(fb, other);
        }
        face_add(fb, rec);
#pragma unroll
        for (int q = 0; q < 6; ++q) sm.face[q][s] = fs[q] + fb[q];
      });
  __syncthreads();
  for (int s = threadIdx.x; s < kB * kB * kB; s += blockDim.x) {
    const int lx = s % kB, ly = (s / kB) % kB, lz = s / (kB * kB);
    const int ti = bx + lx, tj = by + ly, tk = bz + lz;
    if (ti >= G.g[0] || tj >= G.g[1] || tk >= G.g[2]) continue;
    const long long t = glin(G, ti, tj, tk);
    // cell slot of target cell t is l + 1; its lower neighbour in dimension D is l
    const int c = ((lz + 1) * kB1 + (ly + 1)) * kB1 + (lx + 1);
    out_x[t] = sm.face[1][c - 1] + sm.face[0][c];
    out_y[t] = sm.face[3][c - kB1] + sm.face[2][c];
    out_z[t] = sm.face[5][c - kB1 * kB1] + sm.face[4][c];
  }
}

// The cumulative ghost fold (communicator.cpp:422-511 on one rank: z, then y, then x, every layer
// added to its image), the ghost refresh (communicator.cpp:177-278) and the interior sum of up to
// four fields in one launch. A boundary cell's up to seven ghost images belong to no other cell, so
// its thread reads them all, adds them in the order of the three passes and leaves in them what
// the passes leave: fields before `first` keep the partly folded ghosts, the others take the
// refreshed value and are summed over their interior, in an order fixed by the grid alone: a warp a
// row (j, k), the rows over the warps, a tree over the block; the launch's last block adds the blocks.
// Passes, refresh and sums as launches of their own, each a few microseconds of work and a gap, took
// 91 us for the temperature and 205 for C and the momentum at 256^3 cells (and 5 launches each); this
// 73 and 179 us.
struct FieldSet {
  double *f[4];
  int first;
};
constexpr int kRedBlocks = 1024;

__device__ inline double fold_cell(const Geom &G, double *f, int i, int j, int k, bool whole) {
  const bool bx = i == 1 || i == G.n[0], by = j == 1 || j == G.n[1], bz = k == 1 || k == G.n[2];
  const int x[2] = {i, i == 1 ? G.n[0] + 1 : 0}, y[2] = {j, j == 1 ? G.n[1] + 1 : 0}, z[2] = {k, k == 1 ? G.n[2] + 1 : 0};
  double v[8];
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    const bool in = (!(o & 4) || bx) && (!(o & 2) || by) && (!(o & 1) || bz);
    v[o] = in ? f[glin(G, x[o >> 2], y[(o >> 1) & 1], z[o & 1])] : 0.0;
  }
#pragma unroll
  for (int o = 0; o < 8; o += 2)
    if (bz) v[o] += v[o + 1];
  const double z1 = v[2], z3 = v[6];
  if (by) {
    v[0] += v[2];
    v[4] += v[6];
  }
  const double y1 = v[4];
  if (bx) v[0] += v[4];
  const double all = v[0];
  f[glin(G, i, j, k)] = all;
  if (whole) {
#pragma unroll
    for (int o = 1; o < 8; ++o)
      if ((!(o & 4) || bx) && (!(o & 2) || by) && (!(o & 1) || bz))
        f[glin(G, x[o >> 2], y[(o >> 1) & 1], z[o & 1])] = all;
  } else {
    if (by) f[glin(G, i, y[1], k)] = z1;
    if (bx) f[glin(G, x[1], j, k)] = y1;
    if (bx && by) f[glin(G, x[1], y[1], k)] = z3;
  }
  return all;
}

__global__ void __launch_bounds__(kThreads, 6) k_fold(Geom G, FieldSet fs, double scale, double *__restrict__ parts,
                                                   unsigned *__restrict__ tickets, double *__restrict__ out) {
  __shared__ double sm[kThreads / 32];
  __shared__ bool last;
  const bool whole = (int)blockIdx.y >= fs.first;
  double *f = blockIdx.y < 2 ? (blockIdx.y ? fs.f[1] : fs.f[0]) : (blockIdx.y == 2 ? fs.f[2] : fs.f[3]);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, n0 = G.n[0];
  const int rows = G.n[1] * G.n[2];
  double s = 0.0;
  // boundary rows take several times longer: the rows turn over the warps, or a warp would have one at
  // every step where the number of warps is a multiple of n1
  const int warps = (int)gridDim.x * (kThreads / 32);
  int turn = (int)blockIdx.x * (kThreads / 32) + wid;
  for (int first = 0; first < rows; first += warps, turn = turn + 37 < warps ? turn + 37 : (turn + 37) % warps) {
    const int r = first + turn;
    if (r >= rows) continue;
    const int k = r / G.n[1] + 1, j = r - (k - 1) * G.n[1] + 1;
    if (j == 1 || j == G.n[1] || k == 1 || k == G.n[2]) {
      for (int i = lane + 1; i <= n0; i += 32) s += fold_cell(G, f, i, j, k, whole);
      continue;
    }
    double *row = f + glin(G, 0, j, k);
    // folded along x alone: lanes 0 and 1 the two ends
    const int end = lane ? n0 : 1, ghost = lane ? 0 : n0 + 1;
    double e = 0.0, g = 0.0;
    if (lane < 2) {
      e = row[end];
      g = row[ghost];
    }
    if (whole) {
      // four pieces of 32 cells at a time, their loads before the sums
      for (int i0 = lane + 1; i0 - lane <= n0; i0 += 128) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + 32 * u;
          v[u] = i > 1 && i < n0 ? row[i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i0 - lane + 32 * u <= n0) s += v[u];
      }
    }
    if (lane < 2) {
      e += g;
      row[end] = e;
      if (whole) {
        row[ghost] = e;
        s += e;
      }
    }
  }
  if (!whole) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) sm[wid] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < kThreads / 32; ++q) s += sm[q];
    parts[blockIdx.y * kRedBlocks + blockIdx.x] = s;
    __threadfence();
    last = atomicInc(&tickets[blockIdx.y], gridDim.x - 1) == gridDim.x - 1;  // back to 0 with the last
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const double *p = parts + blockIdx.y * kRedBlocks;
  s = 0.0;
  for (int q = threadIdx.x; q < (int)gridDim.x; q += kThreads) s += __ldcg(p + q);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) sm[wid] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < kThreads / 32; ++q) s += sm[q];
    out[(int)blockIdx.y - fs.first] = s * scale;
  }
}

inline int blocks_for(long long n) { return (int)((n + kThreads - 1) / kThreads); }

DepIn make_in(pstep_ctx *h, const Csr &csr, double *const frac[3], const uint32_t *key, const double *v0,
              const double *v1, const double *v2) {
  DepIn d;
  d.cell_start = csr.cell_start;
  d.sidx = csr.identity ? nullptr : csr.sidx;
  d.okey = csr.identity ? h->ref_of_phys : csr.okey;
  for (int q = 0; q < 3; ++q) d.frac[q] = frac[q];
  d.key = key;
  d.val[0] = v0;
  d.val[1] = v1;
  d.val[2] = v2;
  d.kept = nullptr;
  d.keep = nullptr;
  return d;
}

}  // namespace

// folds f[0 .. nf); refreshes f[first .. nf) and leaves scale x their interior sums in out
int fold_fields(pstep_ctx *h, double *const *f, int nf, int first, double scale, double *out) {
  const Geom &G = h->geom;
  FieldSet fs;
  fs.first = first;
  for (int q = 0; q < nf; ++q) fs.f[q] = f[q];
  const long long rows = (long long)G.n[1] * G.n[2], blocks = (rows + kThreads / 32 - 1) / (kThreads / 32);
  k_fold<<<dim3((unsigned)(blocks < kRedBlocks ? blocks : kRedBlocks), nf), kThreads, 0, h->stream>>>(
      G, fs, scale, h->red_partials, h->red_tickets, out);
  PSTEP_LAUNCHED(h);
  return PSTEP_OK;
}

// C and, with TWC, the momentum fields and their balance (the interior sums); without, RHS_RU = 0
// (grid.cpp:671)
int fold_int(pstep_ctx *h) {
  // (the reference does not refresh C's ghosts)
  double *all[4] = {h->dep[PSTEP_FIELD_C], h->dep[PSTEP_FIELD_RU_X], h->dep[PSTEP_FIELD_RU_Y], h->dep[PSTEP_FIELD_RU_Z]};
  const int rc = fold_fields(h, all, h->cfg.twc ? 4 : 1, 1, 1.0, h->mom_dev);
  if (rc || h->cfg.twc) return rc;
  for (int q = 1; q < 4; ++q) PSTEP_CUDA(cudaMemsetAsync(all[q], 0, sizeof(double) * h->geom.gsize, h->stream));
  PSTEP_CUDA(cudaMemsetAsync(h->mom_dev, 0, 3 * sizeof(double), h->stream));
  return PSTEP_OK;
}

// part2gas_Temp_int/new: deposit RHS_T with the records of csr/frac/key, fold, refresh, mean.
bool reference_sums(const pstep_ctx *h) {
  return (h->cfg.flags & PSTEP_TRACK_ORDER) && (h->cfg.flags & PSTEP_REFERENCE_SUMS);
}

int ordered_launch(pstep_ctx *h, const DepIn &d, bool faces, int with_val, double *tri, double *ox, double *oy,
                   double *oz) {
  const Geom &G = h->geom;
  const long long blocks = (long long)((G.g[0] + 3) / 4) * ((G.g[1] + 3) / 4) * ((G.g[2] + 1) / 2);
  const unsigned grid = (unsigned)((blocks + kOrdWarps - 1) / kOrdWarps);
  auto kern = faces ? k_dep_ordered<true> : k_dep_ordered<false>;
  kern<<<grid, 32 * kOrdWarps, 0, h->stream>>>(G, d, with_val, tri, ox, oy, oz);
  PSTEP_LAUNCHED(h);
  return PSTEP_OK;
}

int brick_launch(pstep_ctx *h, const DepIn &d, int mode, double *tri, double *ox, double *oy, double *oz) {
  const Geom &G = h->geom;
  auto kern = mode ? k_dep_brick<1> : k_dep_brick<0>;
  const size_t smem = mode ? sizeof(BrickSmem<1>) : sizeof(BrickSmem<0>);
  // the opt-in applies to the current device, which is the one this launch uses;
  // setting it at every launch keeps it right for handles on several devices
  PSTEP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const long long nb = (long long)((G.g[0] + kB - 1) / kB) * ((G.g[1] + kB - 1) / kB) * ((G.g[2] + kB - 1) / kB);
  kern<<<(unsigned)nb, kBrickThreads, smem, h->stream>>>(G, d, h->cfg.twc, tri, ox, oy, oz);
  PSTEP_LAUNCHED(h);
  return PSTEP_OK;
}

int deposit_temperature(pstep_ctx *h, const Csr &csr, double *const frac[3], const uint32_t *key) {
  const Geom &G = h->geom;
  DepIn d = make_in(h, csr, frac, key, h->s.rhs_t, nullptr, nullptr);
  double *out = h->dep[PSTEP_FIELD_PART_TEMP];
  if (reference_sums(h)) {
    const int rc = ordered_launch(h, d, false, 1, out, nullptr, nullptr, nullptr);
    if (rc) return rc;
  } else {
    int rc = brick_launch(h, d, 1, out, nullptr, nullptr, nullptr);
    if (rc) return rc;
  }
  double *fl[1] = {out};
  return fold_fields(h, fl, 1, 0, 1.0 / (double)((long long)G.n[0] * G.n[1] * G.n[2]), h->emean_dev);
}

// part2gas_concentration + part2gas_velocity at x_int (records of the previous CSR)
int f64_deposit_int(pstep_ctx *h) {
  DepIn d = make_in(h, h->csr_prev, h->s.frac_prev, h->s.key_prev, h->s.rhs_u[0], h->s.rhs_u[1], h->s.rhs_u[2]);
  if (h->t_pending) {
    d.kept = h->tf;
    d.keep = h->t_kept;
  }
  double *c = h->dep[PSTEP_FIELD_C], *x = h->dep[PSTEP_FIELD_RU_X], *y = h->dep[PSTEP_FIELD_RU_Y],
         *z = h->dep[PSTEP_FIELD_RU_Z];
  const int rc = reference_sums(h) ? ordered_launch(h, d, h->cfg.twc, 0, c, x, y, z) : brick_launch(h, d, 0, c, x, y, z);
  return rc ? rc : fold_int(h);
}

}  // namespace pstep
