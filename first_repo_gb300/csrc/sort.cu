// Deterministic counting sort of particles by node key, giving the CSR that the
// deposit gathers walk (cell_start over the ghosted node grid + sorted particle
// indices), and the per-step reorder of particle storage by that sort.
//
// Order within a node is fixed by an explicit secondary key (the particle's
// position in the reference's vectors, or its storage index), so the CSR -- and
// every sum taken over it -- is identical from run to run.
#include "scan.cuh"

namespace pstep {
namespace {

constexpr int kScanItems = 16;                       // per thread
constexpr int kScanTile = kThreads * kScanItems;     // per block

__global__ void k_count(const uint32_t *__restrict__ keys, int shift, int64_t n, int32_t *__restrict__ counts) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < n;
  const uint32_t node = valid ? (keys[i] >> shift) : 0xffffffffu;
  const Run run = run_of(node);
  if (valid && run.place == 0) atomicAdd(&counts[node], run.len);
}

// the particle's place among those of its key, from the keys' running positions (n: none)
__device__ __forceinline__ int32_t place_of(const uint32_t *__restrict__ keys, int shift, int64_t i, int64_t n,
                                            int32_t *__restrict__ cursor) {
  const bool valid = i < n;
  const uint32_t node = valid ? (keys[i] >> shift) : 0xffffffffu;
  const Run run = run_of(node);
  int32_t base = 0;
  if (valid && run.place == 0) base = atomicAdd(&cursor[node], run.len);
  return __shfl_sync(0xffffffffu, base, run.first) + run.place;
}

__device__ __noinline__ int32_t tile_sum(const int32_t *in, int32_t tile) {
  in += (int64_t)tile * kScanTile;
  int32_t sum = 0;
  for (int i = threadIdx.x & 31; i < kScanTile; i += 32) sum += in[i];
  return (int32_t)__reduce_add_sync(0xffffffffu, (unsigned)sum);
}

// Exclusive scan in one pass (scan_take, scan_before). Writes out[0..n] (out[n] = total) and out2
// (optional). The three-launch form (tile sums, their scan by one block, apply) took 9.3 us at 64^3
// keys and 26 us at 256^3, this 4.5 and 25 us.
__global__ void __launch_bounds__(kThreads) k_scan(const int32_t *__restrict__ in, int64_t n, ScanState scan,
                                                   int32_t *__restrict__ out, int32_t *__restrict__ out2) {
  static_assert(kScanItems % 4 == 0, "whole 16-byte vectors per thread");
  __shared__ int32_t sm[kThreads / 32];
  __shared__ int32_t s_before;
  uint32_t epoch;
  const int32_t tile = scan_take(scan, epoch);
  int64_t base = (int64_t)tile * kScanTile + (int64_t)threadIdx.x * kScanItems;
  // whole tiles move as 16-byte vectors (the arrays are 16-byte aligned and base is a
  // multiple of 4 elements); the ragged last tile element by element
  const bool whole = base + kScanItems <= n && (((uintptr_t)in | (uintptr_t)out | (uintptr_t)out2) & 15) == 0;
  int32_t v[kScanItems];
  int32_t s = 0;
  if (whole) {
#pragma unroll
    for (int q = 0; q < kScanItems; q += 4) {
      const int4 a = *reinterpret_cast<const int4 *>(in + base + q);
      v[q] = a.x; v[q + 1] = a.y; v[q + 2] = a.z; v[q + 3] = a.w;
    }
  } else {
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) v[q] = base + q < n ? in[base + q] : 0;
  }
#pragma unroll
  for (int q = 0; q < kScanItems; ++q) s += v[q];
  int32_t total;
  int32_t e = block_excl_scan(s, sm, total);
  if (threadIdx.x < 32) {
    const int32_t before = scan_before<int32_t, tile_sum>(scan, epoch, tile, total, in);
    if (threadIdx.x == 0) s_before = before;
  }
  __syncthreads();
  e += s_before;
  if (whole) {
#pragma unroll
    for (int q = 0; q < kScanItems; q += 4) {
      int4 o;
      o.x = e; e += v[q];
      o.y = e; e += v[q + 1];
      o.z = e; e += v[q + 2];
      o.w = e; e += v[q + 3];
      *reinterpret_cast<int4 *>(out + base + q) = o;
      if (out2) *reinterpret_cast<int4 *>(out2 + base + q) = o;
    }
    if (base + kScanItems == n) out[n] = e;
  } else {
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
      int64_t i = base + q;
      if (i < n) {
        out[i] = e;
        if (out2) out2[i] = e;
      }
      e += v[q];
      if (i == n - 1) out[n] = e;
    }
  }
}

__global__ void k_scatter(const uint32_t *__restrict__ keys, int shift, int64_t n, int32_t *__restrict__ cursor,
                          int32_t *__restrict__ sidx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t to = place_of(keys, shift, i, n, cursor);
  if (i < n) sidx[to] = (int32_t)i;
}

// The order within a node: 64-bit items (secondary key << 32 | particle), where the secondary
// key is the given order value (reference position, or particle id) or the h bits, sorted
// ascending -- so particles of equal h by storage index.
__device__ __forceinline__ unsigned long long seg_item(const int32_t *__restrict__ order,
                                                       const uint32_t *__restrict__ keys, int32_t v) {
  const uint32_t sec = order ? (uint32_t)order[v] : (keys[v] & 7u);
  return ((unsigned long long)sec << 32) | (uint32_t)v;
}

// k_scatter with the particles' items instead of their indices
__global__ void k_scatter_items(const uint32_t *__restrict__ keys, int shift, int64_t n,
                                const int32_t *__restrict__ order, int32_t *__restrict__ cursor,
                                unsigned long long *__restrict__ items, int32_t *__restrict__ big_count) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *big_count = 0;  // k_segrank's list
  const int32_t to = place_of(keys, shift, i, n, cursor);
  if (i < n) items[to] = seg_item(order, keys, (int32_t)i);
}

// Segments of up to kRankSeg items: one thread per item counts the smaller items of its segment
// (neighbouring threads read the same ones) and writes its particle at that place. Longer
// segments are listed for k_segsort_big. The line: a rank costs an item about four
// instructions per other item, a bitonic sort about log2(len)^2 / 2 exchanges of ten
// instructions and as many barriers; they meet near 150 items. (One thread insertion-sorting a
// node of up to 16 in local memory, everything longer through the bitonic kernel: 4.04 ms for
// 2^24 particles in 64 blobs on 256^3 cells; this way 0.18 ms.)
constexpr int kRankSeg = 128;
constexpr int kMidSeg = 2048;         // segments sorted by 256 threads in 16 KB of shared memory
constexpr int kBigSegMax = 16384;     // per-node particles sortable on chip (8 B each in shared memory)

__global__ void __launch_bounds__(256) k_segrank(const unsigned long long *__restrict__ items,
                                                 const uint32_t *__restrict__ keys, int shift, int64_t n,
                                                 const int32_t *__restrict__ cell_start, int32_t *__restrict__ sidx,
                                                 int32_t *__restrict__ okey, int32_t *__restrict__ big_list, int32_t *__restrict__ big_count,
                                                 int32_t *__restrict__ err) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const unsigned long long mine = items[p];
  const int32_t v = (int32_t)(uint32_t)mine;
  const uint32_t node = keys[v] >> shift;
  const int32_t a = cell_start[node], b = cell_start[node + 1];
  if (b - a > kRankSeg) {
    if (p == a) {
      if (b - a > kBigSegMax) atomicOr(err, kErrCapacity);
      big_list[atomicAdd(big_count, 1)] = (int32_t)node;
    }
    if (b - a > kBigSegMax) {  // left unsorted, reported
      sidx[p] = v;
      if (okey) okey[p] = (int32_t)(mine >> 32);
    }
    return;
  }
  int rank = 0;
  for (int32_t q = a; q < b; ++q) rank += items[q] < mine ? 1 : 0;
  sidx[a + rank] = v;
  if (okey) okey[a + rank] = (int32_t)(mine >> 32);
}

// one block per listed long segment of (lo, hi] items: bitonic sort in shared memory
__global__ void k_segsort_big(const int32_t *__restrict__ cell_start, const unsigned long long *__restrict__ items,
                              int32_t *__restrict__ sidx, int32_t *__restrict__ okey,
                              const int32_t *__restrict__ big_list,
                              const int32_t *__restrict__ big_count, int32_t lo, int32_t hi) {
  extern __shared__ unsigned long long sk[];
  const int32_t nbig = *big_count;
  for (int32_t w = blockIdx.x; w < nbig; w += gridDim.x) {
    const int32_t c = big_list[w];
    const int32_t a = cell_start[c];
    const int32_t len = cell_start[c + 1] - a;
    if (len <= lo || len > hi) continue;  // the same for the whole block
    int32_t m = 1;
    while (m < len) m <<= 1;
    for (int32_t q = threadIdx.x; q < m; q += blockDim.x) sk[q] = q < len ? items[a + q] : ~0ull;
    __syncthreads();
    for (int32_t kk = 2; kk <= m; kk <<= 1) {
      for (int32_t j = kk >> 1; j > 0; j >>= 1) {
        for (int32_t t = threadIdx.x; t < m >> 1; t += blockDim.x) {
          const int32_t q = ((t & ~(j - 1)) << 1) | (t & (j - 1)), r = q | j;
          const bool up = (q & kk) == 0;
          const unsigned long long x = sk[q], y = sk[r];
          if ((x > y) == up) {
            sk[q] = y;
            sk[r] = x;
          }
        }
        __syncthreads();
      }
    }
    for (int32_t q = threadIdx.x; q < len; q += blockDim.x) {
      sidx[a + q] = (int32_t)(uint32_t)sk[q];
      if (okey) okey[a + q] = (int32_t)(sk[q] >> 32);
    }
    __syncthreads();
  }
}

}  // namespace

namespace {

// The per-step reorder: a thread a particle, all its values at once, so that the index is read once
// and the gathers (short runs: a particle moves a fraction of a cell a step) are in flight together.
// Bound by memory: 12 values, three words and the index each way. As a launch per array, the words
// through one scratch array and back: 2^24 particles 1.20 ms, 131,072 85 us in 19 launches; this way
// 0.52 ms and 4 us.
constexpr int kReorderArrays = 12;
struct Reorder {
  const double *src[kReorderArrays];
  double *dst[kReorderArrays];
  const int32_t *flag, *ref;
  const uint32_t *key;
  int32_t *flag_to, *ref_to, *phys_of_ref;
  uint32_t *key_to;
};
__global__ void __launch_bounds__(kThreads) k_reorder(Reorder r, int arrays, const int32_t *__restrict__ idx, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t j = __ldcs(idx + i);
  double v[kReorderArrays];
#pragma unroll
  for (int a = 0; a < kReorderArrays; ++a)
    if (a < arrays) v[a] = r.src[a][j];
  const int32_t flag = r.flag[j], ref = r.ref ? r.ref[j] : 0;
  const uint32_t key = r.key[j];
#pragma unroll
  for (int a = 0; a < kReorderArrays; ++a)
    if (a < arrays) __stcs(r.dst[a] + i, v[a]);
  __stcs(r.flag_to + i, flag);
  __stcs(r.key_to + i, key);
  if (r.ref) {
    __stcs(r.ref_to + i, ref);
    r.phys_of_ref[ref] = (int32_t)i;
  }
}

inline int blocks_for(int64_t n, int per = kThreads) { return (int)((n + per - 1) / per); }

}  // namespace

int exclusive_scan(pstep_ctx *h, const int32_t *in, int64_t n, int32_t *out, int32_t *out2) {
  int64_t nb = (n + kScanTile - 1) / kScanTile;
  if (nb > h->scan_nblocks) {
    snprintf(h->err, sizeof h->err, "scan scratch too small");
    return PSTEP_ERR_STATE;
  }
  k_scan<<<(int)nb, kThreads, 0, h->stream>>>(in, n, scan_state(h), out, out2);
  PSTEP_LAUNCHED(h);
  return PSTEP_OK;
}

int64_t scan_blocks_needed(int64_t n) { return (n + kScanTile - 1) / kScanTile; }

// Counting sort of the h->np particles by (keys[i] >> shift) into nkeys buckets:
// cell_start[0..nkeys] and sidx, every bucket ordered by the secondary key. counted: h->counts already
// holds the buckets' sizes.
int csr_sort(pstep_ctx *h, const uint32_t *keys, int shift, int64_t nkeys, const int32_t *order, int32_t *cell_start,
             int32_t *sidx, int32_t *okey, int order_within, bool counted) {
  if (!counted) PSTEP_CUDA(cudaMemsetAsync(h->counts, 0, sizeof(int32_t) * nkeys, h->stream));
  if (h->np > 0 && !counted) {
    k_count<<<blocks_for(h->np), kThreads, 0, h->stream>>>(keys, shift, h->np, h->counts);
    PSTEP_LAUNCHED(h);
  }
  int rc = exclusive_scan(h, h->counts, nkeys, cell_start, h->cursor);
  if (rc) return rc;
  if (h->np > 0 && !order_within) {
    k_scatter<<<blocks_for(h->np), kThreads, 0, h->stream>>>(keys, shift, h->np, h->cursor, sidx);
    PSTEP_LAUNCHED(h);
  } else if (h->np > 0) {
    unsigned long long *items = (unsigned long long *)h->perm_tmp;  // capacity x 8 bytes, free between calls
    k_scatter_items<<<blocks_for(h->np), kThreads, 0, h->stream>>>(keys, shift, h->np, order, h->cursor, items,
                                                                    h->big_count);
    PSTEP_LAUNCHED(h);
    k_segrank<<<blocks_for(h->np, 256), 256, 0, h->stream>>>(items, keys, shift, h->np, cell_start, sidx, okey,
                                                             h->big_list,
                                                             h->big_count, h->err_word);
    PSTEP_LAUNCHED(h);
    k_segsort_big<<<8 * h->num_sms, 256, kMidSeg * sizeof(unsigned long long), h->stream>>>(
        cell_start, items, sidx, okey, h->big_list, h->big_count, kRankSeg, kMidSeg);
    PSTEP_LAUNCHED(h);
    if (h->np > kMidSeg) {
      const size_t smem = (size_t)kBigSegMax * sizeof(unsigned long long);
      PSTEP_CUDA(cudaFuncSetAttribute(k_segsort_big, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      k_segsort_big<<<h->num_sms, 1024, smem, h->stream>>>(cell_start, items, sidx, okey, h->big_list, h->big_count,
                                                           kMidSeg, kBigSegMax);
      PSTEP_LAUNCHED(h);
    }
  }
  return PSTEP_OK;
}

int sort_by_node(pstep_ctx *h, const uint32_t *keys, Csr &out) {
  const int32_t *order =
      ((h->cfg.flags & PSTEP_TRACK_ORDER) && (h->cfg.flags & PSTEP_REFERENCE_SUMS)) ? h->ref_of_phys : nullptr;
  int rc = csr_sort(h, keys, 3, h->geom.gsize, order, out.cell_start, out.sidx,
                    order ? out.okey : nullptr, 1);
  out.identity = 0;
  return rc;
}

// Reorder particle storage by csr_prev.sidx (the sort of the positions the next
// stage starts from): every per-particle array is gathered through the permutation into one that
// holds nothing between steps (*_np1 and *_new are the base then, the new records and the
// new sort not yet made), and the pointers are swapped.
int f64_reorder(pstep_ctx *h) {
  const int64_t n = h->np;
  if (n == 0) return PSTEP_OK;
  Reorder r{};
  int arrays = 0;
  auto move = [&](double *&arr, double *&free_one) {
    r.src[arrays] = arr;
    r.dst[arrays++] = free_one;
    double *t = arr;
    arr = free_one;
    free_one = t;
  };
  for (int q = 0; q < 7; ++q) move(h->s.base[q], h->s.np1[q]);
  move(h->s.rhs_t, h->s.snew[0]);
  if (h->s.itp) move(h->s.itp, h->s.snew[1]);
  for (int d = 0; d < 3; ++d) move(h->s.frac_prev[d], h->s.frac_new[d]);
  r.flag = h->s.flag;
  r.flag_to = h->csr_new.sidx;
  h->csr_new.sidx = h->s.flag;
  h->s.flag = r.flag_to;
  r.key = h->s.key_prev;
  r.key_to = h->s.key_new;
  h->s.key_new = h->s.key_prev;
  h->s.key_prev = r.key_to;
  if (h->cfg.flags & PSTEP_TRACK_ORDER) {
    r.ref = h->ref_of_phys;
    r.ref_to = h->ref_spare;
    r.phys_of_ref = h->phys_of_ref;
    h->ref_of_phys = r.ref_to;
    h->ref_spare = (int32_t *)r.ref;
  }
  k_reorder<<<blocks_for(n), kThreads, 0, h->stream>>>(r, arrays, h->csr_prev.sidx, n);
  PSTEP_LAUNCHED(h);
  h->csr_prev.identity = 1;
  return PSTEP_OK;
}

}  // namespace pstep
