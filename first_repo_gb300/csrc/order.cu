// Reference particle order (PSTEP_TRACK_ORDER): the permutation that the
// reference's single-rank Send_Recv leaves in its vectors (particle.cpp:150-311,
// 745-858), kept as a map between the reference's positions and device storage.
//
// One pass per dimension (z, then y, then x). In a pass, with n particles of
// which l leave the slab (SortValid*: x_new > xh or < xl), m = n - l:
//  - front leavers (position < m) are overwritten, in ascending order, by the
//    stayers of the back region [m, n) taken in descending order (the
//    swap-with-last of SortValid*);
//  - the leavers are emitted in the order the swap loop meets them. Writing
//    each leaver's emission index as s = n - a, the "anchor" a is
//      front leaver of rank r:     a = (r == 0) ? n : q_(r-1)
//      back leaver at q:           a = q,  except q == m (only possible when
//                                  no back stayer lies below it): a = E,
//    where q_0 > q_1 > ... are the back stayers and E = q_(F-1) (or n when
//    there are none). Anchors are distinct, so sorting by descending anchor
//    is a scatter into l+1 slots;
//  - FromBuf appends the low-side leavers first (Rbuf0 carries what was sent to
//    the low neighbour, which is this rank), then the high-side ones, each in
//    emission order.
// All work is O(l) apart from one look at every particle's leave code and, a pass, at a bit per
// particle, and nothing waits on the host: the counts stay on the device and the kernels loop over
// them. A pass is two launches: k_leavers scans the bits, k_pass, one cluster, does the rest between
// its barriers and sets the next pass's bits. (A kernel per step with a scan of its own, seven
// launches a pass, each of the few leavers' steps alone: 22 us a pass at 131,072 particles on 64^3
// cells and 119 us at 2^24 on 256^3, where the bit of every particle was gathered in the reference's
// order; this way 11 and 21 us.)
#include <cooperative_groups.h>

#include "scan.cuh"

namespace pstep {

namespace {

constexpr int kPassBlocks = 8, kPassThreads = 1024;  // one cluster of the portable size
constexpr int kWordItems = 4;                        // bitmap words per thread of k_leavers
constexpr int kWordTile = kThreads * kWordItems;

// scratch layout inside h->ord_scratch
struct OrdBuf {
  uint32_t *bitmap[3];  // per dimension: a bit per position, set for the pass's leavers
  int32_t *wscan;       // per word: the set bits before it; and the total
  int32_t *lpos;        // leaver positions, ascending
  int32_t *bsphys;      // back stayers (descending) -> storage index
  int32_t *bspos;       // back stayers (descending) -> position
  int32_t *slots;       // l + 1 anchor slots -> storage index of the leaver, -1 empty
  int32_t *list;        // storage indices of the particles that leave in some dimension, in no fixed order
  int32_t *cnt;         // [0] = l, [1] = entries of the list
};

int64_t word_len(int64_t cap) { return (cap / 32 + 64) / 4 * 4; }  // whole 16-byte vectors
int64_t pos_len(int64_t cap) { return (cap + 64) / 4 * 4; }

OrdBuf bufs(pstep_ctx *h) {
  OrdBuf b;
  const int64_t W = word_len(h->cap), L = pos_len(h->cap);
  int32_t *at = h->ord_scratch;
  for (int d = 0; d < 3; ++d) b.bitmap[d] = (uint32_t *)(at + d * W);
  b.wscan = at + 3 * W;
  at += 4 * W;
  b.lpos = at;
  b.bsphys = at + L;
  b.bspos = at + 2 * L;
  b.slots = at + 3 * L;
  b.list = at + 4 * L;
  b.cnt = h->ord_count;
  return b;
}

__device__ inline uint32_t leaves(uint32_t code, int d) { return (code >> (2 * d)) & 3u; }

__device__ inline void set_bit(uint32_t *bitmap, int32_t q) { atomicOr(&bitmap[q >> 5], 1u << (q & 31)); }

// Lists the particles that leave in any dimension (the order of the list is immaterial: it only
// sets bits) and sets the first pass's bits. Bounded by the codes' bytes: 16 a thread.
__global__ void __launch_bounds__(kThreads) k_list(const uint8_t *__restrict__ code, const int32_t *__restrict__ ref_of_phys,
                                                   int64_t n, int first, uint32_t *__restrict__ bitmap,
                                                   int32_t *__restrict__ list, int32_t *__restrict__ count) {
  const int64_t base = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * 16;
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  if (base + 16 <= n) {  // the array is aligned and so is base
    const uint4 v = *reinterpret_cast<const uint4 *>(code + base);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  } else {
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (base + q < n) w[q >> 2] |= (uint32_t)code[base + q] << (8 * (q & 3));
  }
  // (a code has six bits: + 0x7f carries into a byte's top bit where it is not 0)
  int mine = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) mine += __popc((w[q] + 0x7f7f7f7fu) & 0x80808080u);
  int before = mine;  // a place in the list: an addition a warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, before, o);
    if ((int)(threadIdx.x & 31) >= o) before += y;
  }
  int at = 0;
  if ((threadIdx.x & 31) == 31 && before) at = atomicAdd(count, before);
  at = __shfl_sync(0xffffffffu, at, 31) + before - mine;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t left = w[q];
    while (left) {
      const int byte = (__ffs(left) - 1) >> 3;
      const uint32_t c = (left >> (8 * byte)) & 255u;
      left &= ~(255u << (8 * byte));
      const int32_t p = (int32_t)base + 4 * q + byte;
      list[at++] = p;
      if (leaves(c, first)) set_bit(bitmap, ref_of_phys[p]);
    }
  }
}

__device__ __noinline__ int32_t word_tile_sum(const uint32_t *bitmap, int32_t tile) {
  bitmap += (int64_t)tile * kWordTile;
  int32_t sum = 0;
  for (int w = threadIdx.x & 31; w < kWordTile; w += 32) sum += __popc(bitmap[w]);
  return (int32_t)__reduce_add_sync(0xffffffffu, (unsigned)sum);
}

// The leavers' positions in ascending order, the set bits before every word, and l; clears the
// bitmap that k_pass sets next.
__global__ void __launch_bounds__(kThreads) k_leavers(const uint32_t *__restrict__ bitmap, uint32_t *__restrict__ clear,
                                                      int64_t nw, ScanState scan, int32_t *__restrict__ wscan,
                                                      int32_t *__restrict__ lpos, int32_t *__restrict__ cnt) {
  __shared__ int32_t sm[kThreads / 32];
  __shared__ int32_t s_before;
  uint32_t epoch;
  const int32_t tile = scan_take(scan, epoch);
  const int64_t base = (int64_t)tile * kWordTile + (int64_t)threadIdx.x * kWordItems;
  uint32_t bits[kWordItems];
  int32_t s = 0;
#pragma unroll
  for (int q = 0; q < kWordItems; ++q) {
    bits[q] = base + q < nw ? bitmap[base + q] : 0u;
    if (base + q < nw) clear[base + q] = 0u;
    s += __popc(bits[q]);
  }
  int32_t total;
  int32_t e = block_excl_scan(s, sm, total);
  if (threadIdx.x < 32) {
    const int32_t before = scan_before<uint32_t, word_tile_sum>(scan, epoch, tile, total, bitmap);
    if (threadIdx.x == 0) s_before = before;
  }
  __syncthreads();
  e += s_before;
#pragma unroll
  for (int q = 0; q < kWordItems; ++q) {
    if (base + q >= nw) break;
    wscan[base + q] = e;
    for (uint32_t left = bits[q]; left; left &= left - 1) lpos[e++] = (int32_t)((base + q) * 32 + __ffs(left) - 1);
    if (base + q == nw - 1) cnt[0] = e;
  }
}

__device__ inline bool is_leaver(const uint32_t *bitmap, int64_t q) { return (bitmap[q >> 5] >> (q & 31)) & 1u; }

// # set bits in [0, q]
__device__ inline int32_t rank_incl(const uint32_t *bitmap, const int32_t *wscan, int64_t q) {
  const int b = (int)(q & 31);
  const uint32_t mask = b == 31 ? 0xffffffffu : ((1u << (b + 1)) - 1u);
  return wscan[q >> 5] + __popc(bitmap[q >> 5] & mask);
}

// The block's exclusive scan of v, and its total. sm: 32 words
__device__ inline unsigned long long scan64(unsigned long long v, unsigned long long *sm, unsigned long long &total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sm[w] = x;
  __syncthreads();
  if (w == 0) {
    unsigned long long s = sm[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    sm[lane] = s;
  }
  __syncthreads();
  total = sm[31];
  return x - v + (w > 0 ? sm[w - 1] : 0ull);
}

// One pass over its l leavers, by one cluster; then the bits of dimension d - 1, into `next` (null: the
// list's count is cleared). What one phase writes the next reads after a cluster barrier, so none of the
// arrays written here is read through the read-only path.
__global__ void __cluster_dims__(kPassBlocks) __launch_bounds__(kPassThreads)
    k_pass(const uint8_t *__restrict__ code, int d, int64_t n, const uint32_t *bitmap, uint32_t *next, OrdBuf b,
           int32_t *phys_of_ref, int32_t *ref_of_phys) {
  namespace cg = cooperative_groups;
  __shared__ unsigned long long sm[32], totals[kPassBlocks];  // low-side leavers, and << 32 the high-side ones
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = rank * kPassThreads + (int)threadIdx.x;
  constexpr int T = kPassBlocks * kPassThreads;
  const int32_t l = b.cnt[0];
  if (l > 0) {
    const int64_t m = n - l;
    const int32_t F = m > 0 ? rank_incl(bitmap, b.wscan, m - 1) : 0;  // front leavers
    // back region [m, n): stayers by descending position; leavers to their anchor slots (not the
    // q == m tail case yet)
    for (int64_t t = tid; t < l; t += T) {
      const int64_t q = m + t;
      const int32_t above_leavers = l - rank_incl(bitmap, b.wscan, q);  // leavers with position > q
      if (!is_leaver(bitmap, q)) {
        const int64_t r = (n - 1 - q) - above_leavers;  // back stayers above q
        b.bsphys[r] = phys_of_ref[q];
        b.bspos[r] = (int32_t)q;
      } else if (q != m) {
        b.slots[q - m] = phys_of_ref[q];
      }
    }
    cluster.sync();
    // front leavers (rank r < F) and the q == m tail leaver
    for (int64_t r = tid; r <= F; r += T) {
      if (r < F) {
        // anchor of front leaver r: q_(r-1) (position of the back stayer of rank r-1), or n
        const int64_t a = r > 0 ? b.bspos[r - 1] : n;
        b.slots[a - m] = phys_of_ref[b.lpos[r]];
      } else if (is_leaver(bitmap, m)) {
        const int64_t E = F > 0 ? b.bspos[F - 1] : n;
        b.slots[E - m] = phys_of_ref[m];
      }
    }
    cluster.sync();
    // the slots from the highest anchor down (= emission order), a run of them a thread:
    // destinations m + rank among low-side leavers, then m + their number + rank among high-side ones
    const int64_t per = ((int64_t)l + 1 + T - 1) / T, u0 = tid * per, u1 = u0 + per <= l + 1 ? u0 + per : l + 1;
    unsigned long long mine = 0;
    for (int64_t u = u0; u < u1; ++u) {
      const int32_t ph = b.slots[l - u];
      if (ph >= 0) mine += (leaves(code[ph], d) & 2u) ? 1ull : 1ull << 32;
    }
    unsigned long long total;
    unsigned long long e = scan64(mine, sm, total);
    if (threadIdx.x < kPassBlocks) *cluster.map_shared_rank(&totals[rank], (int)threadIdx.x) = total;
    cluster.sync();
    int32_t nlo = 0;
#pragma unroll
    for (int q = 0; q < kPassBlocks; ++q) {
      e += q < rank ? totals[q] : 0ull;
      nlo += (int32_t)(uint32_t)totals[q];
    }
    int64_t lo = m + (int64_t)(uint32_t)e, hi = m + nlo + (int64_t)(e >> 32);
    for (int64_t u = u0; u < u1; ++u) {
      const int32_t ph = b.slots[l - u];
      if (ph < 0) continue;
      b.slots[l - u] = -1;
      const int64_t dst = (leaves(code[ph], d) & 2u) ? lo++ : hi++;
      phys_of_ref[dst] = ph;
      ref_of_phys[ph] = (int32_t)dst;
    }
    // front leavers' places receive the back stayers
    for (int64_t r = tid; r < F; r += T) {
      const int32_t q = b.lpos[r], ph = b.bsphys[r];
      phys_of_ref[q] = ph;
      ref_of_phys[ph] = q;
    }
    if (next) cluster.sync();
  }
  if (!next) {
    if (tid == 0) b.cnt[1] = 0;
    return;
  }
  const int32_t listed = b.cnt[1];
  for (int64_t i = tid; i < listed; i += T) {
    const int32_t p = b.list[i];
    if (leaves(code[p], d - 1)) set_bit(next, ref_of_phys[p]);
  }
}

__global__ void k_clear(uint32_t *__restrict__ a, int64_t na, int32_t *__restrict__ slots, int64_t ns,
                        int32_t *__restrict__ cnt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < na) a[i] = 0u;
  if (i < ns) slots[i] = -1;
  if (i < 8) cnt[i] = 0;
}

__global__ void k_iota(int32_t *__restrict__ a, int32_t *__restrict__ b, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    a[i] = (int32_t)i;
    b[i] = (int32_t)i;
  }
}

}  // namespace

int64_t order_scratch_words(int64_t cap) { return 4 * word_len(cap) + 5 * pos_len(cap); }

// capacity words that hold nothing outside a pass
int32_t *order_free_words(pstep_ctx *h) { return bufs(h).bsphys; }

// The state between stages, restored by every pass after use: no bits, empty slots, an empty list.
int order_clear(pstep_ctx *h) {
  OrdBuf b = bufs(h);
  const int64_t na = 3 * word_len(h->cap), ns = pos_len(h->cap), most = na > ns ? na : ns;
  k_clear<<<(int)((most + kThreads - 1) / kThreads), kThreads, 0, h->stream>>>(b.bitmap[0], na, b.slots, ns, b.cnt);
  PSTEP_LAUNCHED(h);
  return PSTEP_OK;
}

int order_init(pstep_ctx *h) {
  if (h->np == 0) return PSTEP_OK;
  k_iota<<<(int)((h->np + kThreads - 1) / kThreads), kThreads, 0, h->stream>>>(h->ref_of_phys, h->phys_of_ref, h->np);
  PSTEP_LAUNCHED(h);
  return PSTEP_OK;
}

// the three Send_Recv passes (z, y, x) of one stage
int order_passes(pstep_ctx *h) {
  const int64_t n = h->np;
  if (n == 0) return PSTEP_OK;
  OrdBuf b = bufs(h);
  const int64_t nw = (n + 31) / 32;
  const int64_t groups = (n + 15) / 16;
  k_list<<<(int)((groups + kThreads - 1) / kThreads), kThreads, 0, h->stream>>>(h->leave_code, h->ref_of_phys, n, 2,
                                                                                  b.bitmap[2], b.list, &b.cnt[1]);
  PSTEP_LAUNCHED(h);
  for (int d = 2; d >= 0; --d) {
    const int next = d > 0 ? d - 1 : 2;  // (z's bits are next set by the next stage's k_list)
    k_leavers<<<(int)((nw + kWordTile - 1) / kWordTile), kThreads, 0, h->stream>>>(b.bitmap[d], b.bitmap[next], nw,
                                                                                   scan_state(h), b.wscan, b.lpos, b.cnt);
    PSTEP_LAUNCHED(h);
    k_pass<<<kPassBlocks, kPassThreads, 0, h->stream>>>(h->leave_code, d, n, b.bitmap[d], d > 0 ? b.bitmap[next] : nullptr, b,
                                                       h->phys_of_ref, h->ref_of_phys);
    PSTEP_LAUNCHED(h);
  }
  return PSTEP_OK;
}

}  // namespace pstep
