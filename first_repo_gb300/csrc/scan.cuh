// One-pass scans over tiles (decoupled look-back), for kernels whose blocks take a tile each: every
// block takes the next tile by a ticket, publishes its tile's sum, then adds up its predecessors'
// published values from the nearest one back until it meets an inclusive prefix. Tickets are handed
// out in order, so a tile's predecessors are running or done; the wait is bounded all the same, and a
// tile that is still missing then is summed by the waiting block itself, so that a scan's result
// never depends on the waits. A tile's word is (epoch, state, value): words of an earlier scan are
// told by their epoch, so nothing is cleared. The epoch is counted on the device beside the ticket, so that a launch that is
// replayed has one of its own each time.
#pragma once
#include "pstep_internal.cuh"

namespace pstep {

struct ScanState {
  unsigned long long *status;  // a word per tile
  unsigned long long *ticket;  // epoch << 32 | the next tile
  uint32_t polls;              // looks at a predecessor's word before its tile is summed here
};

constexpr uint32_t kScanSum = 1, kScanPrefix = 2;
constexpr uint32_t kScanEpochs = 0x3fffffffu;
constexpr uint32_t kScanPolls = 1u << 16;

inline ScanState scan_state(pstep_ctx *h) {
  return ScanState{h->scan_status, h->scan_ticket, h->wait_idle ? 0u : (h->wait_limit ? h->wait_limit : kScanPolls)};
}

// The block's tile of this launch (all threads call).
__device__ inline int32_t scan_take(const ScanState &scan, uint32_t &epoch) {
  __shared__ unsigned long long taken;
  if (threadIdx.x == 0) {
    const unsigned long long t = atomicAdd(scan.ticket, 1ull);
    if ((uint32_t)t == gridDim.x - 1)  // the last one of this launch
      *scan.ticket = (((t >> 32) + 1) & kScanEpochs) << 32;
    taken = t;
  }
  __syncthreads();
  epoch = (uint32_t)(taken >> 32);
  return (int32_t)(uint32_t)taken;
}

// The sum of the tiles before `tile`, whose own sum is `total` (one whole warp calls). sum_of(in, q): tile
// q's sum from the scan's input, by the whole warp, in every lane.
template <typename T, int32_t (*sum_of)(const T *, int32_t)>
__device__ inline int32_t scan_before(const ScanState &scan, uint32_t epoch, int32_t tile, int32_t total, const T *in) {
  const int lane = (int)(threadIdx.x & 31);
  volatile unsigned long long *st = scan.status;
  auto word = [&](uint32_t state, int32_t value) {
    return ((unsigned long long)(epoch * 4 + state) << 32) | (uint32_t)value;
  };
  if (tile == 0) {
    if (lane == 0) st[0] = word(kScanPrefix, total);
    return 0;
  }
  if (lane == 0) st[tile] = word(kScanSum, total);
  int32_t before = 0;
  for (int32_t at = tile - 1; at >= 0; at -= 32) {  // 32 predecessors at a time, the nearest in lane 0
    const int32_t q = at - lane;
    uint32_t state = kScanPrefix;
    int32_t value = 0;
    if (q >= 0) {
      unsigned long long w = st[q];
      uint32_t polls = 1;
      while (((uint32_t)(w >> 34) != epoch || ((uint32_t)(w >> 32) & 3u) == 0) && ++polls <= scan.polls) w = st[q];
      if (polls > scan.polls) w = 0;  // not there
      state = (uint32_t)(w >> 32) & 3u;
      value = (int32_t)(uint32_t)w;
    }
    const unsigned prefix = __ballot_sync(0xffffffffu, state == kScanPrefix);
    const int stop = prefix ? __ffs(prefix) - 1 : 31;
    // (of the tiles up to the prefix; what is behind it does not matter)
    for (unsigned missing = __ballot_sync(0xffffffffu, state == 0u) & (0xffffffffu >> (31 - stop)); missing;
         missing &= missing - 1u) {
      const int l = __ffs(missing) - 1;
      const int32_t sum = sum_of(in, at - l);
      if (lane == l) value = sum;
    }
    before += (int32_t)__reduce_add_sync(0xffffffffu, (unsigned)(lane <= stop ? value : 0));
    if (prefix) break;
  }
  if (lane == 0) st[tile] = word(kScanPrefix, before + total);
  return before;
}

// The lanes that add to a key together: those with lane 7's key, those with lane 24's, and else
// the run of neighbouring lanes with one key. The storage is nearly in key order, so these are
// almost all that a match over the whole warp would find; that takes a pass per distinct key, and
// shuffles over the groups it finds go one group after the other. Runs alone are broken by every particle
// that has moved on, and in a crowded cell each piece's addition waits for the others'. Count and
// scatter of 2^24 particles on 256^3 cells, and of 2^27 on 512^3 with 1000 in the fullest cells:
// by match 83, 166 us and 0.70, 1.46 ms; by runs 55, 97 us and 1.33, 1.81 ms; this way 55, 93 us and
// 0.86, 1.22 ms. A population uploaded in no order into a handful of cells is matched after all (many runs,
// but several lanes with lane 7's or lane 24's key), as are the crowded cells' most broken warps: a prime
// of 2^22 particles in 4 cells 0.99 -> 0.49 ms, count and scatter at 512^3 now 0.65 and 0.94 ms.
struct Run {
  int first, len, place;
};
__device__ __forceinline__ Run run_of(uint32_t key) {
  const int lane = (int)(threadIdx.x & 31);
  const uint32_t before = __shfl_up_sync(0xffffffffu, key, 1);
  const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0 || key != before);
  const uint32_t low = __ballot_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, 7));
  const uint32_t high = __ballot_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, 24));
  const uint32_t upto = 0xffffffffu >> (31 - lane);  // the lane and those below
  const int head = 31 - __clz(heads & upto);
  const uint32_t after = heads & ~upto;
  const uint32_t run = (after ? (1u << (__ffs(after) - 1)) - 1u : 0xffffffffu) & ~((1u << head) - 1u);
  uint32_t mine = (low >> lane) & 1u ? low : ((high >> lane) & 1u ? high : run);
  if (__popc(heads) > 8 && __popc(low) + __popc(high) >= 6) mine = __match_any_sync(0xffffffffu, key);
  return Run{__ffs(mine) - 1, __popc(mine), __popc(mine & upto) - 1};
}

// Exclusive scan over the block's kThreads threads; smem: kThreads / 32 words.
__device__ inline int32_t block_excl_scan(int32_t v, int32_t *smem, int32_t &total) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem[w] = x;
  __syncthreads();
  if (w == 0) {
    int32_t s = lane < (kThreads / 32) ? smem[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < (kThreads / 32)) smem[lane] = s;
  }
  __syncthreads();
  int32_t warp_off = w > 0 ? smem[w - 1] : 0;
  total = smem[kThreads / 32 - 1];
  __syncthreads();
  return warp_off + x - v;
}

}  // namespace pstep
