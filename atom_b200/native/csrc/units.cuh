// Which tile of which request a CTA works on, the longest first.
//
// A step's requests are cut into units of `rows` packed rows (token * group + head in group); a unit walks the key tiles that its rows
// see, between one and hundreds.  CTAs start in the order of their numbers, so with the units sorted by their lengths the last ones to
// start are the shortest and the SMs end together; request by request they end up to a longest unit's time apart.  (Two maps in chunks
// of 1,024, 264 CTAs of 1 to 8 tiles on 148 SMs: 52 -> 44 us; three prompts, 6,007 rows behind up to 2,388 keys: 280 -> 251.)  The
// sort is done by every CTA for itself, before it waits for the kernel in front: a thread a unit, a histogram of the lengths, the
// wanted unit's rank among those of its length.  Lengths of 64 key tiles and more (8,192 keys) count as one: such units come first, in
// the order in which they stand.
#pragma once
#include "common.cuh"

namespace atom {
namespace units {

struct Unit {
  int seq, tile;             // request, unit of the request; seq < 0: there is none
};

// The first key that a row at position pos sees.
__device__ __forceinline__ int first_key(int pos, int window, int chunked) {
  if (window <= 0) return 0;
  return chunked ? pos / window * window : max(0, pos - window + 1);
}

// Units of a request: `rows` packed rows each, none for fewer than min_rows.
__device__ __forceinline__ int units_of(const int* __restrict__ cu_q, int s, int rows, int min_rows, int group) {
  const int n = (cu_q[s + 1] - cu_q[s]) * group;
  return n >= min_rows ? (n + rows - 1) / rows : 0;
}

// Of many requests this thread's unit, request by request (the request in the upper half), the y-th (got), and how many there are, or
// at least that many where there are more than threads: every warp takes 32 requests at a time, a lane a request.  (Many one after
// another: the two maps of 300 requests of 5 rows 348 us and 160, the latent's heads of 128 requests of 20 rows 392 and 238, 128
// requests of which none has a unit 23 and 15.)  A function of its own, so that the kernels' registers stay as they are for few: inlined
// it made attention of 6,007 rows 2 % slower.
template <int THREADS>
__device__ __noinline__ uint64_t find_among_many(int y, int rows, int min_rows, int num_seqs, int group, const int* __restrict__ cu_q, Unit* got,
                                                 int* count) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int all = 0, seq = -1, tile = 0;
  bool found = false;
#pragma unroll 1
  for (int s0 = 0; s0 < num_seqs; s0 += 32) {
    const int n = s0 + lane < num_seqs ? units_of(cu_q, s0 + lane, rows, min_rows, group) : 0;
    int upto = n;                          // units of this lane's request and those before it
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31);
    auto find = [&](int i, Unit& unit) {   // the i-th unit of these requests, if there is one
      int l = 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(0xffffffffu, upto, l + o - 1) <= i) l += o;
      const int end = __shfl_sync(0xffffffffu, upto, l);
      if (i >= 0 && i < total) unit = Unit{s0 + l, end - 1 - i};
    };
    if (y >= all && y < all + total) {
      Unit unit;
      find(y - all, unit);
      if (tid == 0) *got = unit;
      found = true;
    }
    if (warp * 32 < all + total && warp * 32 + 31 >= all) {
      Unit unit{seq, tile};
      find(tid - all, unit);
      seq = unit.seq;
      tile = unit.tile;
    }
    all += total;
    if (all > THREADS && found) break;
  }
  if (tid == 0) *count = all;
  return (uint64_t)(uint32_t)seq << 32 | (uint32_t)tile;
}

// The y-th unit of the step, by falling numbers of key tiles (`keys` keys each; requests of fewer than min_rows packed rows have no
// units).  Called by all THREADS threads of a CTA.  Steps of more than THREADS units take them request by request, a request's last
// (longest) first.
template <int THREADS>
__device__ __forceinline__ Unit longest_first(int y, int rows, int keys, int min_rows, int num_seqs, int group, const int* __restrict__ cu_q,
                                              const int* __restrict__ ctx_len, int window, int chunked) {
  constexpr int BINS = 64, WARPS = THREADS / 32;
  __shared__ int bins[BINS], same[WARPS], count;
  __shared__ Unit got;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this thread's unit, and how many there are
  Unit mine{-1, 0};
  int all = 0;
  if (num_seqs > 8) {
    const uint64_t m = find_among_many<THREADS>(y, rows, min_rows, num_seqs, group, cu_q, &got, &count);
    mine = Unit{(int)(m >> 32), (int)(uint32_t)m};
    __syncthreads();
    all = count;
  } else {
    for (int s = 0; s < num_seqs; ++s) {
      const int n = units_of(cu_q, s, rows, min_rows, group);
      if (tid >= all && tid < all + n) mine = Unit{s, n - 1 - (tid - all)};
      if (y >= all && y < all + n && tid == 0) got = Unit{s, n - 1 - (y - all)};
      all += n;
    }
  }
  if (y >= all) return Unit{-1, 0};
  if (all > THREADS || all == 1) {
    __syncthreads();
    return got;
  }
  if (tid < BINS) bins[tid] = 0;
  __syncthreads();
  int length = -1;
  if (mine.seq >= 0) {
    const int begin = ctx_len[mine.seq] - (cu_q[mine.seq + 1] - cu_q[mine.seq]), last = (cu_q[mine.seq + 1] - cu_q[mine.seq]) * group - 1;
    const int r0 = mine.tile * rows, r1 = min(r0 + rows - 1, last);
    length = min(BINS - 1, (begin + r1 / group) / keys - first_key(begin + r0 / group, window, chunked) / keys);
    atomicAdd(&bins[length], 1);
  }
  __syncthreads();
  // (every warp) the length whose units the y-th is among, and its rank there: bins 63 - 2 lane and 62 - 2 lane
  const int b0 = bins[BINS - 1 - 2 * lane], b1 = bins[BINS - 2 - 2 * lane];
  int before = b0 + b1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += v;
  }
  before -= b0 + b1;         // units longer than this lane's
  const bool in0 = y >= before && y < before + b0, in1 = y >= before + b0 && y < before + b0 + b1;
  const int from = __ffs(__ballot_sync(0xffffffffu, in0 || in1)) - 1;
  const int wanted = __shfl_sync(0xffffffffu, in0 ? BINS - 1 - 2 * lane : BINS - 2 - 2 * lane, from);
  int rank = __shfl_sync(0xffffffffu, y - before - (in0 ? 0 : b0), from);
  const unsigned mask = __ballot_sync(0xffffffffu, length == wanted);
  if (lane == 0) same[warp] = __popc(mask);
  __syncthreads();
  for (int w = 0; w < warp; ++w) rank -= same[w];
  if (length == wanted && __popc(mask & ((1u << lane) - 1)) == rank) got = mine;      // (one thread)
  __syncthreads();
  return got;
}

}  // namespace units
}  // namespace atom
