// Attention of prompt portions whose heads see one another's scores (the formulas stand in attention_mixed.cu) on tcgen05, keys and
// values of 128, four query heads to a key head, 1, 2 or 4 key heads.
//
// Mixing the heads is linear, so it can be done to the queries: with s_g = scale_i q_g . k_kv(g) + rel[bucket, g],
//   s'_h = sum_g talk[h, g] s_g = scale_i sum_kv (sum_(g of kv) talk[h, g] q_g) . k_kv + (talk rel^T)[h, bucket]
// is the score of ONE query of nkv * 128 numbers with a key's numbers of all key heads, plus a bias of the head's own.  Every head
// is then an ordinary attention head: nothing is exchanged between heads, and the products run on the tensor cores (four times as
// many for the scores as without mixing, twice that for the queries' two parts).
//
// A CTA takes 128 rows (32 tokens x the 4 heads of a key head) of one request.  Its mixed queries are formed in 32-bit and kept as
// TWO bfloat16 numbers each, hi in shared memory, lo in tensor memory (17 bits of mantissa; the weights have 16).  It walks the keys
// in tiles of 128: S = Q~ K^T block by block of 64 numbers as they arrive (hi from shared memory, lo from tensor memory); bias,
// mask and softmax in 32-bit by two threads per row, the biases of the distances that occur in a tile from a table in shared memory;
// the weights as hi + lo over S's columns; O += P V.  Warps 0-7 prologue, softmax, epilogue; warp 8 the TMA boxes, warp 9 the MMAs.
// Tensor memory: Q~_lo 64 columns a key head, S and O 128 each.  Shared memory: Q~_hi 32 KB a key head, three blocks of K, V.
//
// Bound by the chain S (4,096 clocks with 4 key heads) -> softmax -> PV of a CTA's only tile.  2,048 tokens of two requests, 16
// heads on 4 key heads: 301 us and 63 for the shares' merge on mma.sync (attention_mixed_tc.cu, which takes the other sizes and
// steps of few rows), 66 here (74 with the MMAs issued by a loop of one thread).
//
// Whole tiles are multiplied, so numbers that a row does not see (a later row's, slots behind the request's last key) enter with a
// weight of zero.  Where one of them is not finite that product is NaN: a row whose sums come out as anything but finite numbers is
// formed again by a warp from the keys that it sees alone (row_again).
// All waits are bounded; tensor memory is freed on every path.
#include "tcgen05.cuh"
#include "units.cuh"

namespace atom {
namespace mixpf {

using namespace atom::tma;
using namespace atom::tc5;

constexpr int TM = 128, TN = 128, D = 128, HALF = TN / 2, GROUP = 4, TOKENS = TM / GROUP;
constexpr int BLOCK = 128 * 128;              // bytes of one [128 rows][64 elements] swizzled block
constexpr int SOFTMAX_WARPS = 8, LOAD_WARP = 8, MMA_WARP = 9, NTHREADS = 320, K_STAGES = 3;
constexpr int TAB = (TOKENS + TN) * GROUP;    // biases of the distances of a tile
constexpr int REL_ROWS = 40, THR = 64;        // the largest table of biases by distance, and of its thresholds

struct Bars {
  uint64_t q_full, k_full[K_STAGES], k_empty[K_STAGES], v_full, v_empty, s_full, p_full, o_full;
  uint32_t tmem_base;
  int aborted;
  float xch[2][2][TM];                        // [step parity][half][row]: the halves' row maxima (at the end: sums)
};

template <int NKV>
struct Layout {
  static constexpr int NB = 2 * NKV;          // blocks of 64 numbers of a key
  static constexpr int Q = 0, K = NB * BLOCK, V = K + K_STAGES * BLOCK, DATA = V + 2 * BLOCK;
  static constexpr int TABLE = DATA + ((sizeof(Bars) + 63) / 64) * 64;           // [2][TAB] floats, then the mixed biases
  static constexpr size_t BYTES = 1024 + TABLE + 4 * (2 * TAB) + 4 * GROUP * REL_ROWS + 4 * THR;
  static constexpr uint32_t QLO = 0, S = 256, O = 384, COLS = 512;
};

struct Params {
  __nv_bfloat16* out;
  const __nv_bfloat16* q;
  int64_t q_stride;
  const __nv_bfloat16 *k, *v;                 // the pages (row_again)
  const int *cu_q, *ctx_len, *block_table;
  int max_pages, num_seqs, page_size, page_shift;
  int window;
  float scale;
  const float *rel, *talk, *sink;             // [rows, nh] or null, [nh, nh], [nh] or null
  int rel_rows, half;
  const int* thr;
  int n_thr;
  float temp_coef;
  int temp_every;
  int* error;
};
struct Maps {
  CUtensorMap k, v;
};

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kLog2e = 1.4426950408889634f;

// One row's attention over the keys low .. pos by a warp, in 32-bit: the output's numbers 4 lane .. 4 lane + 3.  bt: the request's
// pages; relm, thr: the mixed biases and their thresholds in shared memory; c: what a score is multiplied by.
template <int NKV>
__device__ __noinline__ float4 row_again(const Params& p, const int* bt, const float* relm, const int* thr, int tok, int head, int low,
                                         int pos, float c) {
  constexpr int NH = NKV * GROUP;
  const int lane = threadIdx.x & 31, kvh = head / GROUP;
  float4 q[NKV];
#pragma unroll
  for (int kv = 0; kv < NKV; ++kv) {
    q[kv] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int g = 0; g < GROUP; ++g) {
      const float w = p.talk[head * NH + kv * GROUP + g];
      const uint2 raw = *reinterpret_cast<const uint2*>(p.q + (int64_t)tok * p.q_stride + (kv * GROUP + g) * D + 4 * lane);
      q[kv].x = fmaf(w, __uint_as_float(raw.x << 16), q[kv].x);
      q[kv].y = fmaf(w, __uint_as_float(raw.x & 0xffff0000u), q[kv].y);
      q[kv].z = fmaf(w, __uint_as_float(raw.y << 16), q[kv].z);
      q[kv].w = fmaf(w, __uint_as_float(raw.y & 0xffff0000u), q[kv].w);
    }
  }
  float m = -INFINITY, l = 0.f;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int key = low; key <= pos; ++key) {
    const int page = bt[key >> p.page_shift], slot = key & (p.page_size - 1);
    if (page < 0) continue;
    float s = 0.f;
#pragma unroll
    for (int kv = 0; kv < NKV; ++kv) {
      const uint2 raw = *reinterpret_cast<const uint2*>(p.k + (((int64_t)page * NKV + kv) * p.page_size + slot) * D + 4 * lane);
      s = fmaf(q[kv].x, __uint_as_float(raw.x << 16), s);
      s = fmaf(q[kv].y, __uint_as_float(raw.x & 0xffff0000u), s);
      s = fmaf(q[kv].z, __uint_as_float(raw.y << 16), s);
      s = fmaf(q[kv].w, __uint_as_float(raw.y & 0xffff0000u), s);
    }
    s = warp_sum(s) * c;
    if (p.rel) {
      const int n = pos - key;
      int b = n;
      if (n >= p.half) {
        b = p.half;
        for (int k = 0; k < p.n_thr; ++k) b += thr[k] <= n;
      }
      s += relm[b * GROUP + head % GROUP];
    }
    const float to = fmaxf(m, s), corr = m == -INFINITY ? 0.f : ex2(m - to), w = ex2(s - to);
    const uint2 raw = *reinterpret_cast<const uint2*>(p.v + (((int64_t)page * NKV + kvh) * p.page_size + slot) * D + 4 * lane);
    l = fmaf(l, corr, w);
    o.x = fmaf(w, __uint_as_float(raw.x << 16), o.x * corr);
    o.y = fmaf(w, __uint_as_float(raw.x & 0xffff0000u), o.y * corr);
    o.z = fmaf(w, __uint_as_float(raw.y << 16), o.z * corr);
    o.w = fmaf(w, __uint_as_float(raw.y & 0xffff0000u), o.w * corr);
    m = to;
  }
  if (p.sink) {
    const float sk = p.sink[head] * kLog2e, to = fmaxf(m, sk), corr = m == -INFINITY ? 0.f : ex2(m - to);
    l = fmaf(l, corr, sk == -INFINITY ? 0.f : ex2(sk - to));
    o = make_float4(o.x * corr, o.y * corr, o.z * corr, o.w * corr);
  }
  const float f = l == 0.f ? 0.f : 1.f / l;
  return make_float4(o.x * f, o.y * f, o.z * f, o.w * f);
}

template <int NKV>
__global__ void __launch_bounds__(NTHREADS, 1) attention_mixed_prefill_kernel(const __grid_constant__ Params p, const __grid_constant__ Maps maps) {
  atom::pdl_trigger();
  using LY = Layout<NKV>;
  constexpr int NB = LY::NB, NH = NKV * GROUP;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* sgen = smem_raw + (sbase - smem_u32(smem_raw));
  Bars* bars = reinterpret_cast<Bars*>(sgen + LY::DATA);
  float* tab = reinterpret_cast<float*>(sgen + LY::TABLE);        // [2][TAB]
  float* relm = tab + 2 * TAB;                                     // [REL_ROWS][GROUP]
  int* thr_s = reinterpret_cast<int*>(relm + REL_ROWS * GROUP);   // [THR]

  const atom::units::Unit unit = atom::units::longest_first<NTHREADS>(blockIdx.y, TOKENS, TN, 1, p.num_seqs, 1, p.cu_q, p.ctx_len, p.window, 0);
  const int s = unit.seq;
  if (s < 0) {               // (a unit beyond the last)
    atom::pdl_wait();
    return;
  }
  const int kvh = blockIdx.x, q_begin = p.cu_q[s], q_len = p.cu_q[s + 1] - q_begin, q_start = p.ctx_len[s] - q_len;
  const int tok0 = unit.tile * TOKENS, n_tok = min(TOKENS, q_len - tok0);
  const int p0 = q_start + tok0, key_last = p0 + n_tok - 1;
  const int first = p.window > 0 ? max(0, p0 - p.window + 1) : 0;
  const int j0 = first / TN, j1 = key_last / TN + 1;
  const int* bt = p.block_table + (int64_t)s * p.max_pages;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (known to be uniform)

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, SOFTMAX_WARPS * 32);
    for (int i = 0; i < K_STAGES; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], 1);
    }
    mbar_init(&bars->v_full, 1);
    mbar_init(&bars->v_empty, 1);
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->p_full, SOFTMAX_WARPS * 32);
    mbar_init(&bars->o_full, 1);
    bars->aborted = 0;
    mbar_fence_init();
  }
  for (int e = threadIdx.x; e < p.n_thr; e += NTHREADS) thr_s[e] = p.thr[e];
  for (int e = threadIdx.x; e < p.rel_rows * GROUP; e += NTHREADS) {
    const int b = e / GROUP, h = kvh * GROUP + e % GROUP;
    float v = 0.f;
    for (int g = 0; g < NH; ++g) v = fmaf(p.talk[h * NH + g], p.rel[b * NH + g], v);
    relm[e] = v * kLog2e;
  }
  atom::pdl_wait();      // (weights and the step's index arrays, read so far, were complete before its first kernel; tensor memory after it)
  if (warp == MMA_WARP) tmem_alloc(&bars->tmem_base, LY::COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* aborted = &bars->aborted;

  if (warp == LOAD_WARP) {
    // ------------------------------------------------------------------ loader: a box per page and block of 64 numbers
    const int ps = p.page_size, ppt = TN / ps;        // pages of a tile
    auto page_of = [&](int key) {                      // (pages without a key that is seen: the unit's last key's, removed by the mask)
      int page = key <= key_last ? __ldg(bt + (key >> p.page_shift)) : -1;
      if (page < 0) page = __ldg(bt + (key_last >> p.page_shift));
      return page;
    };
    const bool on = lane < ppt;
    int page = on ? page_of(j0 * TN + lane * ps) : 0;
    int it = 0;
#pragma unroll 1
    for (int j = j0; j < j1; ++j) {
      const int i = j - j0;
#pragma unroll 1
      for (int b = 0; b < NB; ++b, ++it) {
        const int st = it % K_STAGES;
        if (it >= K_STAGES) mbar_wait(&bars->k_empty[st], ((it / K_STAGES) & 1) ^ 1, aborted, p.error);
        if (lane == 0) mbar_expect_tx(&bars->k_full[st], BLOCK);
        __syncwarp();
        if (on) load_box(nullptr, &maps.k, (b & 1) * 64, (page * NKV + (b >> 1)) * ps, &bars->k_full[st], sbase + LY::K + st * BLOCK + lane * ps * 128);
      }
      if (i > 0) mbar_wait(&bars->v_empty, (i & 1) ^ 1, aborted, p.error);
      if (lane == 0) mbar_expect_tx(&bars->v_full, 2 * BLOCK);
      __syncwarp();
      if (on) {
#pragma unroll
        for (int half = 0; half < 2; ++half)
          load_box(nullptr, &maps.v, half * 64, (page * NKV + kvh) * ps, &bars->v_full, sbase + LY::V + half * BLOCK + lane * ps * 128);
      }
      page = on && j + 1 < j1 ? page_of((j + 1) * TN + lane * ps) : 0;
    }
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer: the whole warp runs the loop, one thread issues
    constexpr uint32_t idesc_s = instr_desc(TM, TN, false), idesc_o = instr_desc(TM, D, true);
    const uint64_t q_desc = smem_desc(sbase + LY::Q, 16, 1024), k_desc = smem_desc(sbase + LY::K, 16, 1024);
    const uint64_t v_desc = smem_desc(sbase + LY::V, BLOCK, 1024);
    const bool one = elect_one();
    auto issue_pv = [&](int i) {                      // the weights of tile i: O += P V
      mbar_wait(&bars->v_full, i & 1, aborted, p.error);
      mbar_wait(&bars->p_full, i & 1, aborted, p.error);
      tc_fence_after();
      if (one) {
#pragma unroll
        for (int k = 0; k < 16; ++k)
          umma_ts(tmem + LY::O, tmem + LY::S + k * 8, desc_at(v_desc, (k & 7) * 2048), idesc_o, k > 0 || i > 0);
        umma_commit(&bars->o_full);
        umma_commit(&bars->v_empty);
      }
      __syncwarp();
    };
    mbar_wait(&bars->q_full, 0, aborted, p.error);
    tc_fence_after();
    int it = 0;
#pragma unroll 1
    for (int j = j0; j < j1; ++j) {
      if (j > j0) issue_pv(j - j0 - 1);               // (then the weights' columns take S)
#pragma unroll
      for (int b = 0; b < NB; ++b, ++it) {
        const int st = it % K_STAGES;
        mbar_wait(&bars->k_full[st], (it / K_STAGES) & 1, aborted, p.error);
        tc_fence_after();
        const uint64_t kd = desc_at(k_desc, st * BLOCK);
        if (one) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_ts(tmem + LY::S, tmem + LY::QLO + b * 32 + k * 8, desc_at(kd, k * 32), idesc_s, b + k > 0);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma(tmem + LY::S, desc_at(q_desc, b * BLOCK + k * 32), desc_at(kd, k * 32), idesc_s, 1);
          umma_commit(&bars->k_empty[st]);
          if (b == NB - 1) umma_commit(&bars->s_full);
        }
        __syncwarp();
      }
    }
    issue_pv(j1 - j0 - 1);
  } else {
    // ------------------------------------------------------------------ prologue, softmax, epilogue: row r, half c2
    const int c2 = warp >> 2, r = (warp & 3) * 32 + lane, tok = r / GROUP, head = kvh * GROUP + r % GROUP;
    const bool live = tok < n_tok;
    const uint32_t lane_base = ((uint32_t)((warp & 3) * 32)) << 16;
    // the row's mixed query: this thread's 64 numbers of every key head
    {
      const __nv_bfloat16* qrow = p.q + (int64_t)(q_begin + tok0 + (live ? tok : 0)) * p.q_stride + c2 * 64;
      const float* w = p.talk + head * NH;
#pragma unroll 1
      for (int kv = 0; kv < NKV; ++kv) {
        const int b = kv * 2 + c2;
        float f[GROUP];
#pragma unroll
        for (int g = 0; g < GROUP; ++g) f[g] = live ? w[kv * GROUP + g] : 0.f;
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          uint32_t lo[16];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int ch = part * 4 + c;
            uint4 raw[GROUP];
#pragma unroll
            for (int g = 0; g < GROUP; ++g) raw[g] = *reinterpret_cast<const uint4*>(qrow + (kv * GROUP + g) * D + ch * 8);
            float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int g = 0; g < GROUP; ++g) {
              const uint32_t x[4] = {raw[g].x, raw[g].y, raw[g].z, raw[g].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                a[2 * e] = fmaf(f[g], __uint_as_float(x[e] << 16), a[2 * e]);
                a[2 * e + 1] = fmaf(f[g], __uint_as_float(x[e] & 0xffff0000u), a[2 * e + 1]);
              }
            }
            uint32_t hi[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(a[2 * e], a[2 * e + 1]);
              hi[e] = *reinterpret_cast<const uint32_t*>(&h);
              const __nv_bfloat162 l = __floats2bfloat162_rn(a[2 * e] - __uint_as_float(hi[e] << 16), a[2 * e + 1] - __uint_as_float(hi[e] & 0xffff0000u));
              lo[c * 4 + e] = *reinterpret_cast<const uint32_t*>(&l);
            }
            const uint32_t dst = sbase + LY::Q + b * BLOCK + r * 128 + ((ch ^ (r & 7)) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(dst), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
          }
          tmem_st16(tmem + lane_base + LY::QLO + b * 32 + part * 16, lo);
        }
      }
      tmem_wait_st();
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      tc_fence_before();
      mbar_arrive(&bars->q_full);
    }
    const int pos = live ? p0 + tok : -1;
    const int low = p.window > 0 && live ? max(0, pos - p.window + 1) : 0;
    const float temp = p.temp_every > 0 ? 1.f + p.temp_coef * logf((float)((pos + 1) / p.temp_every) + 1.f) : 1.f;
    const float c = p.scale * temp * kLog2e;
    const uint32_t scol = tmem + lane_base + LY::S, ocol = tmem + lane_base + LY::O + c2 * (D / 2);
    const int pair_bar = 1 + (warp & 3);             // named barrier of the two warps that share these 32 rows
    const int n_mine = j1 - j0;
    float m = -INFINITY, l = 0.f;                    // (of scores times log2 e; l: the sum over this thread's keys only)
    for (int i = 0; i < n_mine; ++i) {
      const int key0 = (j0 + i) * TN;
      // the biases of the tile's distances: entry (d, h) at d * GROUP + h stands for distance d - 127 + p0 - key0
      float* tb = tab + (i & 1) * TAB;
      if (p.rel) {
        for (int d = threadIdx.x; d < TOKENS + TN - 1; d += SOFTMAX_WARPS * 32) {
          const int n = p0 - key0 - (TN - 1) + d;
          int b = max(n, 0);
          if (n >= p.half) {
            b = p.half;
            for (int k = 0; k < p.n_thr; ++k) b += thr_s[k] <= n;
          }
          *reinterpret_cast<float4*>(tb + d * GROUP) = *reinterpret_cast<const float4*>(relm + b * GROUP);
        }
        asm volatile("bar.sync 5, %0;\n" ::"n"(SOFTMAX_WARPS * 32) : "memory");
      }
      mbar_wait(&bars->s_full, i & 1, aborted, p.error);
      tc_fence_after();
      const int k0 = key0 + c2 * HALF;
      float sv[HALF];
#pragma unroll
      for (int q = 0; q < HALF / 32; ++q) tmem_ld32(scol + c2 * HALF + q * 32, sv + q * 32);
      tmem_wait_ld();
      if (p.rel) {
        const float* t = tb + r + (TN - 1 - c2 * HALF) * GROUP;
#pragma unroll
        for (int k = 0; k < HALF; ++k) sv[k] = fmaf(sv[k], c, t[-k * GROUP]);
      } else {
#pragma unroll
        for (int k = 0; k < HALF; ++k) sv[k] *= c;
      }
      if (k0 + HALF - 1 > pos || k0 < low) {
#pragma unroll
        for (int k = 0; k < HALF; ++k)
          if (k0 + k > pos || k0 + k < low) sv[k] = -INFINITY;
      }
      float mx8[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) mx8[e] = -INFINITY;
#pragma unroll
      for (int k = 0; k < HALF; k += 16) {
#pragma unroll
        for (int e = 0; e < 8; ++e) mx8[e] = max3(mx8[e], sv[k + e], sv[k + 8 + e]);
      }
      float mt = max3(max3(mx8[0], mx8[1], mx8[2]), max3(mx8[3], mx8[4], mx8[5]), fmaxf(mx8[6], mx8[7]));
      // After this barrier both threads of the row have read their scores, so S's columns may take P.
      bars->xch[i & 1][c2][r] = mt;
      asm volatile("bar.sync %0, 64;\n" ::"r"(pair_bar) : "memory");
      mt = fmaxf(mt, bars->xch[i & 1][c2 ^ 1][r]);
      // The exponent's offset follows the row maximum lazily, by more than 2^8 at a time; both threads of a row decide alike.
      const bool grow = mt - m > 8.f || (m == -INFINITY && mt != -INFINITY);
      const bool rescale = __any_sync(0xffffffffu, grow);
      const float mx = rescale ? fmaxf(m, mt) : m;
      const float m_use = (mx == -INFINITY) ? 0.f : mx;
      const float alpha = ex2(m - m_use);
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < HALF; ++k) {
        sv[k] = ex2(sv[k] - m_use);
        sum4[k & 3] += sv[k];
      }
      m = mx;
      // P as bf16 pairs: hi in columns 0..63, lo in 64..127; this thread's 64 keys are 32 columns of each
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float a = sv[q * 32 + 2 * e], b = sv[q * 32 + 2 * e + 1];
          const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
          hi[e] = *reinterpret_cast<const uint32_t*>(&h);
          const __nv_bfloat162 ll = __floats2bfloat162_rn(a - __uint_as_float(hi[e] << 16), b - __uint_as_float(hi[e] & 0xffff0000u));
          lo[e] = *reinterpret_cast<const uint32_t*>(&ll);
        }
        tmem_st16(scol + c2 * 32 + q * 16, hi);
        tmem_st16(scol + 64 + c2 * 32 + q * 16, lo);
      }
      // O of the tile before: its MMAs were issued before this tile's S, so they are complete; the wait makes that visible here.
      if (i > 0) {
        mbar_wait(&bars->o_full, (i - 1) & 1, aborted, p.error);
        tc_fence_after();
        if (rescale) {
#pragma unroll
          for (int q = 0; q < D / 64; ++q) {
            float o[32];
            tmem_ld32(ocol + q * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] *= alpha;
            tmem_st32(ocol + q * 32, o);
          }
        }
      }
      l = l * alpha + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->p_full);
    }
    bars->xch[n_mine & 1][c2][r] = l;
    asm volatile("bar.sync %0, 64;\n" ::"r"(pair_bar) : "memory");
    l += bars->xch[n_mine & 1][c2 ^ 1][r];
    mbar_wait(&bars->o_full, (n_mine - 1) & 1, aborted, p.error);
    tc_fence_after();
    const float sk = p.sink && live ? p.sink[head] * kLog2e : -INFINITY;
    const float top = fmaxf(m, sk), wm = top == -INFINITY ? 0.f : ex2(m - top);
    const float f = live ? wm / (l * wm + (sk == -INFINITY ? 0.f : ex2(sk - top))) : 0.f;
    __nv_bfloat16* orow = p.out + ((int64_t)(q_begin + tok0 + tok) * NH + head) * D + c2 * (D / 2);
    float bad = l * 0.f;                             // not zero: what zero times a number that is not finite leaves
#pragma unroll
    for (int q = 0; q < D / 64; ++q) {
      float o[32];
      tmem_ld32(ocol + q * 32, o);
      tmem_wait_ld();
#pragma unroll
      for (int k = 0; k < 32; ++k) bad = fmaf(o[k], 0.f, bad);
      if (live && !*aborted) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint4 v;
          __nv_bfloat162* hh = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
          for (int e = 0; e < 4; ++e) hh[e] = __floats2bfloat162_rn(o[8 * k + 2 * e] * f, o[8 * k + 2 * e + 1] * f);
          *reinterpret_cast<uint4*>(orow + q * 32 + k * 8) = v;
        }
      }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, live && bad != 0.f && !*aborted); todo; todo &= todo - 1) {
      const int b = __ffs(todo) - 1, ra = r - lane + b, ta = tok0 + ra / GROUP, ha = kvh * GROUP + ra % GROUP;
      const int pa = q_start + ta;
      const float4 a = row_again<NKV>(p, bt, relm, thr_s, q_begin + ta, ha, p.window > 0 ? max(0, pa - p.window + 1) : 0, pa,
                                      __shfl_sync(0xffffffffu, c, b));
      if (lane >> 4 == c2) {                         // (the other half of the row is the other thread's)
        __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(p.out + ((int64_t)(q_begin + ta) * NH + ha) * D + 4 * lane);
        dst[0] = __floats2bfloat162_rn(a.x, a.y);
        dst[1] = __floats2bfloat162_rn(a.z, a.w);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem, LY::COLS);
}

template <int NKV>
static int launch(const Params& p, const Maps& m, int T, cudaStream_t stream) {
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(attention_mixed_prefill_kernel<NKV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Layout<NKV>::BYTES) !=
        cudaSuccess)
      return ATOM_ERR_LAUNCH;
    attr_set = true;
  }
  const int units = (T + TOKENS - 1) / TOKENS + p.num_seqs;
  if (units > 65535) return ATOM_ERR_ARG;
  atom::launch_pdl(attention_mixed_prefill_kernel<NKV>, dim3(NKV, units), dim3(NTHREADS), Layout<NKV>::BYTES, stream, p, m);
  return atom::check_launch();
}

}  // namespace mixpf
}  // namespace atom

ATOM_EXPORT int atom_attention_mixed_prefill_supports(int nh, int nkv, int dk, int dv, int page_size, int rel_rows, int n_thr) {
  using namespace atom::mixpf;
  return (nkv == 1 || nkv == 2 || nkv == 4) && nh == GROUP * nkv && dk == D && dv == D && page_size >= 8 && page_size <= 128 &&
                 (page_size & (page_size - 1)) == 0 && rel_rows <= REL_ROWS && n_thr <= THR && atom::tma::encode_fn() != nullptr
             ? 1
             : 0;
}

// As attention_mixed.cu's kernel for steps with portions; talk [nh, nh] is needed; rel_rows: rows of rel.
ATOM_EXPORT int atom_attention_mixed_prefill(void* out, const void* q, int64_t q_stride, const void* k_pages, const void* v_pages,
                                             int64_t num_pages, const int* block_table, int max_pages, int page_size, const int* cu_q,
                                             const int* ctx_len, int num_seqs, int T, int nh, int nkv, float scale, int window,
                                             const float* rel, int rel_rows, int half, const int* thr, int n_thr, const float* talk,
                                             const float* sink, float temp_coef, int temp_every, int* error, cudaStream_t stream) {
  using namespace atom::mixpf;
  if (T <= 0 || num_seqs <= 0) return ATOM_OK;
  const int64_t rows = num_pages * nkv * page_size;
  if (!atom_attention_mixed_prefill_supports(nh, nkv, D, D, page_size, rel ? rel_rows : 0, rel ? n_thr : 0) || talk == nullptr || error == nullptr ||
      q_stride % 8 || (((uintptr_t)out | (uintptr_t)q) % 16) != 0 || num_pages <= 0 || rows >= 0x7fffffff ||
      (rel && rel_rows < half + n_thr + (n_thr ? 1 : 0)))
    return ATOM_ERR_ARG;
  Params p{};
  p.out = (__nv_bfloat16*)out;
  p.q = (const __nv_bfloat16*)q;
  p.q_stride = q_stride;
  p.k = (const __nv_bfloat16*)k_pages;
  p.v = (const __nv_bfloat16*)v_pages;
  p.cu_q = cu_q;
  p.ctx_len = ctx_len;
  p.block_table = block_table;
  p.max_pages = max_pages;
  p.num_seqs = num_seqs;
  p.page_size = page_size;
  p.page_shift = __builtin_ctz((unsigned)page_size);
  p.window = window;
  p.scale = scale;
  p.rel = rel;
  p.talk = talk;
  p.sink = sink;
  p.rel_rows = rel ? rel_rows : 0;
  p.half = half;
  p.thr = thr;
  p.n_thr = rel ? n_thr : 0;
  p.temp_coef = temp_coef;
  p.temp_every = temp_every;
  p.error = error;
  Maps m;
  if (!atom::tma::cached_map(&m.k, k_pages, (uint64_t)rows, D, D, page_size) || !atom::tma::cached_map(&m.v, v_pages, (uint64_t)rows, D, D, page_size))
    return ATOM_ERR_LIB;
  if (nkv == 1) return launch<1>(p, m, T, stream);
  return nkv == 2 ? launch<2>(p, m, T, stream) : launch<4>(p, m, T, stream);
}
