// Causal attention of prompt portions over a window, a chunk or all keys (the formulas of window_attention.cu without cap and
// kept first tokens) on tcgen05: values of 128, keys of 64 a map with two maps, or of 128 or 192.
//
// A CTA of 640 threads works on two query tiles A and B of 128 rows of one (request, key head), rows packed as token * group +
// head in group: with one map 256 consecutive rows, with two maps (differential attention) the same 128 rows, A with the first
// map's queries and keys, B with the second's.  It walks the keys that its rows see in tiles of 128:
//     S_X = Q_X K^T     tcgen05.mma from shared memory, 128 x 128 32-bit sums in tensor memory
//     P_X = softmax     two warpgroups per tile, two threads per row (64 keys each): mask, running maximum and sum in 32-bit;
//                       the weights go back over S_X's 128 columns as TWO bfloat16 numbers each, p = hi + lo, so that the
//                       product sees 16 bits of their mantissa
//     O_X += P_X V      tcgen05.mma with A from tensor memory, hi and lo one after the other
// One thread issues every MMA, alternating between the tiles, so that one tile's products run while the other's exponentials
// do, and a key tile serves both.  Warps 0-7 are tile A's softmax and epilogue (0-3 keys 0..63 of a key tile, 4-7 the others),
// 8-15 tile B's, warp 16 issues the TMA boxes, warp 17 the MMAs; the fifth warpgroup cedes registers to the others.  Tensor
// memory: S_A, S_B, O_A, O_B.  Shared memory: Q, two stages of V, two of K (one with keys of 192).
//
// Keys and values come from pages, or (DENSE) from arrays with a row per key in which head h has columns 128 h ..; the third
// block of 64 of keys of 192 then comes from an array that all heads share.
//
// Bound by the two tiles' chains softmax -> PV -> next S; the exponentials (16 a clock) and the MMAs need about the same time.
// 2,048 tokens of two requests, 16 heads of two maps in chunks of 1,024: 152 us on mma.sync (window_attention_tc.cu, which
// takes caps, kept tokens, other sizes and steps of few rows), 44 here (52 with the units request by request; 57 with the MMAs
// issued by one thread's loop).  16 heads of 192 behind a latent of 512 with a window of 1,024: 448 us for the folded form on
// mma.sync (latent_tc.cu), 48 here and 20 to build keys and values.
//
// Whole tiles are multiplied, so numbers that a row does not see (a later row's, another request's rows beside its own in the
// arrays, slots behind a request's last key) enter with a weight of zero.  Where one of them is not finite that product is NaN: a
// row whose sums come out as anything but finite numbers is formed again by a warp from the keys that it sees alone (row_again).
// All waits are bounded; tensor memory is freed on every path.
#include <type_traits>

#include "tcgen05.cuh"
#include "units.cuh"

namespace atom {
namespace wptc {

using namespace atom::tma;
using namespace atom::tc5;

constexpr int TM = 128, TN = 128, DV = 128, HALF = TN / 2;
constexpr int BLOCK = 128 * 128;              // bytes of one [128 rows][64 elements] swizzled block
constexpr int NTHREADS = 640;
// Registers per thread after the warpgroups have traded them.  setmaxnreg.inc waits, without a bound, until the CTA's own pool
// (threads x registers per thread at launch) has that many to give: 512 x 104 + 128 x 64 = 640 x 96; the launch code checks the
// compiled kernels' register counts against it.
constexpr int SOFTMAX_REGS = 104, OTHER_REGS = 64, LAUNCH_REGS = 96;
static_assert(16 * 32 * SOFTMAX_REGS + 4 * 32 * OTHER_REGS <= 640 * LAUNCH_REGS, "the warpgroups' registers exceed the CTA's pool");
constexpr int SOFTMAX_WARPS = 16, LOAD_WARP = 16, MMA_WARP = 17, V_STAGES = 2;
constexpr uint32_t TMEM_COLS = 512, SA_COL = 0, SB_COL = 128, OA_COL = 256, OB_COL = 384;

struct Bars {
  uint64_t q_full, k_full[2], k_empty[2], v_full[V_STAGES], v_empty[V_STAGES];
  uint64_t s_full[2], p_full[2], o_full[2];   // [0] tile A, [1] tile B
  uint32_t tmem_base;
  int aborted;
  float xch[2][2][2][TM];                     // [step parity][query tile][half][row]: the halves' row maxima (at the end: sums)
};

// DKB: 64-number blocks of a key; MAPS: attention maps.
template <int DKB, int MAPS>
struct Layout {
  static constexpr int NKB = DKB * MAPS, K_STAGES = NKB > 2 ? 1 : 2;
  static constexpr int Q = 0, K = 2 * DKB * BLOCK, V = K + K_STAGES * NKB * BLOCK, DATA = V + V_STAGES * 2 * BLOCK;
  static constexpr size_t BYTES = 1024 + DATA + sizeof(Bars) + 64;
  static constexpr int ROWS = MAPS == 2 ? TM : 2 * TM;      // packed rows of a CTA
};
constexpr int LDX = DV + 4;                   // floats per row of the second map's outputs on their way to the first's threads

struct Params {
  __nv_bfloat16* out;
  int64_t out_ld;
  const __nv_bfloat16 *q, *k, *v, *k_shared;  // what the maps describe (row_again)
  int64_t q_ld, k_ld, v_ld, shared_ld;
  const int *cu_q, *ctx_len, *block_table;
  int max_pages, num_seqs, nkv, group, page_size, page_shift;
  int window, chunked;
  float scale_log2;
  const float* sink;
  const __nv_bfloat16* gate;
  int64_t gate_ld;
  float out_mul, lambda, maps_eps;
  const __nv_bfloat16* out_gate;              // DENSE: rows of a number per output, at stride out_gate_ld, or null
  int64_t out_gate_ld;
  int shared_col;                             // DENSE with three blocks: the first column of the shared array's
  int* error;
};
struct Maps {
  CUtensorMap k, v, q, shared;
};

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void fma2(float& x0, float& x1, float c, float d) {
  asm("{\n.reg .b64 a, b, cc, r;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %2};\nmov.b64 cc, {%3, %3};\n"
      "fma.rn.f32x2 r, a, b, cc;\nmov.b64 {%0, %1}, r;\n}\n"
      : "+f"(x0), "+f"(x1) : "f"(c), "f"(d));
}
__device__ __forceinline__ void add2(float& s0, float& s1, float x0, float x1) {
  asm("{\n.reg .b64 a, b, r;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %3};\nadd.rn.f32x2 r, a, b;\nmov.b64 {%0, %1}, r;\n}\n"
      : "+f"(s0), "+f"(s1) : "f"(x0), "f"(x1));
}
__device__ __forceinline__ void sub2(float& s0, float& s1, float x0, float x1) {
  asm("{\n.reg .b64 a, b, r;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %3};\nsub.rn.f32x2 r, a, b;\nmov.b64 {%0, %1}, r;\n}\n"
      : "+f"(s0), "+f"(s1) : "f"(x0), "f"(x1));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kLog2e = 1.4426950408889634f;

using atom::units::first_key;

// One row's attention over the keys low .. pos by a warp, in 32-bit: the output's numbers 4 lane .. 4 lane + 3 over the weights'
// sum, a sink's weight included.  bt: the request's pages; at0 (DENSE): the row of its key 0.
template <int DKB, int MAPS, bool DENSE>
__device__ __noinline__ float4 row_again(const Params& p, const int* bt, int at0, int tok, int head, int kvh, int map, int low, int pos) {
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* q = p.q + (int64_t)tok * p.q_ld + (int64_t)(head * MAPS + map) * (64 * DKB) + 2 * lane;
  float2 qv[DKB];
#pragma unroll
  for (int b = 0; b < DKB; ++b) qv[b] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(q + 64 * b));
  float m = -INFINITY, l = 0.f;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int key = low; key <= pos; ++key) {
    const __nv_bfloat16 *k, *v;
    if (DENSE) {
      k = p.k + (int64_t)(at0 + key) * p.k_ld + kvh * 128;
      v = p.v + (int64_t)(at0 + key) * p.v_ld + kvh * 128;
    } else {
      const int page = bt[key >> p.page_shift], slot = key & (p.page_size - 1);
      if (page < 0) continue;
      k = p.k + ((((int64_t)page * p.nkv + kvh) * MAPS + map) * p.page_size + slot) * (64 * DKB);
      v = p.v + (((int64_t)page * p.nkv + kvh) * p.page_size + slot) * DV;
    }
    float s = 0.f;
#pragma unroll
    for (int b = 0; b < DKB; ++b) {
      const __nv_bfloat16* kb = DENSE && b == 2 ? p.k_shared + (int64_t)(at0 + key) * p.shared_ld + p.shared_col : k + 64 * b;
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(kb + 2 * lane));
      s = fmaf(qv[b].x, f.x, fmaf(qv[b].y, f.y, s));
    }
    s = warp_sum(s) * p.scale_log2;
    const float to = fmaxf(m, s), corr = m == -INFINITY ? 0.f : ex2(m - to), w = ex2(s - to);
    const uint2 raw = *reinterpret_cast<const uint2*>(v + 4 * lane);
    l = fmaf(l, corr, w);
    o.x = fmaf(w, __uint_as_float(raw.x << 16), o.x * corr);
    o.y = fmaf(w, __uint_as_float(raw.x & 0xffff0000u), o.y * corr);
    o.z = fmaf(w, __uint_as_float(raw.y << 16), o.z * corr);
    o.w = fmaf(w, __uint_as_float(raw.y & 0xffff0000u), o.w * corr);
    m = to;
  }
  if (MAPS == 1 && p.sink) {
    const float sk = p.sink[head] * kLog2e, to = fmaxf(m, sk), corr = m == -INFINITY ? 0.f : ex2(m - to);
    l = fmaf(l, corr, ex2(sk - to));
    o = make_float4(o.x * corr, o.y * corr, o.z * corr, o.w * corr);
  }
  const float f = l == 0.f ? 0.f : 1.f / l;
  return make_float4(o.x * f, o.y * f, o.z * f, o.w * f);
}

template <int DKB, int MAPS, bool DENSE>
__global__ void __launch_bounds__(NTHREADS, 1) window_prefill_kernel(const __grid_constant__ Params p, const __grid_constant__ Maps maps) {
  atom::pdl_trigger();
  using LY = Layout<DKB, MAPS>;
  constexpr int NKB = LY::NKB, K_STAGES = LY::K_STAGES, ROWS = LY::ROWS;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* sgen = smem_raw + (sbase - smem_u32(smem_raw));
  Bars* bars = reinterpret_cast<Bars*>(sgen + LY::DATA);

  const atom::units::Unit unit =
      atom::units::longest_first<NTHREADS>(blockIdx.y, ROWS, TN, 1, p.num_seqs, p.group, p.cu_q, p.ctx_len, p.window, p.chunked);
  const int s = unit.seq;
  if (s < 0) {               // (a unit beyond the last)
    atom::pdl_wait();
    return;
  }
  int dense_row = 0;
  if (DENSE) {
    for (int i = threadIdx.x & 31; i < s; i += 32) {      // (every warp)
      const int n = p.cu_q[i + 1] - p.cu_q[i];
      if (n > 0) dense_row += p.ctx_len[i] - first_key(p.ctx_len[i] - n, p.window, p.chunked);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dense_row += __shfl_xor_sync(0xffffffffu, dense_row, o);
  }
  const int kvh = blockIdx.x, q_begin = p.cu_q[s], q_len = p.cu_q[s + 1] - q_begin, ctx = p.ctx_len[s], q_start = ctx - q_len;
  const int rows_total = q_len * p.group, row0 = unit.tile * ROWS;
  const int* bt = DENSE ? nullptr : p.block_table + (int64_t)s * p.max_pages;
  if (DENSE) dense_row -= first_key(q_start, p.window, p.chunked);       // the row of the request's key 0, had it one
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (known to be uniform)
  // key tiles [lo, hi) of each query tile (none where it has no row)
  int lo[2], hi[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int first = row0 + (MAPS == 2 ? 0 : x * TM);
    if (first >= rows_total) {
      lo[x] = hi[x] = hi[0];
    } else {
      lo[x] = first_key(q_start + first / p.group, p.window, p.chunked) / TN;
      hi[x] = (q_start + (min(first + TM, rows_total) - 1) / p.group) / TN + 1;
    }
  }
  const int j0 = lo[0], j1 = max(hi[0], hi[1]);     // (later rows see no earlier keys, and B's tiles begin no later than A's end)
  const int key_last = q_start + (min(row0 + ROWS, rows_total) - 1) / p.group;

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], 1);
      mbar_init(&bars->v_full[i], 1);
      mbar_init(&bars->v_empty[i], 1);
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->p_full[i], 256);
      mbar_init(&bars->o_full[i], 1);
    }
    bars->aborted = 0;
    mbar_fence_init();
  }
  atom::pdl_wait();      // (the step's index arrays, read so far, were complete before its first kernel; tensor memory is taken by CTAs that may run)
  if (warp == MMA_WARP) tmem_alloc(&bars->tmem_base, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* aborted = &bars->aborted;

  if (warp >= SOFTMAX_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(OTHER_REGS));
    if (warp == LOAD_WARP) {
      // ---------------------------------------------------------------- loader: lane l issues box l of a tile
      const int box_rows = DENSE ? TN : p.page_size;
      const int ppt = TN / box_rows;                    // pages of a tile
      const int k_pg = lane / NKB, k_blk = lane % NKB, v_pg = lane >> 1, v_half = lane & 1;
      const bool k_on = k_pg < ppt, v_on = v_pg < ppt;
      // The page of key `key`, or of the unit's last key where that page holds no key that is seen (numbers that the mask removes).
      auto page_of = [&](int key) {
        int page = key <= key_last ? __ldg(bt + (key >> p.page_shift)) : -1;
        if (page < 0) page = __ldg(bt + (key_last >> p.page_shift));
        return page;
      };
      auto k_row = [&](int j) {
        if (DENSE) return dense_row + j * TN;
        return k_on ? ((page_of(j * TN + k_pg * box_rows) * p.nkv + kvh) * MAPS + k_blk / DKB) * p.page_size : 0;
      };
      auto v_row = [&](int j) {
        if (DENSE) return dense_row + j * TN;
        return v_on ? (page_of(j * TN + v_pg * box_rows) * p.nkv + kvh) * p.page_size : 0;
      };
      if (lane < 2 * DKB) {     // Q: a tile is 128 / group tokens of the group's heads, a box per block of 64 columns
        if (lane == 0) mbar_expect_tx(&bars->q_full, 2 * DKB * BLOCK);
        __syncwarp((1u << (2 * DKB)) - 1);
        const int x = lane / DKB, blk = lane % DKB;
        // a tile without rows still gets a box (of rows that exist): the byte count stays fixed
        const int tok0 = q_begin + min(row0 + (MAPS == 2 ? 0 : x * TM), rows_total - 1) / p.group;
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::
                "r"(sbase + LY::Q + lane * BLOCK),
            "l"(&maps.q), "r"((MAPS == 2 ? x : blk) * 64), "r"(kvh * p.group), "r"(tok0), "r"(smem_u32(&bars->q_full))
            : "memory");
      }
      __syncwarp();
      int row_k = k_row(j0), row_v = v_row(j0);
#pragma unroll 1
      for (int j = j0; j < j1; ++j) {
        const int i = j - j0, ks = i % K_STAGES, vs = i % V_STAGES;
        if (i >= K_STAGES) mbar_wait(&bars->k_empty[ks], ((i / K_STAGES) & 1) ^ 1, aborted, p.error);
        if (lane == 0) mbar_expect_tx(&bars->k_full[ks], NKB * BLOCK);
        __syncwarp();
        if (k_on) {
          const uint32_t dst = sbase + LY::K + (ks * NKB + k_blk) * BLOCK + k_pg * box_rows * 128;
          const bool third = DENSE && k_blk == 2;
          load_box(nullptr, third ? &maps.shared : &maps.k, third ? p.shared_col : (DENSE ? kvh * 128 : 0) + (k_blk % DKB) * 64, row_k,
                   &bars->k_full[ks], dst);
        }
        row_k = j + 1 < j1 ? k_row(j + 1) : 0;          // looked up a tile ahead
        if (i >= V_STAGES) mbar_wait(&bars->v_empty[vs], ((i / V_STAGES) & 1) ^ 1, aborted, p.error);
        if (lane == 0) mbar_expect_tx(&bars->v_full[vs], 2 * BLOCK);
        __syncwarp();
        if (v_on)
          load_box(nullptr, &maps.v, (DENSE ? kvh * 128 : 0) + v_half * 64, row_v, &bars->v_full[vs],
                   sbase + LY::V + (vs * 2 + v_half) * BLOCK + v_pg * box_rows * 128);
        row_v = j + 1 < j1 ? v_row(j + 1) : 0;
      }
    } else if (warp == MMA_WARP) {
      // ---------------------------------------------------------------- MMA issuer: the whole warp runs the loop, one thread issues
      constexpr uint32_t idesc_s = instr_desc(TM, TN, false), idesc_o = instr_desc(TM, DV, true);
      const uint64_t q_desc = smem_desc(sbase + LY::Q, 16, 1024), k_desc = smem_desc(sbase + LY::K, 16, 1024);
      const uint64_t v_desc = smem_desc(sbase + LY::V, BLOCK, 1024);
      const bool one = elect_one();
      auto in_range = [&](int x, int j) { return j >= lo[x] && j < hi[x]; };
      int k_ready = j0 - 1;     // the last K tile whose arrival has been waited for
      auto issue_s = [&](auto tile, int j) {
        constexpr int x = decltype(tile)::value;
        const int ks = (j - j0) % K_STAGES;
        if (k_ready < j) {
          mbar_wait(&bars->k_full[ks], ((j - j0) / K_STAGES) & 1, aborted, p.error);
          tc_fence_after();
          k_ready = j;
        }
        const uint64_t kd = desc_at(k_desc, (ks * NKB + (MAPS == 2 ? x * DKB : 0)) * BLOCK);
        if (one) {
#pragma unroll
          for (int k = 0; k < DKB * 4; ++k) {
            const uint32_t o = (k >> 2) * BLOCK + (k & 3) * 32;
            umma(tmem + (x ? SB_COL : SA_COL), desc_at(q_desc, x * DKB * BLOCK + o), desc_at(kd, o), idesc_s, k > 0);
          }
          umma_commit(&bars->s_full[x]);
          if ((in_range(1, j) ? 1 : 0) == x) umma_commit(&bars->k_empty[ks]);     // (tile B's scores come last)
        }
        __syncwarp();
      };
      auto issue_pv = [&](auto tile, int j) {
        constexpr int x = decltype(tile)::value;
        const int vs = (j - j0) % V_STAGES, i = j - lo[x];
        mbar_wait(&bars->p_full[x], i & 1, aborted, p.error);
        tc_fence_after();
        const uint64_t vd = desc_at(v_desc, vs * 2 * BLOCK);
        if (one) {
#pragma unroll
          for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int k = 0; k < TN / 16; ++k)
              umma_ts(tmem + (x ? OB_COL : OA_COL), tmem + (x ? SB_COL : SA_COL) + half * 64 + k * 8, desc_at(vd, k * 2048), idesc_o,
                      half + k > 0 || i > 0);
          umma_commit(&bars->o_full[x]);
          if ((in_range(1, j) ? 1 : 0) == x) umma_commit(&bars->v_empty[vs]);
        }
        __syncwarp();
      };
      constexpr std::integral_constant<int, 0> A{};
      constexpr std::integral_constant<int, 1> B{};
      mbar_wait(&bars->q_full, 0, aborted, p.error);
      tc_fence_after();
      if (in_range(0, j0)) issue_s(A, j0);
      if (in_range(1, j0)) issue_s(B, j0);
#pragma unroll 1
      for (int j = j0; j < j1; ++j) {
        mbar_wait(&bars->v_full[(j - j0) % V_STAGES], ((j - j0) / V_STAGES) & 1, aborted, p.error);
        tc_fence_after();
        if (in_range(0, j)) issue_pv(A, j);
        if (in_range(0, j + 1)) issue_s(A, j + 1);
        if (in_range(1, j)) issue_pv(B, j);
        if (in_range(1, j + 1)) issue_s(B, j + 1);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax and epilogue of tile x, keys / columns of half c
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(SOFTMAX_REGS));
    const int x = warp >> 3, c2 = (warp >> 2) & 1;
    const int r = (warp & 3) * 32 + lane;            // row of the tile = lane of the tensor memory
    const int R = row0 + (MAPS == 2 ? 0 : x * TM) + r;
    const int pos = R < rows_total ? q_start + R / p.group : -1;
    const int low = pos >= 0 ? first_key(pos, p.window, p.chunked) : 0;
    const uint32_t lane_base = ((uint32_t)((warp & 3) * 32)) << 16;
    const uint32_t scol = tmem + lane_base + (x ? SB_COL : SA_COL);
    const uint32_t ocol = tmem + lane_base + (x ? OB_COL : OA_COL) + c2 * (DV / 2);
    const int pair_bar = 1 + x * 4 + (warp & 3);     // named barrier of the two warps that share these 32 rows
    const float c = p.scale_log2;
    const int n_mine = hi[x] - lo[x];
    float m = -INFINITY, l = 0.f;                    // l: the sum over this thread's keys only
    for (int i = 0; i < n_mine; ++i) {
      mbar_wait(&bars->s_full[x], i & 1, aborted, p.error);
      tc_fence_after();
      const int key0 = (lo[x] + i) * TN + c2 * HALF;
      float sv[HALF];
#pragma unroll
      for (int q = 0; q < HALF / 32; ++q) tmem_ld32(scol + c2 * HALF + q * 32, sv + q * 32);
      tmem_wait_ld();
      if (key0 + HALF - 1 > pos || key0 < low) {
#pragma unroll
        for (int k = 0; k < HALF; ++k)
          if (key0 + k > pos || key0 + k < low) sv[k] = -INFINITY;
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
      bars->xch[i & 1][x][c2][r] = mt;
      asm volatile("bar.sync %0, 64;\n" ::"r"(pair_bar) : "memory");
      mt = fmaxf(mt, bars->xch[i & 1][x][c2 ^ 1][r]);
      // The exponent's offset m follows the row maximum lazily: it moves (and O and l are rescaled) only when the maximum has
      // outgrown it by more than 2^8.  Both threads of a row see the same maxima and decide alike.
      const bool grow = (mt - m) * c > 8.f || (m == -INFINITY && mt != -INFINITY);
      const bool rescale = __any_sync(0xffffffffu, grow);
      const float mx = rescale ? fmaxf(m, mt) : m;
      const float m_use = (mx == -INFINITY) ? 0.f : mx;
      const float alpha = ex2((m - m_use) * c);
      const float mc = m_use * c;
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < HALF; k += 4) {
        fma2(sv[k], sv[k + 1], c, -mc);
        fma2(sv[k + 2], sv[k + 3], c, -mc);
#pragma unroll
        for (int e = 0; e < 4; ++e) sv[k + e] = ex2(sv[k + e]);
        add2(sum4[0], sum4[1], sv[k], sv[k + 1]);
        add2(sum4[2], sum4[3], sv[k + 2], sv[k + 3]);
      }
      m = mx;
      // P as bf16 pairs: hi in columns 0..63, lo in 64..127; this thread's 64 keys are 32 columns of each
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(sv[q * 32 + 2 * e], sv[q * 32 + 2 * e + 1]);
          pk[e] = *reinterpret_cast<const uint32_t*>(&h);
          sub2(sv[q * 32 + 2 * e], sv[q * 32 + 2 * e + 1], __uint_as_float(pk[e] << 16), __uint_as_float(pk[e] & 0xffff0000u));
        }
        tmem_st16(scol + c2 * 32 + q * 16, pk);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(sv[q * 32 + 2 * e], sv[q * 32 + 2 * e + 1]);
          pk[e] = *reinterpret_cast<const uint32_t*>(&h);
        }
        tmem_st16(scol + 64 + c2 * 32 + q * 16, pk);
      }
      // O of the tile before: its MMAs were issued before this tile's S, so they are complete; the wait makes that visible here.
      if (i > 0) {
        mbar_wait(&bars->o_full[x], (i - 1) & 1, aborted, p.error);
        tc_fence_after();
        if (rescale) {
#pragma unroll
          for (int q = 0; q < DV / 64; ++q) {
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
      mbar_arrive(&bars->p_full[x]);
    }
    // epilogue: this thread's 64 columns of the row
    const int tok = q_begin + R / p.group, head = kvh * p.group + R % p.group;
    if (n_mine > 0) {
      bars->xch[n_mine & 1][x][c2][r] = l;
      asm volatile("bar.sync %0, 64;\n" ::"r"(pair_bar) : "memory");
      l += bars->xch[n_mine & 1][x][c2 ^ 1][r];
      mbar_wait(&bars->o_full[x], (n_mine - 1) & 1, aborted, p.error);
      tc_fence_after();
    }
    auto gated = [&](float f) {
      return p.gate ? __fdividef(f, 1.f + ex2(-kLog2e * __bfloat162float(p.gate[(int64_t)tok * p.gate_ld + head]))) : f;
    };
    auto store32 = [&](const float* o, float f, int col) {
      __nv_bfloat16* dst = p.out + (int64_t)tok * p.out_ld + head * DV + col;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint4 v;
        __nv_bfloat162* hh = reinterpret_cast<__nv_bfloat162*>(&v);
        float g[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) g[e] = 1.f;
        if (DENSE && p.out_gate) {
          const uint4 raw = *reinterpret_cast<const uint4*>(p.out_gate + (int64_t)tok * p.out_gate_ld + head * DV + col + 8 * k);
          const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 z = __bfloat1622float2(gb[e]);
            g[2 * e] = __fdividef(1.f, 1.f + ex2(-kLog2e * z.x));
            g[2 * e + 1] = __fdividef(1.f, 1.f + ex2(-kLog2e * z.y));
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) hh[e] = __floats2bfloat162_rn(o[8 * k + 2 * e] * f * g[2 * e], o[8 * k + 2 * e + 1] * f * g[2 * e + 1]);
        *reinterpret_cast<uint4*>(dst + k * 8) = v;
      }
    };
    // what zero times a number that is not finite leaves in a sum of zeros
    auto check = [](float& t, const float* o, int n) {
#pragma unroll
      for (int k = 0; k < n; ++k) t = fmaf(o[k], 0.f, t);
    };
    float bad = 0.f;                                 // not zero: this thread's part of the row is formed again
    if constexpr (MAPS == 1) {
      if (n_mine > 0) {
        if (p.sink && pos >= 0) l += ex2(p.sink[head] * kLog2e - (m == -INFINITY ? 0.f : m * c));
        float f = l > 0.f ? p.out_mul / l : 0.f;
        if (pos >= 0) f = gated(f);
#pragma unroll
        for (int q = 0; q < DV / 64; ++q) {
          float o[32];
          tmem_ld32(ocol + q * 32, o);
          tmem_wait_ld();
          check(bad, o, 32);
          if (pos >= 0 && !*aborted) store32(o, f, c2 * (DV / 2) + q * 32);
        }
        bad = fmaf(l, 0.f, bad);
      }
    } else {
      // The second map's outputs pass through shared memory (keys and values are not needed any more: this tile's last product,
      // the CTA's last, has completed) to the first's threads, which subtract them and divide every row by its root mean square.
      float* xb = reinterpret_cast<float*>(sgen + LY::K) + r * LDX + c2 * (DV / 2);
      float o[DV / 2];
#pragma unroll
      for (int q = 0; q < DV / 64; ++q) tmem_ld32(ocol + q * 32, o + q * 32);
      tmem_wait_ld();
      if (x == 1) {
        const float f = l > 0.f ? p.lambda / l : 0.f;
#pragma unroll
        for (int k = 0; k < DV / 2; k += 4)
          *reinterpret_cast<float4*>(xb + k) = make_float4(o[k] * f, o[k + 1] * f, o[k + 2] * f, o[k + 3] * f);
      }
      asm volatile("bar.sync 9, 512;\n" ::: "memory");
      if (x == 0) {
        const float f = l > 0.f ? 1.f / l : 0.f;
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < DV / 2; k += 4) {
          const float4 b = *reinterpret_cast<const float4*>(xb + k);
          o[k] = fmaf(o[k], f, -b.x);
          o[k + 1] = fmaf(o[k + 1], f, -b.y);
          o[k + 2] = fmaf(o[k + 2], f, -b.z);
          o[k + 3] = fmaf(o[k + 3], f, -b.w);
          ss = fmaf(o[k], o[k], fmaf(o[k + 1], o[k + 1], fmaf(o[k + 2], o[k + 2], fmaf(o[k + 3], o[k + 3], ss))));
        }
        bars->xch[(n_mine & 1) ^ 1][x][c2][r] = ss;
        asm volatile("bar.sync %0, 64;\n" ::"r"(pair_bar) : "memory");
        ss += bars->xch[(n_mine & 1) ^ 1][x][c2 ^ 1][r];
        bad = ss * 0.f;
        if (pos >= 0 && !*aborted) {
          const float g = gated(p.out_mul * rsqrtf(ss / (float)DV + p.maps_eps));
          store32(o, g, c2 * (DV / 2));
          store32(o + 32, g, c2 * (DV / 2) + 32);
        }
      }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, pos >= 0 && bad != 0.f && !*aborted); todo; todo &= todo - 1) {
      const int Ra = R - lane + __ffs(todo) - 1, ta = q_begin + Ra / p.group, ha = kvh * p.group + Ra % p.group;
      const int pa = q_start + Ra / p.group, la = first_key(pa, p.window, p.chunked);
      float4 a = row_again<DKB, MAPS, DENSE>(p, bt, dense_row, ta, ha, kvh, 0, la, pa);
      float f = p.out_mul;
      if (MAPS == 2) {
        const float4 b = row_again<DKB, MAPS, DENSE>(p, bt, dense_row, ta, ha, kvh, 1, la, pa);
        a = make_float4(fmaf(-p.lambda, b.x, a.x), fmaf(-p.lambda, b.y, a.y), fmaf(-p.lambda, b.z, a.z), fmaf(-p.lambda, b.w, a.w));
        f *= rsqrtf(warp_sum(fmaf(a.x, a.x, fmaf(a.y, a.y, fmaf(a.z, a.z, a.w * a.w)))) / (float)DV + p.maps_eps);
      }
      if (p.gate) f /= 1.f + ex2(-kLog2e * __bfloat162float(p.gate[(int64_t)ta * p.gate_ld + ha]));
      const float v[4] = {a.x, a.y, a.z, a.w};
      if (lane >> 4 == c2) {                         // (the other half of the row is the other thread's)
        for (int e = 0; e < 4; ++e) {
          const int col = ha * DV + 4 * lane + e;
          const float g = DENSE && p.out_gate ? 1.f / (1.f + ex2(-kLog2e * __bfloat162float(p.out_gate[(int64_t)ta * p.out_gate_ld + col]))) : 1.f;
          p.out[(int64_t)ta * p.out_ld + col] = __float2bfloat16_rn(v[e] * f * g);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem, TMEM_COLS);
}

// Once per kernel: its register count and shared memory.  False if it cannot run.
template <int DKB, int MAPS, bool DENSE>
static bool ready() {
  static int state = -1;
  if (state < 0) {
    cudaFuncAttributes fa;
    auto k = window_prefill_kernel<DKB, MAPS, DENSE>;
    state = cudaFuncGetAttributes(&fa, k) == cudaSuccess && fa.numRegs == LAUNCH_REGS &&
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Layout<DKB, MAPS>::BYTES) == cudaSuccess;
  }
  return state == 1;
}

template <int DKB, int MAPS, bool DENSE>
static int launch(const Params& p, const Maps& m, int T, cudaStream_t stream) {
  if (!ready<DKB, MAPS, DENSE>()) return ATOM_ERR_LIB;
  const int units = (int)(((int64_t)T * p.group + Layout<DKB, MAPS>::ROWS - 1) / Layout<DKB, MAPS>::ROWS) + p.num_seqs;
  if (units > 65535) return ATOM_ERR_ARG;
  atom::launch_pdl(window_prefill_kernel<DKB, MAPS, DENSE>, dim3(p.nkv, units), dim3(NTHREADS), Layout<DKB, MAPS>::BYTES, stream, p, m);
  return atom::check_launch();
}

// (kept by what it describes, as tma::cached_map does: a buffer of queries serves many steps)
static bool map_q(CUtensorMap* m, const void* q, int cols, int nh, int T, int64_t q_stride, int group) {
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  static std::mutex mu;
  const MapKey key{q, (uint64_t)T, (uint64_t)cols, (uint64_t)q_stride, (uint32_t)group, (uint32_t)nh};
  std::lock_guard<std::mutex> lock(mu);
  const auto it = cache.find(key);
  if (it != cache.end()) {
    *m = it->second;
    return true;
  }
  const uint64_t d[3] = {(uint64_t)cols, (uint64_t)nh, (uint64_t)T}, st[2] = {(uint64_t)cols * 2, (uint64_t)q_stride * 2};
  const uint32_t b[3] = {64, (uint32_t)group, (uint32_t)(TM / group)};
  if (!atom::tma::make_map_raw(m, q, 3, d, st, b)) return false;
  if (cache.size() > 65536) cache.clear();
  cache.emplace(key, *m);
  return true;
}

}  // namespace wptc
}  // namespace atom

// 1 if portions of these sizes run here: pages of a power of two of 8 to 128 tokens, a group that divides 128.
ATOM_EXPORT int atom_window_prefill_supports(int nh, int nkv, int dk, int dv, int maps, int page_size) {
  using namespace atom::wptc;
  if (nkv <= 0 || nh <= 0 || nh % nkv || 128 % (nh / nkv) || dv != 128 || page_size < 8 || page_size > 128 || (page_size & (page_size - 1)))
    return 0;
  if (maps == 2) return dk == 64 && ready<1, 2, false>();
  return maps == 1 && dk == 128 && ready<2, 1, false>();
}

// As atom_window_attention_tc for steps with portions, without cap, kept tokens and shares; ctx_len [num_seqs].
ATOM_EXPORT int atom_window_prefill(void* out, int64_t out_ld, const void* q, int64_t q_stride, const void* k_pages, const void* v_pages,
                                    int64_t num_pages, const int* block_table, int max_pages, int page_size, const int* cu_q,
                                    const int* ctx_len, int num_seqs, int T, int nh, int nkv, int dk, float scale, int window,
                                    int chunked, const float* sink, const void* gate, int64_t gate_ld, float out_mul, int maps, float lambda,
                                    float maps_eps, int* error, cudaStream_t stream) {
  using namespace atom::wptc;
  if (T <= 0 || num_seqs <= 0) return ATOM_OK;
  const int64_t k_rows = num_pages * nkv * maps * page_size;
  if (!atom_window_prefill_supports(nh, nkv, dk, 128, maps, page_size) || error == nullptr || q_stride % 8 || out_ld % 8 ||
      ((uintptr_t)out % 16) != 0 || num_pages <= 0 || k_rows >= 0x7fffffff)
    return ATOM_ERR_ARG;
  Params p{};
  p.out = (__nv_bfloat16*)out;
  p.out_ld = out_ld;
  p.cu_q = cu_q;
  p.ctx_len = ctx_len;
  p.block_table = block_table;
  p.max_pages = max_pages;
  p.num_seqs = num_seqs;
  p.nkv = nkv;
  p.group = nh / nkv;
  p.page_size = page_size;
  p.page_shift = __builtin_ctz((unsigned)page_size);
  p.window = window;
  p.chunked = chunked;
  p.scale_log2 = scale * kLog2e;
  p.sink = sink;
  p.gate = (const __nv_bfloat16*)gate;
  p.gate_ld = gate_ld;
  p.out_mul = out_mul;
  p.lambda = lambda;
  p.maps_eps = maps_eps;
  p.error = error;
  p.q = (const __nv_bfloat16*)q;
  p.q_ld = q_stride;
  p.k = (const __nv_bfloat16*)k_pages;
  p.v = (const __nv_bfloat16*)v_pages;
  Maps m;
  if (!map_q(&m.q, q, dk * maps, nh, T, q_stride, p.group) ||
      !atom::tma::cached_map(&m.k, k_pages, (uint64_t)k_rows, dk, dk, page_size) ||
      !atom::tma::cached_map(&m.v, v_pages, (uint64_t)(k_rows / maps), DV, DV, page_size))
    return ATOM_ERR_LIB;
  m.shared = m.k;
  return maps == 2 ? launch<1, 2, false>(p, m, T, stream) : launch<2, 1, false>(p, m, T, stream);
}

// 1 if attention with every head's keys and values of 128 numbers in arrays (and `shared` more numbers of a key for all heads,
// 0 or 64) runs here.
ATOM_EXPORT int atom_dense_prefill_supports(int shared) {
  using namespace atom::wptc;
  return shared == 64 ? ready<3, 1, true>() : (shared == 0 ? ready<2, 1, true>() : 0);
}

// Keys k and values v [keys, heads, 128], rows k_ld and v_ld apart: for every request of the step with rows, one request after
// another, the keys from the first that one of its rows sees to its last.  keys_shared: rows shared_ld apart whose columns
// shared_col .. hold the numbers behind a head's own 128 (shared = 64).  q [T, heads, 128 + shared] at q_stride.  out_gate: outputs
// are multiplied by its sigmoid, [T, heads, 128] at out_gate_ld, or null.
ATOM_EXPORT int atom_dense_prefill(void* out, int64_t out_ld, const void* q, int64_t q_stride, const void* k, int64_t k_ld, const void* v,
                                   int64_t v_ld, const void* keys_shared, int64_t shared_ld, int shared_col, int shared, int64_t keys,
                                   const int* cu_q, const int* ctx_len, int num_seqs, int T, int heads, float scale, int window,
                                   const float* sink, const void* out_gate, int64_t out_gate_ld, int* error, cudaStream_t stream) {
  using namespace atom::wptc;
  if (T <= 0 || num_seqs <= 0) return ATOM_OK;
  if (!atom_dense_prefill_supports(shared) || heads <= 0 || error == nullptr || q_stride % 8 || out_ld % 8 || shared_col % 8 ||
      (((uintptr_t)out | (uintptr_t)out_gate) % 16) != 0 || out_gate_ld % 8 || keys <= 0 || keys >= 0x7fffffff)
    return ATOM_ERR_ARG;
  Params p{};
  p.out = (__nv_bfloat16*)out;
  p.out_ld = out_ld;
  p.cu_q = cu_q;
  p.ctx_len = ctx_len;
  p.num_seqs = num_seqs;
  p.nkv = heads;
  p.group = 1;
  p.window = window;
  p.scale_log2 = scale * kLog2e;
  p.sink = sink;
  p.out_mul = 1.f;
  p.out_gate = (const __nv_bfloat16*)out_gate;
  p.out_gate_ld = out_gate_ld;
  p.shared_col = shared_col;
  p.error = error;
  p.q = (const __nv_bfloat16*)q;
  p.q_ld = q_stride;
  p.k = (const __nv_bfloat16*)k;
  p.k_ld = k_ld;
  p.v = (const __nv_bfloat16*)v;
  p.v_ld = v_ld;
  p.k_shared = (const __nv_bfloat16*)keys_shared;
  p.shared_ld = shared_ld;
  Maps m;
  if (!map_q(&m.q, q, 128 + shared, heads, T, q_stride, 1) || !atom::tma::cached_map(&m.k, k, (uint64_t)keys, (uint64_t)heads * 128, k_ld, TN) ||
      !atom::tma::cached_map(&m.v, v, (uint64_t)keys, (uint64_t)heads * 128, v_ld, TN))
    return ATOM_ERR_LIB;
  m.shared = m.k;
  if (shared && !atom::tma::cached_map(&m.shared, keys_shared, (uint64_t)keys, (uint64_t)shared_ld, shared_ld, TN)) return ATOM_ERR_LIB;
  return shared ? launch<3, 1, true>(p, m, T, stream) : launch<2, 1, true>(p, m, T, stream);
}
