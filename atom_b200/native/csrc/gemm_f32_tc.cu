// The 32-bit matrix product C[M, N] = A[M, K] W[N, K]^T (+ bias) on tcgen05.  Every number enters as THREE bfloat16 numbers, each
// what is left rounded to nearest, that hold all 24 bits of its mantissa, in the six products down to 2^-16 of the largest, smallest
// first; the sums of 64 k's are formed in tensor memory and added up in 32-bit registers, because the tensor cores cut off what a
// long sum cannot hold.  Against 64-bit the result is nearer than one sequential 32-bit sum over K (4,096 normal numbers: see the
// test), so this is no reduced-precision mode.
//
// A row's result does not depend on which other rows share the launch: W's rows are always the 128 rows of an MMA and A's its
// columns, 16 to 128 of them by M, and an output's sum is always that of the sums over the four quarters of K, in this order.
//
// A CTA per tile of 128 columns of C and NX rows, in stages of 64 k's; where the tiles leave SMs idle, four of them (a cluster), each
// with a quarter of K, whose sums meet through distributed shared memory.  W's numbers come as they are through TMA (the first ones
// before the kernel in front has ended), half a stage at a time; eight warps split them, a thread a row, and lay the planes down in
// TENSOR memory, from where the MMAs read them (128 x NX x 16, 24 a stage).  Four or eight warps add the finished sums of a stage to
// their numbers.  Up to 64 rows the same eight warps split A's rows into shared memory; beyond that f32_rows_kernel has laid their
// planes out (every column tile would split them again) and TMA brings them.
//
// Bound by the MMAs and the reads of A's planes from shared memory beside them with 128 rows, by memory (W) with few.  (With W's planes
// in shared memory, written there by sixteen warps that read W themselves, shared memory was the bound with 128 rows: 196 KB of MMA
// operands and 96 KB of planes a stage where it moves 128 bytes a clock.)
// us at K 4,096 and N 6,144 / 4,096, in that form and now: 1 row 93 / 88, 30 / 21 (W alone is a read of 15 / 10 us); 32 rows 86 / 96,
// 35 / 25; 64 rows 103 / 102, 44 / 31; 128 rows 99 / 100, 52 / 30; 500 rows 194 / 104, 149 / 82; 1,030 rows 327 / 220, 250 / 168 (1.2
// PFLOP/s of bf16 products).  Few rows are bound by the splits (four warps to a scheduler with two CTAs on an SM) and by the starts and
// ends.
//
// A number that three bfloat16 numbers do not hold (not finite, beyond their range, or with bits below 2^-133) marks its row: the
// outputs of marked rows of A and W are formed again in 32-bit as gemm_f32.cu does, an output by one thread.
#include "gemm_f32.cuh"
#include "tcgen05.cuh"

namespace atom {
namespace f32tc {

using namespace atom::tma;
using namespace atom::tc5;

constexpr int TILE = 128, KS = 64, HALF = KS / 2;           // rows of W, k's of a stage, of half a stage
constexpr int BLK_RAW = TILE * HALF * 4;                    // bytes of half a stage of W as it comes
constexpr int PLANE_COLS = KS / 2, W_COLS = 3 * PLANE_COLS; // columns of tensor memory of a plane, of a stage of W
constexpr int SPLIT_WARPS = 8, QUARTERS = 4;
// The same where rows begin anywhere: of a row's 16 numbers the five 16-byte pieces that they lie in, a warp's 32 rows one after another.
constexpr int ROW_ANY = 80, BLK_ANY = SPLIT_WARPS * 32 * ROW_ANY, ANY = 3;
// Barriers that say a stage's MMAs have ended, one after another: for whoever waits for the stage, the one two or the one three before
// (one commit a stage: each holds the issuing thread up by some 130 clocks).
constexpr int DONE = 6;

// How W's numbers come: through TMA where its rows begin on 16-byte boundaries and hold whole 16-byte pieces, in pieces that a warp copies
// or number by number (see pick) where they begin anywhere.  (A kernel each: with TMA and pieces in one, 8 to 64 rows whose W TMA brings
// took 3 to 14 % longer; with pieces and numbers in one, pieces 10 %.)
enum Form { BY_TMA, IN_PIECES, BY_NUMBER };
template <int NX, Form FORM>
struct Cfg {
  static constexpr bool PRE = NX == 128;                    // A's planes come from memory
  static constexpr int SUM_WARPS = NX >= 64 ? 8 : 4, COLS = NX / (SUM_WARPS / 4);     // warps that add up, sums of a thread
  static constexpr int LOAD_WARP = SPLIT_WARPS + SUM_WARPS, MMA_WARP = LOAD_WARP + 1, X_WARP = MMA_WARP + 1,
                       THREADS = (X_WARP + (PRE ? 1 : 0)) * 32;
  static constexpr int CTAS = PRE ? 1 : 2;                  // on an SM
  static constexpr int SUMS = NX == 64 ? 1 : 2;             // stages whose sums tensor memory holds
  static constexpr int W_COL = SUMS * NX, COLUMNS = PRE ? 512 : 256;
  static constexpr int BLK_X = NX * 128, XS = PRE ? 3 : 2;  // bytes of a plane of A, stages of A's planes
  static constexpr int RAW = NX == 64 ? 3 : 4;              // halves of stages of W
  // Where a CTA takes all quarters of K: how many of a thread's totals lie in tensor memory, in shared memory, in the thread, and (with
  // 64 rows, whose CTAs have no room) in C.
  static constexpr int T_TOTALS = PRE ? 32 : 0, S_TOTALS = PRE ? 16 : (NX == 64 ? 0 : COLS), R_TOTALS = PRE ? COLS - T_TOTALS - S_TOTALS : 0;
  static constexpr int X = FORM != IN_PIECES ? RAW * BLK_RAW : ANY * BLK_ANY, TOTALS = X + XS * 3 * BLK_X, T_COL = W_COL + 2 * W_COLS;
  static constexpr size_t SMEM = 1024 + (size_t)TOTALS + SUM_WARPS * 32 * S_TOTALS * 4;
  static_assert(T_COL + SUM_WARPS / 4 * T_TOTALS <= COLUMNS && CTAS * COLUMNS <= 512, "tensor memory");
  // (a third CTA on an SM would wait for tensor memory that two hold, and these perhaps for others of its cluster)
  static_assert(CTAS * (SMEM + 2048) <= 228 * 1024 && 3 * (SMEM + 1024) > 228 * 1024 && NX * TILE * 4 <= SMEM - 1024, "shared memory");
};

struct Params {
  float* C;
  const float *A, *W, *bias;
  int64_t lda, ldc;
  int M, N, K, vec;         // vec: rows of A begin on 16-byte boundaries and hold whole 16-byte pieces
  int parts;                // sums over parts of K that make an output: 4, or 1
  int cluster;              // CTAs to a tile: 1, or 4 with a quarter of K each
  const int* odd_rows;      // [M] of f32_rows_kernel, NX = 128
  int* error;
};

// Eight numbers of a row, its numbers k ..; zeros behind the row's end.  whole: all eight exist, on a 16-byte boundary.
__device__ __forceinline__ void load_group(float (&v)[8], const float* x, bool whole, int k, int K) {
  if (whole) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 f = *reinterpret_cast<const float4*>(x + 4 * h);
      v[4 * h] = f.x;
      v[4 * h + 1] = f.y;
      v[4 * h + 2] = f.z;
      v[4 * h + 3] = f.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = k + i < K ? x[i] : 0.f;
  }
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// The group's three planes; true if they do not hold it.
__device__ __forceinline__ bool split_group(const float (&v)[8], uint4 (&q)[3]) {
  uint32_t p[3][4], left = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 r = make_float2(v[2 * i], v[2 * i + 1]);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(r.x, r.y);
      p[m][i] = *reinterpret_cast<const uint32_t*>(&b);
      r = sub2(r, make_float2(__uint_as_float(p[m][i] << 16), __uint_as_float(p[m][i] & 0xffff0000u)));
    }
    left = left | __float_as_uint(r.x) | __float_as_uint(r.y);
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) q[m] = make_uint4(p[m][0], p[m][1], p[m][2], p[m][3]);
  return left != 0;
}
// The same into shared memory, `plane` bytes apart.
__device__ __forceinline__ bool store_planes(const float (&v)[8], uint32_t addr, int plane) {
  uint4 q[3];
  const bool bad = split_group(v, q);
#pragma unroll
  for (int m = 0; m < 3; ++m)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr + m * plane), "r"(q[m].x), "r"(q[m].y), "r"(q[m].z), "r"(q[m].w) : "memory");
  return bad;
}
// 8 consecutive 32-bit columns of this thread's lane.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float (&v)[8]) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint4& v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(taddr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// The place `addr` of this CTA's shared memory in the CTA of rank `rank`, and what stands there.
__device__ __forceinline__ uint32_t peer_at(uint32_t addr, uint32_t rank) {
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(d) : "r"(addr), "r"(rank));
  return d;
}
__device__ __forceinline__ float peer_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t peer_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// A's rows as planes [3][gridDim.x][Kp], a CTA a row; odd[row]: they do not hold it.
__global__ void __launch_bounds__(256) f32_rows_kernel(__nv_bfloat16* __restrict__ planes, int* __restrict__ odd, const float* __restrict__ A,
                                                       int64_t lda, int K, int Kp, int vec) {
  atom::pdl_trigger();
  atom::pdl_wait();
  const int64_t size = (int64_t)gridDim.x * Kp;
  const float* row = A + blockIdx.x * lda;
  bool bad = false;
  for (int k = threadIdx.x * 8; k < Kp; k += 256 * 8) {
    float v[8];
    uint4 q[3];
    load_group(v, row + k, vec && k + 8 <= K, k, K);
    bad |= split_group(v, q);
#pragma unroll
    for (int m = 0; m < 3; ++m) *reinterpret_cast<uint4*>(planes + m * size + (int64_t)blockIdx.x * Kp + k) = q[m];
  }
  const int any = __syncthreads_or(bad);
  if (threadIdx.x == 0) odd[blockIdx.x] = any;
}

template <int NX, Form FORM>
__global__ void __launch_bounds__(Cfg<NX, FORM>::THREADS, Cfg<NX, FORM>::CTAS)
    gemm_f32_tc_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w) {
  atom::pdl_trigger();
  using C = Cfg<NX, FORM>;
  constexpr int XS = C::XS, RAW = C::RAW, SUMS = C::SUMS, COLS = C::COLS, THREADS = C::THREADS;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t raw_full[RAW], raw_empty[RAW], w_full[2], x_full[XS], done[DONE], taken[2];
  __shared__ uint32_t tmem_base, odd_w[TILE / 32], odd_x[4];
  __shared__ int aborted_flag;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  volatile int* aborted = &aborted_flag;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (known to be uniform)
  const int rank = blockIdx.x % p.cluster, n0 = blockIdx.x / p.cluster * TILE, m0 = blockIdx.y * NX;
  const int KT = (p.K + KS - 1) / KS;
  auto quarter = [&](int i) { return p.parts == 1 ? (i > 0 ? KT : 0) : (int)((int64_t)KT * i / QUARTERS); };      // the parts' first stages
  const int k_from = p.cluster == 1 ? 0 : quarter(rank), k_to = p.cluster == 1 ? KT : quarter(rank + 1), n_it = k_to - k_from;
  if (threadIdx.x == 0) {
    for (int s = 0; s < RAW; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], SPLIT_WARPS);
    }
    for (int s = 0; s < XS; ++s) mbar_init(&x_full[s], 1);
    for (int s = 0; s < DONE; ++s) mbar_init(&done[s], 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&w_full[s], SPLIT_WARPS);
      mbar_init(&taken[s], C::SUM_WARPS);
    }
    for (int i = 0; i < 4; ++i) odd_w[i] = odd_x[i] = 0;
    aborted_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  auto load_raw = [&](int h) {                              // half a stage of W
    mbar_expect_tx(&raw_full[h % RAW], BLK_RAW);
    load_box(nullptr, &map_w, (k_from * 2 + h) * (HALF * 2), n0, &raw_full[h % RAW], sbase + (h % RAW) * BLK_RAW);
  };
  auto wait_done = [&](int it) { mbar_wait(&done[it % DONE], (it / DONE) & 1, aborted, p.error); };
  const int halves = 2 * n_it;
  // The same for rows that begin anywhere: a warp that splits brings its own rows' 16 numbers, a lane five of their pieces (rows behind
  // the last one repeat it, or are left out: their outputs are not written).  K 4,097, N 12,288: 1 row 79 us, 64 rows 115, 128 rows
  // 106 (102, 202 and 185 where every thread read its row; with 4 bytes a lane N 32,000, 17 rows 267, 229 so).
  const int first_row = n0 + (warp & 3) * 32, last = min(31, p.N - 1 - first_row), K4 = p.K * 4;
  const char *w0 = reinterpret_cast<const char*>(p.W), *w1 = w0 + (int64_t)p.N * K4;
  const char* first = w0 + (int64_t)first_row * K4 + (warp >> 2) * 64;
  const uint32_t own = sbase + warp * 32 * ROW_ANY;
  const int low = (int)((uintptr_t)first & 15);
  auto copy_any = [&](int h) {
    if (h < halves && last >= 0) {
      const char* from = first - low + (int64_t)(k_from * 2 + h) * (HALF * 4);
      const uint32_t dst = own + (h % ANY) * BLK_ANY + lane * 16;
      const bool inside = from >= w0 && from + (low + last * K4 + ROW_ANY) <= w1;      // every piece lies in W
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const int e = lane + 32 * j, r = e / 5;
        const char* src = from + (((low + min(r, last) * K4) & ~15) + (e - 5 * r) * 16);
        if (inside) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + j * 512), "l"(src) : "memory");
        } else {
#pragma unroll 1
          for (int i = 0; i < 16; i += 4) {
            const bool in = src + i >= w0 && src + i < w1;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst + j * 512 + i), "l"(in ? src + i : w0), "r"(in ? 4 : 0) : "memory");
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // (a weight, which no kernel of the step writes: this does not wait for the kernel in front)
  if (warp == C::LOAD_WARP && lane == 0 && FORM == BY_TMA)
    for (int h = 0; h < min(RAW, halves); ++h) load_raw(h);
  if (FORM == IN_PIECES && warp < SPLIT_WARPS)
    for (int h = 0; h < ANY - 1; ++h) copy_any(h);
  atom::pdl_wait();
  if (warp == C::MMA_WARP) tmem_alloc(&tmem_base, C::COLUMNS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;

  if (warp < SPLIT_WARPS) {
    // W: a thread a row (a lane of tensor memory), 16 of half a stage's 32 numbers
    const int row = (warp & 3) * 32 + lane, part = warp >> 2;
    const uint32_t wcol = tmem + ((uint32_t)((warp & 3) * 32) << 16) + C::W_COL + part * 8;
    // A up to 64 rows: eight neighbouring threads hold the 64 numbers of a row
    constexpr int XG = C::PRE ? 0 : (NX + 31) / 32;         // groups of eight a thread
    const int xrow = threadIdx.x >> 3, ch = threadIdx.x & 7;
    const bool x_on = !C::PRE && xrow < NX;
    uint32_t bad = 0;                                       // bit 0: W's row, bits 1 ..: A's groups
    float xv[8];                                            // the next group of A, asked for half a stage (two groups) or a stage ahead
    auto load_x = [&](int h) {
      const int xg = XG == 2 ? h & 1 : 0, kx = (k_from + (h >> 1)) * KS + ch * 8;
      if (x_on && h < halves) load_group(xv, p.A + (int64_t)min(m0 + xrow + 32 * xg, p.M - 1) * p.lda + kx, p.vec && kx + 8 <= p.K, kx, p.K);
    };
    if (!C::PRE) load_x(0);
#pragma unroll 1
    for (int h = 0; h < halves; ++h) {
      const int it = h >> 1, b = it & 1, second = h & 1;
      float v[2][8];
      if constexpr (FORM == BY_TMA) {
        mbar_wait(&raw_full[h % RAW], (h / RAW) & 1, aborted, p.error);
        const uint32_t src = sbase + (h % RAW) * BLK_RAW + row * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                       : "=f"(v[c >> 1][(c & 1) * 4]), "=f"(v[c >> 1][(c & 1) * 4 + 1]), "=f"(v[c >> 1][(c & 1) * 4 + 2]), "=f"(v[c >> 1][(c & 1) * 4 + 3])
                       : "r"(src + (((part * 4 + c) ^ (row & 7)) << 4)));
      } else if constexpr (FORM == IN_PIECES) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(ANY - 2) : "memory");
        __syncwarp();
        float f[20];
#pragma unroll
        for (int c = 0; c < 5; ++c)
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(f[4 * c]), "=f"(f[4 * c + 1]), "=f"(f[4 * c + 2]), "=f"(f[4 * c + 3])
                       : "r"(own + (h % ANY) * BLK_ANY + lane * ROW_ANY + c * 16));
        const int k = (k_from * 2 + h) * HALF + part * 16, by = (low + min(lane, last) * K4) >> 2 & 3;
#pragma unroll
        for (int i = 0; i < 19; ++i) f[i] = by & 1 ? f[i + 1] : f[i];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i >> 3][i & 7] = by & 2 ? f[i + 2] : f[i];
        if (k + 16 > p.K) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i >> 3][i & 7] = k + i < p.K ? v[i >> 3][i & 7] : 0.f;
        }
      } else {
        const int k = (k_from * 2 + h) * HALF + part * 16;
        const float* wr = p.W + (int64_t)min(n0 + row, p.N - 1) * p.K + k;
#pragma unroll
        for (int g = 0; g < 2; ++g) load_group(v[g], wr + g * 8, false, k + g * 8, p.K);
      }
      if (!second && it >= 2) wait_done(it - 2);            // (the planes' place is free)
      tc_fence_after();
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint4 q[3];
        if (split_group(v[g], q)) bad |= 1u;
#pragma unroll
        for (int m = 0; m < 3; ++m) tmem_st4(wcol + b * W_COLS + m * PLANE_COLS + second * 16 + g * 4, q[m]);
      }
      // (only now have the loads from shared memory ended for certain: their numbers have been used)
      __syncwarp();
      if (FORM == IN_PIECES) copy_any(h + ANY - 1);         // (where the half before this one lay)
      if (FORM == BY_TMA && lane == 0) mbar_arrive(&raw_empty[h % RAW]);
      if (!C::PRE && (XG == 2 || !second)) {
        const int xg = XG == 2 ? second : 0;
        if (x_on && store_planes(xv, sbase + C::X + b * 3 * C::BLK_X + (xrow + 32 * xg) * 128 + ((ch ^ (xrow & 7)) << 4), C::BLK_X)) bad |= 2u << xg;
        load_x(XG == 2 ? h + 1 : h + 2);
      }
      if (second) {
        tmem_wait_st();
        if (!C::PRE) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_full[b]);
      }
    }
    if (bad & 1u) atomicOr(&odd_w[row / 32], 1u << (row % 32));
#pragma unroll
    for (int g = 0; g < XG; ++g)
      if (bad >> (1 + g) & 1) atomicOr(&odd_x[(xrow + 32 * g) / 32], 1u << (xrow % 32));
  } else if (warp == C::LOAD_WARP) {
    if (lane == 0 && FORM == BY_TMA)
      for (int h = RAW; h < halves; ++h) {
        mbar_wait(&raw_empty[h % RAW], ((h / RAW) - 1) & 1, aborted, p.error);
        load_raw(h);
      }
  } else if (C::PRE && warp == C::X_WARP) {
    if (lane == 0)
      for (int it = 0; it < n_it; ++it) {
        const int s = it % XS;
        if (it >= XS) wait_done(it - XS);
        mbar_expect_tx(&x_full[s], 3 * C::BLK_X);
#pragma unroll
        for (int m = 0; m < 3; ++m)
          load_box(nullptr, &map_a, (k_from + it) * KS, m * p.M + m0, &x_full[s], sbase + C::X + (s * 3 + m) * C::BLK_X);
      }
    __syncwarp();
    for (int i = lane; i < NX; i += 32)
      if (m0 + i < p.M && p.odd_rows[m0 + i]) atomicOr(&odd_x[i / 32], 1u << (i % 32));
  } else if (warp == C::MMA_WARP) {
    // The whole warp runs the loop, so that descriptors stay in uniform registers; one thread issues.
    constexpr int PX[6] = {2, 1, 0, 1, 0, 0}, PW[6] = {0, 1, 2, 0, 1, 0};
    constexpr uint32_t idesc = instr_desc(TILE, NX, false);
    const uint64_t desc = smem_desc(sbase + C::X, 16, 1024);
    const bool one = elect_one();
#pragma unroll 1
    for (int it = 0; it < n_it; ++it) {
      const int b = it & 1, xs = C::PRE ? it % XS : b, d = it % SUMS;
      {                                                     // (asked all at once)
        const bool w_now = mbar_try_wait(&w_full[b], (it >> 1) & 1), x_now = !C::PRE || mbar_try_wait(&x_full[xs], (it / XS) & 1);
        const bool t_now = it < SUMS || mbar_try_wait(&taken[d], ((it / SUMS) - 1) & 1);
        if (!w_now) mbar_wait(&w_full[b], (it >> 1) & 1, aborted, p.error);
        if (!x_now) mbar_wait(&x_full[xs], (it / XS) & 1, aborted, p.error);
        if (!t_now) mbar_wait(&taken[d], ((it / SUMS) - 1) & 1, aborted, p.error);
      }
      tc_fence_after();
      const uint64_t xd = desc_at(desc, xs * 3 * C::BLK_X);
      const uint32_t wt = tmem + C::W_COL + b * W_COLS;
      if (one) {
#pragma unroll
        for (int x = 0; x < 6; ++x)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_ts(tmem + d * NX, wt + PW[x] * PLANE_COLS + ks * 8, desc_at(xd, PX[x] * C::BLK_X + ks * 32), idesc, x + ks > 0);
        umma_commit(&done[it % DONE]);
      }
      __syncwarp();
    }
  } else {
    const int q = warp & 3, half = (warp - SPLIT_WARPS) >> 2;      // (a warp reads the quarter of the lanes that its index selects)
    const uint32_t tbase = tmem + ((uint32_t)(32 * q) << 16) + half * COLS;
    const int n = n0 + 32 * q + lane, m = m0 + half * COLS;
    float* c0 = p.C + (int64_t)m * p.ldc + n;
    const uint32_t totals_t = tmem + ((uint32_t)(32 * q) << 16) + C::T_COL + half * C::T_TOTALS;
    const uint32_t totals_s = sbase + C::TOTALS + (threadIdx.x - SPLIT_WARPS * 32) * 4;
    float acc[COLS], total[C::R_TOTALS > 0 ? C::R_TOTALS : 1];
#pragma unroll
    for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
    int it = 0;
    for (int part = p.cluster == 1 ? 0 : rank; part < (p.cluster == 1 ? p.parts : rank + 1); ++part) {
      for (const int to = quarter(part + 1) - k_from; it < to; ++it) {
        const int d = it % SUMS;
        wait_done(it);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < COLS; c += 8) {
          float v[8];
          tmem_ld8(tbase + d * NX + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[c + i] += v[i];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&taken[d]);
      }
      if (p.cluster > 1) {
        // to shared memory for the cluster (whose loads into it, and whose reads by splits and MMAs, have all ended with the last MMA)
#pragma unroll
        for (int i = 0; i < COLS; ++i)
          asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(sbase + ((half * COLS + i) * TILE + 32 * q + lane) * 4), "f"(acc[i]) : "memory");
        break;
      }
      // The quarters' sums meet where this thread keeps its own totals, and the last ones go to C.  (All of them in C, four writes and
      // three reads of it: 1,030 rows, N 4,096, K 1,024 61 us and 54, K 4,096 174 and 168; 128 rows, N 4,096, K 512 22 and 17.)
      const bool end = part == p.parts - 1, writes = n < p.N && !*aborted;
      const float b = end && p.bias && writes ? p.bias[n] : 0.f;
      if constexpr (C::T_TOTALS + C::S_TOTALS + C::R_TOTALS == 0) {
        if (writes) {
#pragma unroll
          for (int c = 0; c < COLS; c += 8) {
            float t[8];
            float* at = c0 + (int64_t)c * p.ldc;
#pragma unroll
            for (int i = 0; i < 8; ++i, at += p.ldc) t[i] = part > 0 && m + c + i < p.M ? *at : 0.f;
            at = c0 + (int64_t)c * p.ldc;
#pragma unroll
            for (int i = 0; i < 8; ++i, at += p.ldc) {
              t[i] += acc[c + i];
              if (end && p.bias) t[i] += b;
              if (m + c + i < p.M) *at = t[i];
              acc[c + i] = 0.f;
            }
          }
        }
      } else {
#pragma unroll
        for (int c = 0; c < COLS; c += 8) {
          float t[8];
          const int s = c - C::T_TOTALS, r = s - C::S_TOTALS;
          if (part > 0) {
            if (s < 0) {
              tmem_ld8(totals_t + c, t);
              tmem_wait_ld();
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              if (s >= 0 && r < 0) asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(t[i]) : "r"(totals_s + (s + i) * (C::SUM_WARPS * 128)) : "memory");
              if (r >= 0) t[i] = total[r + i];
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            t[i] = part > 0 ? t[i] + acc[c + i] : acc[c + i];
            if (end && p.bias) t[i] += b;
            acc[c + i] = 0.f;
          }
          if (!end) {
            if (s < 0) tmem_st8(totals_t + c, t);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              if (s >= 0 && r < 0) asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(totals_s + (s + i) * (C::SUM_WARPS * 128)), "f"(t[i]) : "memory");
              if (r >= 0) total[r + i] = t[i];
            }
          } else if (writes) {
            float* at = c0 + (int64_t)c * p.ldc;
#pragma unroll
            for (int i = 0; i < 8; ++i, at += p.ldc)
              if (m + c + i < p.M) *at = t[i];
          }
        }
        if (C::T_TOTALS > 0 && !end) tmem_wait_st();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == C::MMA_WARP) tmem_dealloc(tmem, C::COLUMNS);
  int j0 = 0, j1 = NX;                                      // the rows of A whose outputs this CTA has
  uint32_t marks[8];
  if (p.cluster > 1) {
    // a CTA puts a quarter of the rows together
    cluster_sync_all();
    j0 = rank * (NX / QUARTERS);
    j1 = j0 + NX / QUARTERS;
    uint32_t from[QUARTERS];
#pragma unroll
    for (int r = 0; r < QUARTERS; ++r) from[r] = peer_at(sbase, r);
    for (int e = j0 * TILE + threadIdx.x; e < j1 * TILE; e += THREADS) {
      const int m = m0 + e / TILE, n = n0 + e % TILE;
      if (m >= p.M || n >= p.N || *aborted) continue;
      float t[QUARTERS], sum = 0.f;
#pragma unroll
      for (int r = 0; r < QUARTERS; ++r) t[r] = peer_f32(from[r] + e * 4);
#pragma unroll
      for (int r = 0; r < QUARTERS; ++r) sum += t[r];
      p.C[(int64_t)m * p.ldc + n] = p.bias ? sum + p.bias[n] : sum;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      marks[i] = marks[4 + i] = 0;
#pragma unroll
      for (int r = 0; r < QUARTERS; ++r) {
        marks[i] |= peer_u32(peer_at(smem_u32(&odd_w[i]), r));
        marks[4 + i] |= peer_u32(peer_at(smem_u32(&odd_x[i]), r));
      }
    }
    cluster_sync_all();                                     // (the others' shared memory is read until all are here)
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      marks[i] = odd_w[i];
      marks[4 + i] = odd_x[i];
    }
  }
  uint32_t any = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) any |= marks[i];
  if (any == 0) return;
  auto marked = [&](int base, int i) {
    uint32_t w = 0;
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (x == i / 32) w = marks[base + x];
    return w >> (i % 32) & 1;
  };
  for (int e = j0 * TILE + threadIdx.x; e < j1 * TILE; e += THREADS) {
    const int i = e % TILE, j = e / TILE, n = n0 + i, m = m0 + j;
    if (n >= p.N || m >= p.M || !(marked(0, i) | marked(4, j))) continue;
    const float *a = p.A + (int64_t)m * p.lda, *w = p.W + (int64_t)n * p.K;
    float even = 0.f, uneven = 0.f;                         // (two sums, as gemm_f32.cu's tiles form them)
    for (int k = 0; k < p.K; k += 2) {
      even = fmaf(a[k], w[k], even);
      if (k + 1 < p.K) uneven = fmaf(a[k + 1], w[k + 1], uneven);
    }
    p.C[(int64_t)m * p.ldc + n] = even + uneven + (p.bias ? p.bias[n] : 0.f);
  }
}

// Sums over parts of K that make an output: four, which four CTAs may take, but one up to four stages, whose sums are added in the same
// order so.  us in one part and in the better form of four, K 256, N 4,096: 1 row 8.7, 8.6; 64 rows 11.6, 10.1; 128 rows 12.2, 12.7;
// 1,030 rows 23, 28.  (One for K up to 1,024 and tall matrices is faster too, N 12,288, 1,030 rows: K 512 87, 98, K 1,024 135, 154; but its
// error against 64 bits is larger: K 512 0.96e-7 for 0.92e-7, K 1,024 1.09e-7 for 0.97e-7.)
static int parts_for(int K) { return K <= 4 * KS ? 1 : QUARTERS; }

// CTAs to a tile: four where that takes fewer rounds of the device's SMs (of which clusters of four reach 132), a round being a
// quarter as long but for its start and the meeting of the sums, some ten stages' time against six.  With 128 rows a tile and K 4,096
// that is up to 66 tiles and again from 149 to 165, where one CTA to a tile leaves its second round nearly empty; with up to 32 rows
// (two CTAs an SM) up to 132 tiles and from 297 to 330.  With 64 rows, whose CTAs hold one stage's sums and keep totals in C, a stage takes
// 1.36 times as long: N 12,288 and K 1,280, 1,792: 39 and 58 us with one, 35 and 43 with four; 96 to 400 tiles within 8 % of the better
// one.  us with one and with four: M 128, K 4,096: 66 tiles 88, 62; 100 tiles 90, 107;
// 148 tiles 101, 140; 150 tiles 173, 136; 165 tiles 174, 142; 220 tiles 181, 193; K 9,728: 66 tiles 202, 120; 150 tiles 381, 265; 198
// tiles 433, 388; 250 tiles 452, 474.  M 1, K 4,096: 132 tiles 74, 66; 148 tiles 72, 84; 250 tiles 103, 121; 300 tiles 162, 142.  Where
// it errs it takes one: M 32, K 4,096: 140 tiles 95, 74, 150 tiles 119, 99, 335 tiles 205, 173.
template <int NX>
static int cluster_for(int64_t tiles, int K) {
  const double stages = (K + KS - 1) / KS;
  const double whole = (double)((tiles + 148 * Cfg<NX, BY_TMA>::CTAS - 1) / (148 * Cfg<NX, BY_TMA>::CTAS)) * (NX == 64 ? 1.36 * stages + 8 : stages + 6);
  const double split = (double)((4 * tiles + 132 * Cfg<NX, BY_TMA>::CTAS - 1) / (132 * Cfg<NX, BY_TMA>::CTAS)) * (stages / 4 + 10);
  return split < whole ? QUARTERS : 1;
}

template <int NX, Form FORM>
static int launch(const Params& p, int64_t nt, int64_t mt, const CUtensorMap& map_a, const CUtensorMap& map_w, cudaStream_t stream) {
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_f32_tc_kernel<NX, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<NX, FORM>::SMEM) != cudaSuccess)
      return ATOM_ERR_LAUNCH;
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nt * p.cluster), (unsigned)mt);
  cfg.blockDim = dim3(Cfg<NX, FORM>::THREADS);
  cfg.dynamicSmemBytes = Cfg<NX, FORM>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = atom::pdl_enabled() ? 2 : 1;
  (void)cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel<NX, FORM>, p, map_a, map_w);
  return atom::check_launch();
}

// W's rows that begin anywhere: pieces save memory's time and cost instructions, so up to 64 rows with no more than a CTA an SM the numbers
// come one by one (the rows of a K that is a multiple of 4 lie at one distance, where that is slow).  us in pieces and so,
// K 4,097: N 1,024 (32 CTAs) 1 row 42, 34; 17 rows 53, 38; 64 rows 59, 43; N 4,096 (128 CTAs) 44, 37; 54, 43; 58, 58; but N 6,144 (192
// CTAs) 53, 59; 58, 64; 74, 151; and K 4,096 beginning 4 bytes on, N 1,024, 28, 79.
template <int NX>
static int pick(Params p, bool by_tma, const CUtensorMap& map_a, const CUtensorMap& map_w, cudaStream_t stream) {
  const int64_t nt = (p.N + TILE - 1) / TILE, mt = (p.M + NX - 1) / NX;
  if (mt > 65535 || nt > (1 << 28)) return ATOM_ERR_ARG;
  p.parts = parts_for(p.K);
  p.cluster = p.parts == QUARTERS ? cluster_for<NX>(nt * mt, p.K) : 1;
  if (by_tma) return launch<NX, BY_TMA>(p, nt, mt, map_a, map_w, stream);
  if constexpr (NX < 128)
    if (p.K % 4 != 0 && nt * mt * p.cluster <= 148) return launch<NX, BY_NUMBER>(p, nt, mt, map_a, map_w, stream);
  return launch<NX, IN_PIECES>(p, nt, mt, map_a, map_w, stream);
}

}  // namespace f32tc
}  // namespace atom

// As atom_gemm_f32 (gemm_f32.cu).  From 65 rows on with scratch, on a 16-byte boundary, for the planes of A and a mark for every row:
// 6 bytes for every number of M rows of whole stages, and 4 a row.  K < 2^24 (offsets inside a tile are 32-bit).
ATOM_EXPORT int atom_gemm_f32_tc(float* C, const float* A, const float* W, const float* bias, int M, int N, int K, int64_t lda,
                                 int64_t ldc, void* scratch, int64_t scratch_bytes, int* error, cudaStream_t stream) {
  using namespace atom::f32tc;
  if (M <= 0 || N <= 0) return ATOM_OK;
  if (K <= 0 || K >= 1 << 24 || lda < K || lda >= 1 << 24 || ldc < N || error == nullptr ||
      (M > 64 && (scratch == nullptr || ((uintptr_t)scratch % 16) != 0 || scratch_bytes < (6 * (int64_t)((K + 63) / 64 * 64) + 4) * M)))
    return ATOM_ERR_ARG;
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A % 16) == 0, by_tma = K % 4 == 0 && K >= HALF && ((uintptr_t)W % 16) == 0;
  Params p{C, A, W, bias, lda, ldc, M, N, K, vec, 1, 1, nullptr, error};
  CUtensorMap map{}, map_w{};
  // (W as twice as many 16-bit numbers: a box of 64 is 32 of its numbers)
  if (by_tma && !atom::tma::cached_map(&map_w, W, (uint64_t)N, 2 * (uint64_t)K, 2 * (uint64_t)K, TILE)) return ATOM_ERR_LIB;
  if (M <= 16) return pick<16>(p, by_tma, map, map_w, stream);
  if (M <= 32) return pick<32>(p, by_tma, map, map_w, stream);
  if (M <= 64) return pick<64>(p, by_tma, map, map_w, stream);
  const int Kp = (K + 63) / 64 * 64;
  __nv_bfloat16* planes = (__nv_bfloat16*)scratch;
  int* odd = (int*)(planes + 3 * (int64_t)M * Kp);
  p.odd_rows = odd;
  if (!atom::tma::cached_map(&map, planes, 3 * (uint64_t)M, Kp, Kp, 128)) return ATOM_ERR_LIB;
  atom::launch_pdl(f32_rows_kernel, dim3(M), dim3(256), 0, stream, planes, odd, A, lda, K, Kp, (int)vec);
  return pick<128>(p, by_tma, map, map_w, stream);
}
