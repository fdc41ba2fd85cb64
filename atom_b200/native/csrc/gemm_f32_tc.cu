// The 32-bit matrix product C[M, N] = A[M, K] W[N, K]^T (+ bias) on tcgen05.  Every number enters as THREE bfloat16 numbers, each
// what is left rounded to nearest, that hold all 24 bits of its mantissa, in the six products down to 2^-16 of the largest, smallest
// first; the sums of 64 k's are formed in tensor memory and added up in 32-bit registers, because the tensor cores cut off what a
// long sum cannot hold.  Against 64-bit the result is nearer than one sequential 32-bit sum over K (4,096 normal numbers: see the
// test), so this is no reduced-precision mode.
//
// A row's result does not depend on which other rows share the launch: W's rows are always the 128 rows of an MMA and A's its
// columns, 16 to 128 of them by M, and an output's sums run in one order over K whatever that width.
//
// A CTA per tile of 128 columns of C and NX rows, in stages of 64 k's.  Warps 0-15 load groups of eight numbers two stages ahead,
// split them and write the planes in the layout that the MMAs read; warp 24 issues 24 MMAs of 128 x NX x 16 a stage; warps 16-23 add
// the finished sums of the stage before to their NX / 2 numbers a thread (tensor memory holds two tiles of sums).  Up to 64 rows the
// CTA splits A's too; beyond that f32_rows_kernel has laid their planes out (every column tile would split them again) and warp 25
// fetches them with TMA.  With few rows bound by the MMAs' reads of W's planes, some 90 clocks each whatever their width, with 128 by
// shared memory.  us at K 4,096 and N 6,144 / 4,096: 1 row 82 / 81 (on the FMA units 51 / 39), 32 rows 86 / 85 (98 / 66), 64 rows 101 /
// 100 (141 / 125), 1,030 rows 310 / 210 (1,298 / 881; with W's planes laid out by a kernel of their own, too, 510 for the two).
//
// A number that three bfloat16 numbers do not hold (not finite, beyond their range, or with bits below 2^-133) marks its row: the
// outputs of marked rows of A and W are formed again in 32-bit as gemm_f32.cu does, an output by one thread.
#include "gemm_f32.cuh"
#include "tcgen05.cuh"

namespace atom {
namespace f32tc {

using namespace atom::tma;
using namespace atom::tc5;

constexpr int TILE = 128, KS = 64, BLK_W = TILE * 128;      // rows of W, k's of a stage, bytes of a plane of W
constexpr int SPLIT_WARPS = 16, SUM_WARPS = 8, MMA_WARP = SPLIT_WARPS + SUM_WARPS, LOAD_WARP = MMA_WARP + 1,
              THREADS = (LOAD_WARP + 1) * 32;

constexpr int WI = TILE * 8 / (SPLIT_WARPS * 32);           // groups of eight of W a thread

template <int NX>
struct Cfg {
  static constexpr bool PRE = NX == 128;                    // A's planes come from memory
  static constexpr int BLK_X = NX * 128, STAGE = 3 * (BLK_W + BLK_X), STAGES = NX == 128 ? 2 : (NX == 16 ? 4 : 3);
  static constexpr int G = WI + (PRE ? 0 : 1);              // groups of eight a thread: of W, one of A
  static constexpr int COLS = NX / 2;                       // sums of a thread
  static constexpr size_t SMEM = 1024 + (size_t)STAGES * STAGE;
  static_assert(SMEM + 1024 <= 227 * 1024, "shared memory");
};

struct Params {
  float* C;
  const float *A, *W, *bias;
  int64_t lda, ldc;
  int M, N, K, vec;         // vec: rows of A and W begin on 16-byte boundaries and hold whole 16-byte pieces
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
// N (8 or 16) consecutive 32-bit columns of this thread's lane.
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  if constexpr (N == 8)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
  else
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
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

template <int NX>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tc_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap map_a) {
  atom::pdl_trigger();
  atom::pdl_wait();
  using C = Cfg<NX>;
  constexpr int STAGES = C::STAGES, COLS = C::COLS;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t full[STAGES], empty[STAGES], done[2], taken[2];
  __shared__ uint32_t tmem_base, odd_w[TILE / 32], odd_x[4];
  __shared__ int aborted_flag;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  volatile int* aborted = &aborted_flag;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (known to be uniform)
  const int n0 = blockIdx.x * TILE, m0 = blockIdx.y * NX, KT = (p.K + KS - 1) / KS;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], SPLIT_WARPS + (C::PRE ? 1 : 0));
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&done[s], 1);
      mbar_init(&taken[s], SUM_WARPS);
    }
    for (int i = 0; i < 4; ++i) odd_w[i] = odd_x[i] = 0;
    aborted_flag = 0;
    mbar_fence_init();
  }
  if (warp == MMA_WARP) tmem_alloc(&tmem_base, 2 * NX);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;

  if (warp < SPLIT_WARPS) {
    // eight neighbouring threads hold a row's 64 numbers of the stage
    const int row = threadIdx.x >> 3, ch = threadIdx.x & 7;
    constexpr int STEP = SPLIT_WARPS * 32 / 8;              // rows between a thread's groups
    const bool x_on = !C::PRE && row < NX;
    constexpr int G = C::G;
    // rows behind the last one repeat it (their outputs are not written); where a group begins, from the tile's first row on
    const float *wt = p.W + (int64_t)n0 * p.K, *xt = p.A + (int64_t)m0 * p.lda;
    uint32_t at[G];
#pragma unroll
    for (int i = 0; i < WI; ++i) at[i] = (uint32_t)min(row + i * STEP, p.N - 1 - n0) * (uint32_t)p.K + ch * 8;
    if (!C::PRE) at[G - 1] = (uint32_t)min(row, p.M - 1 - m0) * (uint32_t)p.lda + ch * 8;
    float v[2][G][8];
    auto load = [&](float (&to)[G][8], int it) {
      const int k = min(it, KT - 1) * KS;                   // (behind the last stage it comes again: no branch)
      const bool whole = p.vec && k + KS <= p.K;
#pragma unroll
      for (int i = 0; i < G; ++i)
        if (i < WI || x_on) load_group(to[i], (i < WI ? wt : xt) + k + at[i], whole, k + ch * 8, p.K);
    };
    // W comes from memory: its lines are asked for AHEAD stages before they are split
    constexpr int AHEAD = 6;
    const float* line = wt + (int64_t)min((int)(threadIdx.x & 255) >> 1, p.N - 1 - n0) * p.K + (threadIdx.x & 1) * 32;
    auto ask = [&](int it) {
      if (threadIdx.x < 256 && it * KS + (int)(threadIdx.x & 1) * 32 < p.K) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(line + it * KS));
    };
#pragma unroll
    for (int it = 2; it < AHEAD; ++it) ask(it);
    load(v[0], 0);
    load(v[1], 1);
    uint32_t bad = 0;                                       // bit i: group i did not fit its planes
    auto split = [&](float (&from)[G][8], int it) {
      const int s = it % STAGES;
      if (it >= STAGES) mbar_wait(&empty[s], ((it / STAGES) - 1) & 1, aborted, p.error);
      const uint32_t base = sbase + s * C::STAGE + row * 128 + ((ch ^ (row & 7)) << 4);
      ask(it + AHEAD);
#pragma unroll
      for (int i = 0; i < G; ++i)
        if (i < WI || x_on) {
          const bool odd = i < WI ? store_planes(from[i], base + i * STEP * 128, BLK_W) : store_planes(from[i], base + 3 * BLK_W, C::BLK_X);
          if (odd) bad |= 1u << i;
        }
      load(from, it + 2);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[s]);
    };
#pragma unroll 1
    for (int it = 0; it < KT; it += 2) {
      split(v[0], it);
      if (it + 1 < KT) split(v[1], it + 1);
    }
    if (bad) {
#pragma unroll
      for (int i = 0; i < WI; ++i)
        if (bad >> i & 1) atomicOr(&odd_w[(row + i * STEP) / 32], 1u << ((row + i * STEP) % 32));
      if (!C::PRE && (bad >> WI & 1)) atomicOr(&odd_x[row / 32], 1u << (row % 32));
    }
  } else if (C::PRE && warp == LOAD_WARP) {
    if (lane == 0) {
      for (int it = 0; it < KT; ++it) {
        const int s = it % STAGES;
        if (it >= STAGES) mbar_wait(&empty[s], ((it / STAGES) - 1) & 1, aborted, p.error);
        mbar_expect_tx(&full[s], 3 * C::BLK_X);
#pragma unroll
        for (int m = 0; m < 3; ++m)
          load_box(nullptr, &map_a, it * KS, m * p.M + m0, &full[s], sbase + s * C::STAGE + 3 * BLK_W + m * C::BLK_X);
      }
    }
    __syncwarp();
    for (int i = lane; i < NX; i += 32)
      if (m0 + i < p.M && p.odd_rows[m0 + i]) atomicOr(&odd_x[i / 32], 1u << (i % 32));
  } else if (warp == MMA_WARP) {
    // The whole warp runs the loop, so that descriptors stay in uniform registers; one thread issues.
    constexpr int PX[6] = {2, 1, 0, 1, 0, 0}, PW[6] = {0, 1, 2, 0, 1, 0};
    constexpr uint32_t idesc = instr_desc(TILE, NX, false);
    const uint64_t desc = smem_desc(sbase, 16, 1024);
    const bool one = elect_one();
    for (int it = 0; it < KT; ++it) {
      const int s = it % STAGES, d = it & 1;
      mbar_wait(&full[s], (it / STAGES) & 1, aborted, p.error);
      if (it >= 2) mbar_wait(&taken[d], ((it >> 1) - 1) & 1, aborted, p.error);
      tc_fence_after();
      const uint64_t base = desc + (uint32_t)(s * (C::STAGE >> 4));
      if (one) {
#pragma unroll
        for (int x = 0; x < 6; ++x)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma(tmem + d * NX, base + (uint32_t)((PW[x] * BLK_W >> 4) + 2 * ks), base + (uint32_t)(((3 * BLK_W + PX[x] * C::BLK_X) >> 4) + 2 * ks), idesc,
                     x + ks > 0);
        umma_commit(&empty[s]);
        umma_commit(&done[d]);
      }
      __syncwarp();
    }
  } else if (warp < MMA_WARP) {
    const int q = warp & 3, half = (warp - SPLIT_WARPS) >> 2;      // (a warp reads the quarter of the lanes that its index selects)
    const uint32_t tbase = tmem + ((uint32_t)(32 * q) << 16) + half * COLS;
    float acc[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
    for (int it = 0; it < KT; ++it) {
      const int d = it & 1;
      mbar_wait(&done[d], (it >> 1) & 1, aborted, p.error);
      tc_fence_after();
      constexpr int LD = 8;
#pragma unroll
      for (int c = 0; c < COLS; c += LD) {
        float v[LD];
        tmem_ld<LD>(tbase + d * NX + c, v);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < LD; ++i) acc[c + i] += v[i];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&taken[d]);
    }
    const int n = n0 + 32 * q + lane;
    if (n < p.N && !*aborted) {
      const float b = p.bias ? p.bias[n] : 0.f;
#pragma unroll
      for (int i = 0; i < COLS; ++i) {
        const int m = m0 + half * COLS + i;
        if (m < p.M) p.C[(int64_t)m * p.ldc + n] = acc[i] + b;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem, 2 * NX);
  uint32_t any = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) any |= odd_w[i] | odd_x[i];
  if (any == 0) return;
  for (int e = threadIdx.x; e < TILE * NX; e += THREADS) {
    const int i = e % TILE, j = e / TILE, n = n0 + i, m = m0 + j;
    if (n >= p.N || m >= p.M || !((odd_w[i / 32] >> (i % 32) & 1) | (odd_x[j / 32] >> (j % 32) & 1))) continue;
    const float *a = p.A + (int64_t)m * p.lda, *w = p.W + (int64_t)n * p.K;
    float even = 0.f, uneven = 0.f;                         // (two sums, as gemm_f32.cu's tiles form them)
    for (int k = 0; k < p.K; k += 2) {
      even = fmaf(a[k], w[k], even);
      if (k + 1 < p.K) uneven = fmaf(a[k + 1], w[k + 1], uneven);
    }
    p.C[(int64_t)m * p.ldc + n] = even + uneven + (p.bias ? p.bias[n] : 0.f);
  }
}

template <int NX>
static int launch(const Params& p, const CUtensorMap& map_a, cudaStream_t stream) {
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_f32_tc_kernel<NX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<NX>::SMEM) != cudaSuccess)
      return ATOM_ERR_LAUNCH;
    attr_set = true;
  }
  const dim3 grid((p.N + TILE - 1) / TILE, (p.M + NX - 1) / NX);
  if (grid.y > 65535) return ATOM_ERR_ARG;
  atom::launch_pdl(gemm_f32_tc_kernel<NX>, grid, dim3(THREADS), Cfg<NX>::SMEM, stream, p, map_a);
  return atom::check_launch();
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
  const int vec = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) % 16) == 0;
  Params p{C, A, W, bias, lda, ldc, M, N, K, vec, nullptr, error};
  CUtensorMap map{};
  if (M <= 16) return launch<16>(p, map, stream);
  if (M <= 32) return launch<32>(p, map, stream);
  if (M <= 64) return launch<64>(p, map, stream);
  const int Kp = (K + 63) / 64 * 64;
  __nv_bfloat16* planes = (__nv_bfloat16*)scratch;
  int* odd = (int*)(planes + 3 * (int64_t)M * Kp);
  p.odd_rows = odd;
  if (!atom::tma::cached_map(&map, planes, 3 * (uint64_t)M, Kp, Kp, 128)) return ATOM_ERR_LIB;
  atom::launch_pdl(f32_rows_kernel, dim3(M), dim3(256), 0, stream, planes, odd, A, lda, K, Kp, vec);
  return launch<128>(p, map, stream);
}
