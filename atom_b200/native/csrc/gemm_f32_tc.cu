// The 32-bit matrix product C[M, N] = A[M, K] W[N, K]^T (+ bias) of many rows on tcgen05.  Every number enters as THREE
// bfloat16 numbers that hold all 24 bits of its mantissa (eight each, cut off), in the six products down to 2^-16 of the
// largest, smallest first; the sums of 64 k's are formed in tensor memory and added up in 32-bit registers, because the tensor
// cores cut off what a long sum cannot hold.  Against 64-bit the result is nearer than one sequential 32-bit sum over K (4,096
// normal numbers: see the test), so this is no reduced-precision mode.
//
// f32_planes_kernel lays the three planes of a matrix out, rows padded with zeros to whole blocks of 64; W goes through in
// slabs of output columns whose planes stay in L2 and whose tiles are about one per SM (so a matrix of any height needs a
// bounded workspace).  gemm_f32_tc_kernel: a CTA per 128 x 128 tile; warp 0 loads a stage (six blocks of 128 x 64: the
// planes of A and W) with TMA, warp 1 issues 24 MMAs of 128 x 128 x 16 a stage, warps 2-5 add the finished sums of the stage
// before to their 128 numbers a thread (tensor memory holds two tiles of sums).  Bound by shared memory: a stage's MMAs read
// 192 KB of it and TMA writes 96 KB.  1,030 rows, N 6,144, K 4,096: 2,550 us for 4 x 4 outputs a thread on the FMA units, 1,290
// for 8 x 8 of them, 260 here with the planes (K 4,096, N 4,096: 1,720, 870, 190); 64-bit error 1.1e-6, 0.8e-6, 0.3e-6.
//
// A number that is not finite has no such planes: f32_planes_kernel raises a flag when it meets one, and the product is then
// computed again on the FMA units (gemm_f32.cu), by a kernel that otherwise returns at once.
#include "gemm_f32.cuh"
#include "tcgen05.cuh"

namespace atom {
namespace f32tc {

using namespace atom::tma;
using namespace atom::tc5;

constexpr int TILE = 128, BLK = TILE * 64 * 2, STAGE = 6 * BLK, STAGES = 2, THREADS = 192, EPI_WARPS = 4;

struct Bars {
  uint64_t full[STAGES], done[STAGES], taken[STAGES];
  uint32_t tmem;
  int aborted;
};
constexpr size_t SMEM = 1024 + STAGES * STAGE + 256;
static_assert(SMEM <= 227 * 1024, "shared memory");

struct Params {
  float* C;
  const float* bias;
  int64_t ldc;
  int M, N, Kp;       // N: columns of this slab; Kp: K in whole blocks of 64
  int rows_a, rows_w; // rows between the planes of A and of the slab of W
  int* error;
};

constexpr uint32_t kInstr = instr_desc(TILE, TILE, false);

// planes [3][R][Kp] <- x [R, K] (rows ld apart): eight numbers a thread.  vec: rows begin on 16-byte boundaries and K % 4 == 0.
__global__ void __launch_bounds__(256) f32_planes_kernel(__nv_bfloat16* __restrict__ planes, const float* __restrict__ x, int64_t ld,
                                                          int R, int K, int Kp, int vec, int* __restrict__ odd) {
  atom::pdl_trigger();
  atom::pdl_wait();
  const int64_t total = (int64_t)R * (Kp / 8), size = (int64_t)R * Kp;
  bool bad = false;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / (Kp / 8);
    const int k = (int)(e - r * (Kp / 8)) * 8;
    const float* src = x + r * ld + k;
    float v[8];
    if (vec) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 f = k + 4 * h < K ? *reinterpret_cast<const float4*>(src + 4 * h) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * h] = f.x;
        v[4 * h + 1] = f.y;
        v[4 * h + 2] = f.z;
        v[4 * h + 3] = f.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = k + i < K ? src[i] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) bad |= (__float_as_uint(v[i]) & 0x7f800000u) == 0x7f800000u;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        w[i] = __byte_perm(__float_as_uint(v[2 * i]), __float_as_uint(v[2 * i + 1]), 0x7632);
        v[2 * i] -= __uint_as_float(__float_as_uint(v[2 * i]) & 0xffff0000u);
        v[2 * i + 1] -= __uint_as_float(__float_as_uint(v[2 * i + 1]) & 0xffff0000u);
      }
      *reinterpret_cast<uint4*>(planes + m * size + r * Kp + k) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  if (bad) *odd = 1;
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapW, const Params p) {
  atom::pdl_trigger();
  atom::pdl_wait();
  extern __shared__ unsigned char smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  Bars* bars = reinterpret_cast<Bars*>(smem_raw + (sbase - smem_u32(smem_raw)) + STAGES * STAGE);
  volatile int* aborted = &bars->aborted;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * TILE, n0 = blockIdx.x * TILE, KT = p.Kp / 64;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->done[s], 1);
      mbar_init(&bars->taken[s], EPI_WARPS);
    }
    bars->aborted = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&bars->tmem, 2 * TILE);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem;

  if (warp == 0) {
    if (lane == 0) {
      prefetch_map(&mapA);
      prefetch_map(&mapW);
      for (int it = 0; it < KT; ++it) {
        const int s = it % STAGES;
        if (it >= STAGES) mbar_wait(&bars->done[s], ((it / STAGES) - 1) & 1, aborted, p.error);
        mbar_expect_tx(&bars->full[s], STAGE);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          load_box(nullptr, &mapA, it * 64, m * p.rows_a + m0, &bars->full[s], sbase + s * STAGE + m * BLK);
          load_box(nullptr, &mapW, it * 64, m * p.rows_w + n0, &bars->full[s], sbase + s * STAGE + (3 + m) * BLK);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PW[6] = {0, 1, 2, 0, 1, 0};
      for (int it = 0; it < KT; ++it) {
        const int s = it % STAGES;
        mbar_wait(&bars->full[s], (it / STAGES) & 1, aborted, p.error);
        if (it >= STAGES) mbar_wait(&bars->taken[s], ((it / STAGES) - 1) & 1, aborted, p.error);
        tc_fence_after();
        const uint32_t base = sbase + s * STAGE;
#pragma unroll
        for (int x = 0; x < 6; ++x) {
          const uint64_t a = smem_desc(base + PA[x] * BLK, 16, 1024), w = smem_desc(base + (3 + PW[x]) * BLK, 16, 1024);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) umma(tmem + s * TILE, a + 2 * ks, w + 2 * ks, kInstr, x + ks > 0);
        }
        umma_commit(&bars->done[s]);
      }
    }
  } else {
    const int q = warp & 3, row = m0 + 32 * q + lane;      // (a warp reads the quarter of the lanes that its index selects)
    const uint32_t tbase = tmem + ((uint32_t)(32 * q) << 16);
    float acc[TILE];
#pragma unroll
    for (int i = 0; i < TILE; ++i) acc[i] = 0.f;
    for (int it = 0; it < KT; ++it) {
      const int s = it % STAGES;
      mbar_wait(&bars->done[s], (it / STAGES) & 1, aborted, p.error);
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < TILE; c += 32) {
        float v[32];
        tmem_ld32(tbase + s * TILE + c, v);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[c + i] += v[i];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->taken[s]);
    }
    if (row < p.M) {
      float* dst = p.C + (int64_t)row * p.ldc + n0;
      const bool vec = p.ldc % 4 == 0 && ((uintptr_t)p.C % 16) == 0;
#pragma unroll
      for (int c = 0; c < TILE; c += 4) {
        if (p.bias) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (n0 + c + i < p.N) acc[c + i] += p.bias[n0 + c + i];
        }
        if (vec && n0 + c + 4 <= p.N) {
          *reinterpret_cast<float4*>(dst + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (n0 + c + i < p.N) dst[c + i] = acc[c + i];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 2 * TILE);
}

// Columns of a slab: as many tiles as the row tiles leave SMs for, their planes within `bytes`; at least one tile.
static int slab_columns(int M, int N, int Kp, int64_t bytes) {
  const int mt = (M + TILE - 1) / TILE;
  int64_t tiles = 148 / mt > 1 ? 148 / mt : 1;
  const int64_t room = bytes / ((int64_t)6 * Kp * TILE);
  if (tiles > room) tiles = room;
  const int64_t all = (N + TILE - 1) / TILE;
  if (tiles > all) tiles = all;
  return (int)tiles * TILE;
}

static void planes_of(__nv_bfloat16* planes, const float* x, int64_t ld, int R, int K, int Kp, int* odd, cudaStream_t stream) {
  const int vec = K % 4 == 0 && ld % 4 == 0 && ((uintptr_t)x % 16) == 0;
  const int64_t total = (int64_t)R * (Kp / 8);
  const int blocks = (int)(total / 256 + 1 < 148 * 8 ? total / 256 + 1 : 148 * 8);
  atom::launch_pdl(f32_planes_kernel, dim3(blocks), dim3(256), 0, stream, planes, x, ld, R, K, Kp, vec, odd);
}

}  // namespace f32tc
}  // namespace atom

// As atom_gemm_f32 (gemm_f32.cu), with a workspace of `ws_bytes` on a 1024-byte boundary.  Launches: *launches kernels.
ATOM_EXPORT int atom_gemm_f32_tc(float* C, const float* A, const float* W, const float* bias, int M, int N, int K, int64_t lda,
                                 int64_t ldc, void* ws, int64_t ws_bytes, int* error, int* launches, cudaStream_t stream) {
  using namespace atom::f32tc;
  *launches = 0;
  if (M <= 0 || N <= 0) return ATOM_OK;
  if (K <= 0 || lda < K || ldc < N || ws == nullptr || error == nullptr || ((uintptr_t)ws % 1024) != 0) return ATOM_ERR_ARG;
  const int Kp = (K + 63) / 64 * 64;
  // | flag | planes of A | planes of a slab of W |
  const int64_t head = 1024 + (6 * (int64_t)M * Kp + 1023) / 1024 * 1024;
  const int slab = slab_columns(M, N, Kp, ws_bytes - head);
  if (slab < TILE || (M + TILE - 1) / TILE > 65535) return ATOM_ERR_ARG;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) != cudaSuccess) return ATOM_ERR_LAUNCH;
    attr_set = true;
  }
  int* odd = (int*)ws;
  __nv_bfloat16* pa = (__nv_bfloat16*)((char*)ws + 1024);
  __nv_bfloat16* pw = (__nv_bfloat16*)((char*)ws + head);
  CUtensorMap ma, mw;
  if (!atom::tma::cached_map(&ma, pa, 3 * (uint64_t)M, Kp, Kp, TILE)) return ATOM_ERR_LIB;
  if (cudaMemsetAsync(odd, 0, sizeof(int), stream) != cudaSuccess) return ATOM_ERR_LAUNCH;
  planes_of(pa, A, lda, M, K, Kp, odd, stream);
  ++*launches;
  for (int n0 = 0; n0 < N; n0 += slab) {
    const int cols = N - n0 < slab ? N - n0 : slab;
    planes_of(pw, W + (int64_t)n0 * K, K, cols, K, Kp, odd, stream);
    if (!atom::tma::cached_map(&mw, pw, 3 * (uint64_t)cols, Kp, Kp, TILE)) return ATOM_ERR_LIB;
    Params p{C + n0, bias ? bias + n0 : nullptr, ldc, M, cols, Kp, M, cols, error};
    atom::launch_pdl(gemm_f32_tc_kernel, dim3((cols + TILE - 1) / TILE, (M + TILE - 1) / TILE), dim3(THREADS), SMEM, stream, ma, mw, p);
    *launches += 2;
  }
  const int rc = atom::check_launch();
  if (rc != ATOM_OK) return rc;
  ++*launches;
  return atom::gemm_f32(atom::GemmF32{C, A, W, bias, M, N, K, lda, ldc, 0, 0, 0, odd}, 1, stream);
}
