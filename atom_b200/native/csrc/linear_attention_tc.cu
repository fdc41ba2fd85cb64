// Matrix-state recurrences over long portions in bfloat16, in chunks of 64 rows on the tensor cores:
//   S_t = diag(a_t) S_(t-1) + k_t v_t^T   per head, with
//   LT    one constant decay per head, q, k, v = silu(.) of the projection;           o_t = S_t^T q_t
//   GLA   a_t = sigmoid(z_t + b)^(1 / tau) per key channel;                            o_t = S_t^T (q_t q_scale)
//   WKV   a_t = exp(-exp(d_t + w0)) per key channel, a bonus for the present token;   o_t = (S_(t-1) + diag(u) k_t v_t^T)^T r_t,
//         then o / rms(o) * w * silu(gate), written in bfloat16
// In three launches, the chunks of all requests side by side in the first and the last:
//   la_chunk_sum_kernel   B = sum_j 2^(G_end - G_j) k_j v_j^T of every chunk, the chunk's decays, the logarithms' sums G
//   la_prefix_kernel      the state every chunk begins with (in B's place), over a request's chunks in order
//   la_chunk_out_kernel   o_i = (2^(G_i) q_i) S_begin + sum_(j <= i) (sum_c q_i k_j 2^(G_i - G_j)) v_j
// G is the sum of the decays' base-2 logarithms from a chunk's first row on, per key channel.  It is kept as sums within
// blocks of 16 rows and over whole blocks, so that 2^(G_i - G_j) of rows in different blocks is 2^(sum from i's block on)
// times 2^(sum from j's next row to the block before), two factors of at most one.  Within a block the reference is the
// eighth row of the block: rows before it and columns behind it take the inverse factor, which stays below 2^80 or the
// half block's pairs are formed one by one.  Where a block's sum lies below -640 in some channel (a decay of zero among them)
// differences of the sums lose what the decays hold, and the chunk is walked row by row from the state it begins with
// (walk_chunk); the chunks' sums of keys and values take any decay.
//
// Every 32-bit operand (decayed q and k, silu's values, the state, the pair sums) enters its products as THREE bfloat16
// numbers, each what is left rounded to nearest, that hold all 24 bits of its mantissa, in the six products down to 2^-16 of
// the largest (three where the other operand is bfloat16 already); the sums are 32-bit.  (Dot products of 64 normal numbers in
// steps of 16: 6.3e-8 from 64-bit; 1.07e-7 where the three are cut off instead; one sequential 32-bit sum 1.4e-7.)  Powers of a
// constant decay are formed in 64-bit.
//
// Rows that a row does not see enter its products with a weight of zero, which a number that is not finite turns into NaN: a
// chunk with an output that is not finite is walked too, so that no row depends on later ones.
//
// Why chunks: the walk row by row (lightning.cu, gla.cu, wkv.cu) is bound by 32-bit multiply-adds and shared-memory loads per
// state element and row, twice over the rows.  A chunk costs 2 dk + 64 multiply-adds per row and value column on the tensor
// cores instead, and the states of the chunk borders (dk * dv numbers per 64 rows and head) stay in L2.  At 2,048 rows of two
// or three requests, 16 heads of 128 x 128 (WKV: 32 heads of 64 x 64), plain launches: LT 424 -> 115 us, GLA 543 -> 104 us,
// WKV 541 -> 103 us.  LT's sums run in two numbers each (mma_six with a rest): 0.82e-7 from 64-bit at 2,048 rows of 16 heads
// (1.3e-7 in one number, 0.85e-7 walked), for 142 us.
#include "common.cuh"

namespace atom {
namespace latc {

constexpr int LT = 0, GLA = 1, WKV = 2;
constexpr int L = 64, THREADS = 256;              // rows of a chunk, threads of a CTA
constexpr int LP = L + 8;                         // bf16 elements per row of the pairs' sums
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kStrong = -80.f, kWalk = -640.f;

__device__ __forceinline__ void ldm_x4(uint32_t (&r)[4], const void* smem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void ldm_x4_trans(uint32_t (&r)[4], const void* smem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// d = a b
__device__ __forceinline__ void mma_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float2 unpack(uint32_t x) {
  return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
}
__device__ __forceinline__ uint32_t pack(float x, float y) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&b);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// Two numbers as three pairs of bfloat16 numbers, x = p[0] + p[1] + p[2].
__device__ __forceinline__ void split3(float x, float y, uint32_t (&p)[3]) {
  float2 v = make_float2(x, y);
  p[0] = pack(v.x, v.y);
  v = sub2(v, unpack(p[0]));
  p[1] = pack(v.x, v.y);
  v = sub2(v, unpack(p[1]));
  p[2] = pack(v.x, v.y);
}
__device__ __forceinline__ float power(float x, int n) {
  double r = 1., b = x;
  for (; n > 0; n >>= 1) {
    if (n & 1) r *= b;
    b *= b;
  }
  return (float)r;
}
// d[i] += a[i] b[i] over the planes of both, the smallest products first.  The tensor cores cut off what a sum cannot hold
// instead of rounding it, so a step of 16 is summed up by itself and added in 32-bit; the products of one accumulator stand
// apart.
template <int N>
__device__ __forceinline__ void mma_six(float (*const (&d)[N])[4], const uint32_t (*const (&a)[N])[4], const uint32_t (*const (&b)[N])[2]) {
  constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};
  float t[N][4];
#pragma unroll
  for (int i = 0; i < N; ++i) mma_first(t[i], a[i][2], b[i][0][0], b[i][0][1]);
#pragma unroll
  for (int x = 1; x < 6; ++x)
#pragma unroll
    for (int i = 0; i < N; ++i) mma_bf16(t[i], a[i][PA[x]], b[i][PB[x]][0], b[i][PB[x]][1]);
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) (*d[i])[e] += t[i][e];
}
// The same with a sum in two numbers, d + r: the five small products run up in r, and so does what d loses when a step's large
// one is added to it.
template <int N>
__device__ __forceinline__ void mma_six(float (*const (&d)[N])[4], float (*const (&r)[N])[4], const uint32_t (*const (&a)[N])[4],
                                        const uint32_t (*const (&b)[N])[2]) {
  constexpr int PA[5] = {2, 1, 0, 1, 0}, PB[5] = {0, 1, 2, 0, 1};
  float t[N][4];
#pragma unroll
  for (int i = 0; i < N; ++i) mma_first(t[i], a[i][0], b[i][0][0], b[i][0][1]);
#pragma unroll
  for (int x = 0; x < 5; ++x)
#pragma unroll
    for (int i = 0; i < N; ++i) mma_bf16(*r[i], a[i][PA[x]], b[i][PB[x]][0], b[i][PB[x]][1]);
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = (*d[i])[e], sum = x + t[i][e], got = sum - x;
      (*r[i])[e] += (x - (sum - got)) + (t[i][e] - got);
      (*d[i])[e] = sum;
    }
}
// The same where b is bfloat16 as it is.
template <int N>
__device__ __forceinline__ void mma_three(float (*const (&d)[N])[4], const uint32_t (*const (&a)[N])[4], const uint32_t (&b)[N][2]) {
  float t[N][4];
#pragma unroll
  for (int i = 0; i < N; ++i) mma_first(t[i], a[i][2], b[i][0], b[i][1]);
#pragma unroll
  for (int x = 1; x >= 0; --x)
#pragma unroll
    for (int i = 0; i < N; ++i) mma_bf16(t[i], a[i][x], b[i][0], b[i][1]);
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) (*d[i])[e] += t[i][e];
}

struct Params {
  const __nv_bfloat16 *q, *k, *v;   // rows of H dk, H dk, H dv columns, ld, ld and ldv elements apart
  int64_t ld, ldv;
  const float* z;                   // [T, H dk] at stride ldz: what the decays are formed from (GLA, WKV)
  int64_t ldz;
  const void* zb;                   // [H dk]
  int zb_dtype;
  float inv_tau, q_scale;
  const float* decay;               // [H] (LT)
  const void *u, *norm_w;           // [H dk], [H dv] (WKV), of the type of zb
  const __nv_bfloat16* gate;        // rows as v (WKV)
  __nv_bfloat16* y;                 // [T, H dv] (WKV)
  float eps;
  float* out;                       // [T, H dv]
  float* state;                     // [slots, H, dk, dv]
  float* g;                         // [T, H dk]: sums of the logarithms from the row's block of 16 rows on (GLA, WKV)
  float* sB;                        // [chunks, H, dk, dv]
  float* sA;                        // [chunks, H, dk]
  const int* cu_q;
  const int* state_slots;
  int num_seqs, H, dk, dv, write_state;
};

// Chunk x -> request and chunk number: requests take ceil(len / L) chunks one after another.
__device__ __forceinline__ bool find_chunk(int x, const int* __restrict__ cu_q, int num_seqs, int& s, int& r) {
  int acc = 0;
  for (s = 0; s < num_seqs; ++s) {
    const int n = (cu_q[s + 1] - cu_q[s] + L - 1) / L;
    if (x < acc + n) {
      r = x - acc;
      return true;
    }
    acc += n;
  }
  return false;
}

// The base-2 logarithm of a decay.
template <int MODE>
__device__ __forceinline__ float log_decay(float x, float inv_tau) {
  return MODE == GLA ? (fminf(x, 0.f) - log1pf(expf(-fabsf(x)))) * (inv_tau * kLog2e) : -expf(x) * kLog2e;
}

// 64 rows x VT columns of values: as they are, or (LT) silu's values in three planes; rows of VT + 8 elements.
template <int MODE, int VT, int TH>
__device__ __forceinline__ void load_values(__nv_bfloat16* Vs, const __nv_bfloat16* __restrict__ v, int64_t ldv, int rows, int cols) {
  constexpr int LDV = VT + 8;
#pragma unroll 4
  for (int e = threadIdx.x; e < L * (VT / 8); e += TH) {
    const int i = e / (VT / 8), c = (e % (VT / 8)) * 8;
    const bool in = i < rows && c < cols;
    if (MODE != LT) {
      cp_async16(Vs + i * LDV + c, v + (in ? (int64_t)i * ldv + c : 0), in);
    } else {
      uint4 raw = make_uint4(0u, 0u, 0u, 0u);
      if (in) raw = *reinterpret_cast<const uint4*>(v + (int64_t)i * ldv + c);
      const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
      uint32_t o[3][4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float2 f = unpack(r[x]);
        uint32_t p[3];
        split3(silu(f.x), silu(f.y), p);
#pragma unroll
        for (int m = 0; m < 3; ++m) o[m][x] = p[m];
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
        *reinterpret_cast<uint4*>(Vs + (m * L + i) * LDV + c) = make_uint4(o[m][0], o[m][1], o[m][2], o[m][3]);
    }
  }
}

// ------------------------------------------------------------------ the chunks' sums

// A CTA of TH / 32 warps: a chunk, a head, VT value columns; a warp owns 16 key channels (or half of the columns of them).
// GLA, WKV: a thread owns two key channels of a block of 16 rows.  Their logarithms and keys are under way together, the
// sums behind every row stay in registers and only the blocks' sums pass through shared memory, so that three CTAs of 256
// threads (or five of 128: up to 64 key channels have no work for more) fit an SM.  (With every row's sums in shared memory
// and the keys loaded after them, two CTAs to an SM: GLA 38 us, WKV 29 us at the sizes above; 31.7 and 19.0 now.)
template <int MODE, int VT, int TH>
__global__ void __launch_bounds__(TH, MODE == LT ? 2 : (TH == 256 ? 3 : 5)) la_chunk_sum_kernel(const Params p) {
  atom::pdl_trigger();
  atom::pdl_wait();
  extern __shared__ __align__(16) unsigned char la_smem[];
  int s, r;
  if (!find_chunk(blockIdx.x, p.cu_q, p.num_seqs, s, r)) return;
  const int h = blockIdx.y, c0 = blockIdx.z * VT, tid = threadIdx.x;
  const int t0 = p.cu_q[s] + r * L, rows = min(L, p.cu_q[s + 1] - t0);
  const int np = (p.dk + 15) & ~15, ldn = np + 8;
  constexpr int VP = MODE == LT ? 3 : 1, LDV = VT + 8;
  __nv_bfloat16* Kp = reinterpret_cast<__nv_bfloat16*>(la_smem);          // [3][L][ldn]
  __nv_bfloat16* Vs = Kp + 3 * L * ldn;                                      // [VP][L][LDV]
  float* tot = reinterpret_cast<float*>(Vs + VP * L * LDV);                  // [4][np] the blocks' sums; LT: powers [L]
  load_values<MODE, VT, TH>(Vs, p.v + (int64_t)t0 * p.ldv + (int64_t)h * p.dv + c0, p.ldv, rows, p.dv - c0);
  asm volatile("cp.async.commit_group;\n" ::);
  float* sA = p.sA + ((int64_t)blockIdx.x * p.H + h) * p.dk;
  // K^: every row's k times what the state keeps of it at the chunk's end
  const __nv_bfloat16* kg = p.k + (int64_t)t0 * p.ld + (int64_t)h * p.dk;
  if constexpr (MODE == LT) {
    const float lam = p.decay[h];
    if (tid < L) tot[tid] = power(lam, tid);
    if (blockIdx.z == 0) {
      const float all = power(lam, rows);
      for (int c = tid; c < p.dk; c += TH) sA[c] = all;
    }
    __syncthreads();
#pragma unroll 4
    for (int e = tid; e < L * (np / 8); e += TH) {
      const int i = e / (np / 8), c = (e - i * (np / 8)) * 8;
      uint4 raw = make_uint4(0u, 0u, 0u, 0u);
      if (i < rows && c < p.dk) raw = *reinterpret_cast<const uint4*>(kg + (int64_t)i * p.ld + c);
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
      uint32_t o[3][4];
      const float d = tot[max(rows - 1 - i, 0)];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float2 f = unpack(w[x]);
        uint32_t q[3];
        split3(silu(f.x) * d, silu(f.y) * d, q);
#pragma unroll
        for (int m = 0; m < 3; ++m) o[m][x] = q[m];
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
        *reinterpret_cast<uint4*>(Kp + (m * L + i) * ldn + c) = make_uint4(o[m][0], o[m][1], o[m][2], o[m][3]);
    }
  } else {
    const bool wide = p.ldz % 2 == 0 && ((uintptr_t)p.z % 8) == 0;
    const int pairs = np / 2;
    const int b = tid / pairs, c = (tid - b * pairs) * 2;      // (4 pairs <= TH)
    const bool own = b < 4 && c < p.dk;
    const int n = own ? min(16, rows - 16 * b) : 0;      // rows of the block (may be less than none)
    const float* zr = p.z + (int64_t)(t0 + 16 * b) * p.ldz + (int64_t)h * p.dk + c;
    float2 l[16];
    uint32_t kr[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      l[i] = make_float2(0.f, 0.f);
      if (i < n) {
        if (wide) {
          l[i] = *reinterpret_cast<const float2*>(zr + i * p.ldz);
        } else {
          l[i].x = zr[i * p.ldz];
          l[i].y = zr[i * p.ldz + 1];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) kr[i] = i < n ? *reinterpret_cast<const uint32_t*>(kg + (int64_t)(16 * b + i) * p.ld + c) : 0u;
    const float bx = own ? load_as_float(p.zb, p.zb_dtype, (int64_t)h * p.dk + c) : 0.f;
    const float by = own ? load_as_float(p.zb, p.zb_dtype, (int64_t)h * p.dk + c + 1) : 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      l[i] = i < n ? make_float2(log_decay<MODE>(l[i].x + bx, p.inv_tau), log_decay<MODE>(l[i].y + by, p.inv_tau)) : make_float2(0.f, 0.f);
    if (blockIdx.z == 0) {
      float* g = p.g + ((int64_t)(t0 + 16 * b) * p.H + h) * p.dk + c;
      float2 sum = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        sum.x += l[i].x;
        sum.y += l[i].y;
        if (i < n) *reinterpret_cast<float2*>(g + (int64_t)i * p.H * p.dk) = sum;
      }
    }
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 15; i >= 0; --i) {                       // l: the sums behind a row in its block
      const float2 x = l[i];
      l[i] = sum;
      sum.x += x.x;
      sum.y += x.y;
    }
    if (b < 4) *reinterpret_cast<float2*>(tot + b * np + c) = sum;
    __syncthreads();
    if (b < 4) {
      float2 t[4];
#pragma unroll
      for (int x = 1; x < 4; ++x) t[x] = *reinterpret_cast<const float2*>(tot + x * np + c);
      if (b == 0 && blockIdx.z == 0 && own)
        *reinterpret_cast<float2*>(sA + c) = make_float2(ex2(sum.x + (t[1].x + (t[2].x + t[3].x))), ex2(sum.y + (t[1].y + (t[2].y + t[3].y))));
      float2 behind = make_float2(0.f, 0.f);              // the sum of the blocks behind this one
#pragma unroll
      for (int x = 3; x >= 1; --x)
        if (x > b) {
          behind.x += t[x].x;
          behind.y += t[x].y;
        }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 f = unpack(kr[i]);
        uint32_t q[3];
        split3(f.x * ex2(l[i].x + behind.x), f.y * ex2(l[i].y + behind.y), q);
#pragma unroll
        for (int m = 0; m < 3; ++m) *reinterpret_cast<uint32_t*>(Kp + (m * L + 16 * b + i) * ldn + c) = q[m];
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  float* dst = p.sB + (((int64_t)blockIdx.x * p.H + h) * p.dk) * p.dv;
  const int steps = (rows + 15) / 16;
  constexpr int NT = 8;                       // 8-column tiles of a warp
  for (int item = warp; item < (np / 16) * (VT / 64); item += TH / 32) {
    const int mt = item / (VT / 64), n0 = (item % (VT / 64)) * 64;
    float acc[NT][4], rest[MODE == LT ? NT : 1][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    if constexpr (MODE == LT) {
#pragma unroll
      for (int i = 0; i < NT; ++i) rest[i][0] = rest[i][1] = rest[i][2] = rest[i][3] = 0.f;
    }
#pragma unroll 1
    for (int kk = 0; kk < steps; ++kk) {
      uint32_t a[3][4];      // rows of the product are key channels, its inner dimension the chunk's rows
#pragma unroll
      for (int m = 0; m < 3; ++m)
        ldm_x4_trans(a[m], Kp + (m * L + kk * 16 + (lane >> 4) * 8 + (lane & 7)) * ldn + mt * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int n = 0; n < NT; n += 4) {
        uint32_t b[4][VP][2];
#pragma unroll
        for (int m = 0; m < VP; ++m)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            uint32_t t[4];
            ldm_x4_trans(t, Vs + (m * L + kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * LDV + n0 + n * 8 + x * 16 + (lane >> 4) * 8);
            b[2 * x][m][0] = t[0];
            b[2 * x][m][1] = t[1];
            b[2 * x + 1][m][0] = t[2];
            b[2 * x + 1][m][1] = t[3];
          }
        if constexpr (MODE == LT) {
          mma_six<4>({&acc[n], &acc[n + 1], &acc[n + 2], &acc[n + 3]}, {&rest[n], &rest[n + 1], &rest[n + 2], &rest[n + 3]}, {a, a, a, a},
                     {b[0], b[1], b[2], b[3]});
        } else {
          const uint32_t c[4][2] = {{b[0][0][0], b[0][0][1]}, {b[1][0][0], b[1][0][1]}, {b[2][0][0], b[2][0][1]}, {b[3][0][0], b[3][0][1]}};
          mma_three<4>({&acc[n], &acc[n + 1], &acc[n + 2], &acc[n + 3]}, {a, a, a, a}, c);
        }
      }
    }
    if constexpr (MODE == LT) {
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] += rest[i][e];
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int c = c0 + n0 + i * 8 + (lane & 3) * 2;
      if (c >= p.dv) continue;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int n = mt * 16 + (lane >> 2) + 8 * m;
        if (n < p.dk) *reinterpret_cast<float2*>(dst + (int64_t)n * p.dv + c) = make_float2(acc[i][2 * m], acc[i][2 * m + 1]);
      }
    }
  }
}

// ------------------------------------------------------------------ the states at the chunks' borders

__global__ void __launch_bounds__(256) la_prefix_kernel(const Params p) {
  atom::pdl_trigger();
  atom::pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y;
  const int len = p.cu_q[s + 1] - p.cu_q[s];
  const int64_t mat = (int64_t)p.dk * p.dv;
  const int64_t e = ((int64_t)blockIdx.z * blockDim.x + threadIdx.x) * 4;
  if (len <= 0 || e >= mat) return;
  int x0 = 0;
  for (int q = 0; q < s; ++q) x0 += (p.cu_q[q + 1] - p.cu_q[q] + L - 1) / L;
  const int n = (len + L - 1) / L, ch = (int)(e / p.dv);
  float4* st = reinterpret_cast<float4*>(p.state + ((int64_t)p.state_slots[s] * p.H + h) * mat + e);
  float* B = p.sB + ((int64_t)x0 * p.H + h) * mat + e;
  const float* A = p.sA + ((int64_t)x0 * p.H + h) * p.dk + ch;
  const int64_t next = (int64_t)p.H * mat, next_a = (int64_t)p.H * p.dk;
  float4 S = *st;
  constexpr int kAhead = 8;              // the chunks' sums do not depend on S: eight loads are under way together
  for (int r0 = 0; r0 < n; r0 += kAhead) {
    float4 b[kAhead];
    float a[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      if (r0 + j < n) {
        b[j] = *reinterpret_cast<const float4*>(B + (r0 + j) * next);
        a[j] = A[(r0 + j) * next_a];
      }
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      if (r0 + j < n) {
        *reinterpret_cast<float4*>(B + (r0 + j) * next) = S;
        S.x = fmaf(a[j], S.x, b[j].x);
        S.y = fmaf(a[j], S.y, b[j].y);
        S.z = fmaf(a[j], S.z, b[j].z);
        S.w = fmaf(a[j], S.w, b[j].w);
      }
  }
  if (p.write_state) *st = S;
}

// ------------------------------------------------------------------ the outputs

// A CTA of 8 warps: a chunk, a head, VT value columns.  First the pairs' sums, shared out in tiles of 16 rows x 8 columns (block
// 3 of the rows has 8 of them, 2 has 6, 1 has 4, 0 has 2: two or three a warp), left in shared memory as the planes of the last
// product; then a warp owns VT / 8 of the value columns for all rows, so that the state's numbers are split by one warp alone, on
// their way from memory, and the decayed queries once, into planes that take the place of keys and logarithms.  (A warp per 16
// rows with the state's planes in shared memory, every warp forming its queries: 88 us for GLA at 2,048 rows and 16 heads of 128
// x 128, one CTA to an SM; 60 us now.)  NQ: 32 key
// channels each; with two and 64 value columns three CTAs fit an SM's registers (WKV: 77 us, 88 us with two CTAs).
// The chunk's outputs row by row from the state it begins with, as the formulas at the top say: a thread holds one value column's
// share of the state in registers.  About 30 us for a chunk of 128 x 128.
template <int MODE, int VT, int NQ>
__device__ __noinline__ void walk_chunk(const Params& p, int h, int c0, int t0, int rows, float* smem) {
  constexpr int G = THREADS / VT, LDC = 32 * NQ, NC = LDC / G;      // channels of a thread: NC from part * NC on
  float *qs = smem, *ks = qs + LDC, *as = ks + LDC, *bs = as + LDC, *red = bs + LDC, *sq = red + THREADS;
  const int tid = threadIdx.x, col = tid % VT, part = tid / VT, c = c0 + col;
  const bool in = c < p.dv;
  const float* B = p.sB + (((int64_t)blockIdx.x * p.H + h) * p.dk) * p.dv + c;
  float S[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) S[i] = in && part * NC + i < p.dk ? B[(int64_t)(part * NC + i) * p.dv] : 0.f;
  for (int row = 0; row < rows; ++row) {
    const int64_t t = t0 + row;
    if (tid < LDC) {
      const int64_t at = (int64_t)h * p.dk + tid;
      float q = 0.f, k = 0.f, a = 1.f, b = 0.f;
      if (tid < p.dk) {
        q = to_float(p.q[t * p.ld + at]);
        k = to_float(p.k[t * p.ld + at]);
        if (MODE == LT) {
          q = silu(q);
          k = silu(k);
          a = p.decay[h];
        } else {
          const float z = p.z[t * p.ldz + at] + load_as_float(p.zb, p.zb_dtype, at);
          a = MODE == GLA ? expf((fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) * p.inv_tau) : expf(-expf(z));
          if (MODE == GLA) q *= p.q_scale;
          else b = q * load_as_float(p.u, p.zb_dtype, at) * k;
        }
      }
      qs[tid] = q;
      ks[tid] = k;
      as[tid] = a;
      bs[tid] = b;
    }
    float v = in ? to_float(p.v[t * p.ldv + (int64_t)h * p.dv + c]) : 0.f;
    if (MODE == LT) v = silu(v);
    __syncthreads();
    float o = 0.f;
#pragma unroll
    for (int i = 0; i < NC; i += 4) {
      const float4 q = *reinterpret_cast<const float4*>(qs + part * NC + i), k = *reinterpret_cast<const float4*>(ks + part * NC + i);
      const float4 a = *reinterpret_cast<const float4*>(as + part * NC + i);
      const float qe[4] = {q.x, q.y, q.z, q.w}, ke[4] = {k.x, k.y, k.z, k.w}, ae[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (MODE == WKV) o = fmaf(qe[e], S[i + e], o);
        S[i + e] = fmaf(ae[e], S[i + e], ke[e] * v);
        if (MODE != WKV) o = fmaf(qe[e], S[i + e], o);
      }
    }
    red[tid] = o;
    __syncthreads();
    if (part == 0) {
#pragma unroll
      for (int g = 1; g < G; ++g) o += red[g * VT + col];
      if (MODE == WKV) {
        float b = 0.f;
        for (int i = 0; i < p.dk; ++i) b += bs[i];
        o = fmaf(b, v, o);
        sq[col] = in ? o * o : 0.f;
      } else if (in) {
        p.out[(t * p.H + h) * p.dv + c] = o;
      }
    }
    if (MODE == WKV) {
      __syncthreads();
      if (part == 0 && in) {
        float ss = 0.f;
        for (int i = 0; i < p.dv; ++i) ss += sq[i];
        const int64_t at = t * p.ldv + (int64_t)h * p.dv + c;
        p.y[at] = __float2bfloat16_rn(o * rsqrtf(ss / (float)p.dv + p.eps) * load_as_float(p.norm_w, p.zb_dtype, (int64_t)h * p.dv + c) *
                                      silu(to_float(p.gate[at])));
      }
    }
    __syncthreads();
  }
}

template <int MODE, int VT, int NQ>
__global__ void __launch_bounds__(THREADS, NQ == 2 && VT == 64 ? 3 : 2) la_chunk_out_kernel(const __grid_constant__ Params p) {
  atom::pdl_trigger();
  atom::pdl_wait();
  extern __shared__ __align__(16) unsigned char la_smem[];
  int s, r;
  if (!find_chunk(blockIdx.x, p.cu_q, p.num_seqs, s, r)) return;
  const int h = blockIdx.y, c0 = blockIdx.z * VT, tid = threadIdx.x;
  const int t0 = p.cu_q[s] + r * L, rows = min(L, p.cu_q[s + 1] - t0);
  const int np = (p.dk + 15) & ~15, ldk = np + 8, lds = np + 4;
  constexpr int LDV = VT + 8;
  // values [L][LDV]; GLA, WKV: sums over whole blocks [6][np], LT: powers [L + 1]; then GLA, WKV: planes of the pairs' sums
  // [3][L][LP] | logarithms' sums [L][lds], keys [L][ldk], later in their place the queries' planes [3][L][ldk];
  // LT: the queries' planes | silu of the keys [L][lds], later in its place the planes of the pairs' sums
  __nv_bfloat16* Vs = reinterpret_cast<__nv_bfloat16*>(la_smem);
  float* off = reinterpret_cast<float*>(Vs + L * LDV);
  __nv_bfloat16* first = reinterpret_cast<__nv_bfloat16*>(off + (MODE == LT ? L + 4 : 6 * np));
  __nv_bfloat16* second = first + 3 * L * (MODE == LT ? ldk : LP);
  __nv_bfloat16 *P = MODE == LT ? second : first, *Q = MODE == LT ? first : second;
  float* gs = reinterpret_cast<float*>(second);
  __nv_bfloat16* Ks = second + 2 * L * lds;
  {
    const __nv_bfloat16* vg = p.v + (int64_t)t0 * p.ldv + (int64_t)h * p.dv + c0;
    for (int e = tid; e < L * (VT / 8); e += THREADS) {
      const int i = e / (VT / 8), c = (e % (VT / 8)) * 8;
      const bool in = i < rows && c0 + c < p.dv;
      cp_async16(Vs + i * LDV + c, vg + (in ? (int64_t)i * p.ldv + c : 0), in);
    }
  }
  const __nv_bfloat16* kg = p.k + (int64_t)t0 * p.ld + (int64_t)h * p.dk;
  const __nv_bfloat16* qg = p.q + (int64_t)t0 * p.ld + (int64_t)h * p.dk;
  if (MODE == LT) {
    for (int e = tid; e < L * (np / 8); e += THREADS) {
      const int i = e / (np / 8), c = (e - i * (np / 8)) * 8;
      uint4 kr = make_uint4(0u, 0u, 0u, 0u), qr = kr;
      if (i < rows && c < p.dk) {
        kr = *reinterpret_cast<const uint4*>(kg + (int64_t)i * p.ld + c);
        qr = *reinterpret_cast<const uint4*>(qg + (int64_t)i * p.ld + c);
      }
      const float2 a = unpack(kr.x), b = unpack(kr.y), d = unpack(kr.z), f = unpack(kr.w);
      *reinterpret_cast<float4*>(gs + i * lds + c) = make_float4(silu(a.x), silu(a.y), silu(b.x), silu(b.y));
      *reinterpret_cast<float4*>(gs + i * lds + c + 4) = make_float4(silu(d.x), silu(d.y), silu(f.x), silu(f.y));
      const uint32_t w[4] = {qr.x, qr.y, qr.z, qr.w};
      uint32_t o[4][3];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float2 t = unpack(w[x]);
        split3(silu(t.x), silu(t.y), o[x]);
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
        *reinterpret_cast<uint4*>(Q + (m * L + i) * ldk + c) = make_uint4(o[0][m], o[1][m], o[2][m], o[3][m]);
    }
    if (tid <= L) off[tid] = power(p.decay[h], tid);
  } else {
    const float* gg = p.g + ((int64_t)t0 * p.H + h) * p.dk;
    for (int e = tid; e < L * (np / 4); e += THREADS) {
      const int i = e / (np / 4), c = (e - i * (np / 4)) * 4;
      const bool in = i < rows && c < p.dk;
      cp_async16(gs + i * lds + c, gg + (in ? (int64_t)i * p.H * p.dk + c : 0), in);
    }
    for (int e = tid; e < L * (np / 8); e += THREADS) {
      const int i = e / (np / 8), c = (e - i * (np / 8)) * 8;
      const bool in = i < rows && c < p.dk;
      cp_async16(Ks + i * ldk + c, kg + (in ? (int64_t)i * p.ld + c : 0), in);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::);
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  bool walk = false;
  if (MODE != LT) {
    // row I (I - 1) / 2 + J, J < I: the sum over the blocks J .. I - 1 (whole ones, if block I has rows)
    for (int c = tid; c < np; c += THREADS) {
      const float a = gs[15 * lds + c], b = gs[31 * lds + c], d = gs[47 * lds + c], e = gs[(rows - 1) * lds + c];
      walk |= !(a >= kWalk && b >= kWalk && d >= kWalk && e >= kWalk);
      off[c] = a;
      off[np + c] = a + b;
      off[2 * np + c] = b;
      off[3 * np + c] = a + (b + d);
      off[4 * np + c] = b + d;
      off[5 * np + c] = d;
    }
    __syncthreads();
  }
  const int warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  auto set_a = [&](uint32_t (&a)[3][4], int e, float x, float y) {
    uint32_t t[3];
    split3(x, y, t);
    a[0][e] = t[0];
    a[1][e] = t[1];
    a[2][e] = t[2];
  };
  auto set_b = [&](uint32_t (&b)[3][2], int y, float2 v) {
    uint32_t t[3];
    split3(v.x, v.y, t);
    b[0][y] = t[0];
    b[1][y] = t[1];
    b[2][y] = t[2];
  };
  auto planes = [&](uint32_t (&a)[3][4], const __nv_bfloat16* X, int ldx, int row0, int col0) {
#pragma unroll
    for (int m = 0; m < 3; ++m)
      ldm_x4(a[m], X + (m * L + row0 + ((lane >> 3) & 1) * 8 + (lane & 7)) * ldx + col0 + (lane >> 4) * 8);
  };

  // ---- the pairs' sums: tiles jt0 .. of row block I
  const int I = warp < 3 ? 3 : (warp < 5 ? 2 : (warp < 7 ? 1 : 0));
  const int jt0 = warp < 3 ? 3 * warp : (warp < 5 ? 3 * (warp - 3) : (warp < 7 ? 2 * (warp - 5) : 0));
  const int tiles = warp == 2 || warp >= 5 ? 2 : 3;
  const int ia = 16 * I + gq, ib = ia + 8;
  float sc[3][4];
#pragma unroll
  for (int x = 0; x < 3; ++x) sc[x][0] = sc[x][1] = sc[x][2] = sc[x][3] = 0.f;
  if (16 * I < rows) {
    const bool ends = jt0 + tiles == 2 * I + 2;             // the warp has the two tiles of the row block's own columns
    float bonus_a = 0.f, bonus_b = 0.f;
    if constexpr (MODE == LT) {
      float rest[3][4];
#pragma unroll
      for (int x = 0; x < 3; ++x) rest[x][0] = rest[x][1] = rest[x][2] = rest[x][3] = 0.f;
#pragma unroll 1
      for (int kk = 0; kk < np; kk += 16) {
        uint32_t a[3][4], b[3][3][2];
        planes(a, Q, ldk, 16 * I, kk);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          const float* kr = gs + (8 * min(jt0 + x, 2 * I + 1) + gq) * lds + kk + 2 * tq;
#pragma unroll
          for (int y = 0; y < 2; ++y) set_b(b[x], y, *reinterpret_cast<const float2*>(kr + 8 * y));
        }
        mma_six<3>({&sc[0], &sc[1], &sc[2]}, {&rest[0], &rest[1], &rest[2]}, {a, a, a}, {b[0], b[1], b[2]});
      }
#pragma unroll
      for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[x][e] += rest[x][e];
    } else {
      auto load_q = [&](uint32_t (&x)[4], int c) {          // (rows gq and gq + 8 of the block, channels c + 2 tq .. and 8 further)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = ia + (e & 1) * 8, cc = c + 2 * tq + (e >> 1) * 8;
          x[e] = row < rows && cc < p.dk ? *reinterpret_cast<const uint32_t*>(qg + (int64_t)row * p.ld + cc) : 0u;
        }
      };
      const float* mid = gs + min(16 * I + 7, rows - 1) * lds;      // the own block's reference: its eighth row
      uint32_t qn[4];
      load_q(qn, 0);
#pragma unroll 1
      for (int kk = 0; kk < np; kk += 16) {
        float2 qf[4], gi[4];
        const int c = kk + 2 * tq;                          // this lane's channels: c, c + 1, c + 8, c + 9
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          qf[e] = unpack(qn[e]);
          if (MODE == GLA) {
            qf[e].x *= p.q_scale;
            qf[e].y *= p.q_scale;
          }
          // the logarithms' sum up to the query's own row (WKV: up to the row before), from its block on
          const int row = ia + (e & 1) * 8 - (MODE == WKV ? 1 : 0);
          gi[e] = row >= 16 * I ? *reinterpret_cast<const float2*>(gs + row * lds + c + (e >> 1) * 8) : make_float2(0.f, 0.f);
        }
        if (kk + 16 < np) load_q(qn, kk + 16);
        if (MODE == WKV && ends) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 kf = unpack(*reinterpret_cast<const uint32_t*>(Ks + ((e & 1) ? ib : ia) * ldk + c + (e >> 1) * 8));
            const int cc = c + (e >> 1) * 8;
            float v = 0.f;
            if (cc < p.dk)
              v = qf[e].x * load_as_float(p.u, p.zb_dtype, (int64_t)h * p.dk + cc) * kf.x +
                  qf[e].y * load_as_float(p.u, p.zb_dtype, (int64_t)h * p.dk + cc + 1) * kf.y;
            if (e & 1) bonus_b += v;
            else bonus_a += v;
          }
        }
        float2 rv[2];
        uint32_t b[3][3][2];
        auto keys = [&](int x) {                            // the column tile's keys, decayed up to the reference
          const int j = 8 * (jt0 + x) + gq;
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            const float2 g = sub2(rv[y], *reinterpret_cast<const float2*>(gs + j * lds + c + 8 * y));
            float2 k2 = unpack(*reinterpret_cast<const uint32_t*>(Ks + j * ldk + c + 8 * y));
            k2.x *= ex2(g.x);
            k2.y *= ex2(g.y);
            set_b(b[x], y, k2);
          }
        };
        auto earlier = [&](int x) {                         // (columns of an earlier block: their sums up to block I)
          const float* ref = off + (I * (I - 1) / 2 + ((jt0 + x) >> 1)) * np + c;
          rv[0] = *reinterpret_cast<const float2*>(ref);
          rv[1] = *reinterpret_cast<const float2*>(ref + 8);
          keys(x);
        };
        uint32_t a[3][4];
        if (!ends || tiles == 3) {
#pragma unroll
          for (int e = 0; e < 4; ++e) set_a(a, e, qf[e].x * ex2(gi[e].x), qf[e].y * ex2(gi[e].y));
          earlier(0);
          if (ends) {
            mma_six<1>({&sc[0]}, {a}, {b[0]});
          } else {
            earlier(1);
            if (tiles == 3) {
              earlier(2);
              mma_six<3>({&sc[0], &sc[1], &sc[2]}, {a, a, a}, {b[0], b[1], b[2]});
            } else {
              mma_six<2>({&sc[0], &sc[1]}, {a, a}, {b[0], b[1]});
            }
          }
        }
        if (ends) {
          rv[0] = *reinterpret_cast<const float2*>(mid + c);
          rv[1] = *reinterpret_cast<const float2*>(mid + c + 8);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 g = sub2(gi[e], rv[e >> 1]);
            set_a(a, e, qf[e].x * ex2(g.x), qf[e].y * ex2(g.y));
          }
          if (tiles == 3) {
            keys(1);
            keys(2);
            mma_six<2>({&sc[1], &sc[2]}, {a, a}, {b[1], b[2]});
          } else {
            keys(0);
            keys(1);
            mma_six<2>({&sc[0], &sc[1]}, {a, a}, {b[0], b[1]});
          }
        }
      }
      if (ends) {
        if (MODE == WKV) {
          bonus_a += __shfl_xor_sync(0xffffffffu, bonus_a, 1);
          bonus_a += __shfl_xor_sync(0xffffffffu, bonus_a, 2);
          bonus_b += __shfl_xor_sync(0xffffffffu, bonus_b, 1);
          bonus_b += __shfl_xor_sync(0xffffffffu, bonus_b, 2);
        }
        // half blocks whose decays reach beyond the factors' range: pair by pair (a lane's own two pairs of each)
        bool strong[2] = {false, false};
        for (int c = lane; c < np; c += 32) {
          const float g7 = mid[c], g15 = gs[min(16 * I + 15, rows - 1) * lds + c];
          strong[0] |= g7 < kStrong;
          strong[1] |= g15 - g7 < kStrong;
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          if (!__any_sync(0xffffffffu, strong[n])) continue;
          const int i = n ? ib : ia, from = i - (MODE == WKV ? 1 : 0);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = 16 * I + 8 * n + 2 * tq + e;
            float sum = 0.f;
            if (j <= from && i < rows) {
              for (int c = 0; c < p.dk; ++c) {
                const float w = __bfloat162float(Ks[j * ldk + c]) * ex2(gs[from * lds + c] - gs[j * lds + c]);
                sum = fmaf(__bfloat162float(qg[(int64_t)i * p.ld + c]) * (MODE == GLA ? p.q_scale : 1.f), w, sum);
              }
            }
            if (tiles == 2) sc[n][2 * n + e] = sum;
            else sc[n + 1][2 * n + e] = sum;
          }
        }
      }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = (e < 2 ? ia : ib) - (8 * (jt0 + x) + 2 * tq + (e & 1));
        if (MODE == LT)
          sc[x][e] = d >= 0 ? sc[x][e] * off[max(d, 0)] : 0.f;
        else if (MODE == GLA)
          sc[x][e] = d >= 0 ? sc[x][e] : 0.f;
        else
          sc[x][e] = d > 0 ? sc[x][e] : (d == 0 ? (e < 2 ? bonus_a : bonus_b) : 0.f);
      }
    }
  }
  auto write_pairs = [&]() {
    if (16 * I >= rows) return;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      if (x >= tiles) continue;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t t[3];
        split3(sc[x][2 * half], sc[x][2 * half + 1], t);
#pragma unroll
        for (int m = 0; m < 3; ++m)
          *reinterpret_cast<uint32_t*>(P + (m * L + ia + 8 * half) * LP + 8 * (jt0 + x) + 2 * tq) = t[m];
      }
    }
  };
  if constexpr (MODE == LT) {
    __syncthreads();                                        // (the keys are not needed any more)
    write_pairs();
  } else {
    write_pairs();
    // the queries, decayed from the chunk's first row on
    uint32_t q3[NQ][4][3];
#pragma unroll
    for (int x = 0; x < NQ; ++x) {
      const int e = tid + x * THREADS, i = e / (np / 8), c = (e - i * (np / 8)) * 8;
      if (e < L * (np / 8)) {
        uint4 raw = make_uint4(0u, 0u, 0u, 0u);
        if (i < rows && c < p.dk) raw = *reinterpret_cast<const uint4*>(qg + (int64_t)i * p.ld + c);
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
        const int blk = i >> 4, from = i - (MODE == WKV ? 1 : 0);
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          float2 f = unpack(w[y]), g = make_float2(0.f, 0.f);
          if (MODE == GLA) {
            f.x *= p.q_scale;
            f.y *= p.q_scale;
          }
          if (from >= 16 * blk) g = *reinterpret_cast<const float2*>(gs + from * lds + c + 2 * y);
          if (blk > 0) {
            const float2 o2 = *reinterpret_cast<const float2*>(off + (blk * (blk - 1) / 2) * np + c + 2 * y);
            g.x += o2.x;
            g.y += o2.y;
          }
          split3(f.x * ex2(g.x), f.y * ex2(g.y), q3[x][y]);
        }
      }
    }
    __syncthreads();                                        // (keys and logarithms are not needed any more)
#pragma unroll
    for (int x = 0; x < NQ; ++x) {
      const int e = tid + x * THREADS, i = e / (np / 8), c = (e - i * (np / 8)) * 8;
      if (e < L * (np / 8)) {
#pragma unroll
        for (int m = 0; m < 3; ++m)
          *reinterpret_cast<uint4*>(Q + (m * L + i) * ldk + c) = make_uint4(q3[x][0][m], q3[x][1][m], q3[x][2][m], q3[x][3][m]);
      }
    }
  }

  // ---- the state's part: VT / 8 columns of all rows, NT tiles of eight at a time (LT: one, its sums in two numbers)
  constexpr int TILES = VT / 64, NT = MODE == LT ? 1 : TILES;
#pragma unroll 1
  for (int n0 = warp * 8 * TILES; n0 < (warp + 1) * 8 * TILES; n0 += 8 * NT) {
  const float* S = p.sB + (((int64_t)blockIdx.x * p.H + h) * p.dk) * p.dv + c0 + n0 + gq;
  float sv[NT][4];
  auto load_state = [&](int kk) {
#pragma unroll
    for (int x = 0; x < NT; ++x)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = kk + 2 * tq + (e & 1) + (e >> 1) * 8;
        sv[x][e] = c < p.dk && c0 + n0 + 8 * x + gq < p.dv ? S[(int64_t)c * p.dv + 8 * x] : 0.f;
      }
  };
  load_state(0);
  __syncthreads();                                          // the planes stand
  float o[4][NT][4], rest[MODE == LT ? 4 : 1][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int x = 0; x < NT; ++x) o[i][x][0] = o[i][x][1] = o[i][x][2] = o[i][x][3] = 0.f;
  if constexpr (MODE == LT) {
#pragma unroll
    for (int i = 0; i < 4; ++i) rest[i][0] = rest[i][1] = rest[i][2] = rest[i][3] = 0.f;
  }
#pragma unroll 1
  for (int kk = 0; kk < np; kk += 16) {
    uint32_t b[NT][3][2];
#pragma unroll
    for (int x = 0; x < NT; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y) set_b(b[x], y, make_float2(sv[x][2 * y], sv[x][2 * y + 1]));
    if (kk + 16 < np) load_state(kk + 16);
#pragma unroll
    for (int mt = 0; mt < 4; mt += 2) {
      if (16 * mt >= rows) break;
      uint32_t a0[3][4], a1[3][4];
      planes(a0, Q, ldk, 16 * mt, kk);
      planes(a1, Q, ldk, 16 * mt + 16, kk);
      if constexpr (MODE == LT)
        mma_six<2>({&o[mt][0], &o[mt + 1][0]}, {&rest[mt], &rest[mt + 1]}, {a0, a1}, {b[0], b[0]});
      else if constexpr (NT == 2)
        mma_six<4>({&o[mt][0], &o[mt][1], &o[mt + 1][0], &o[mt + 1][1]}, {a0, a0, a1, a1}, {b[0], b[1], b[0], b[1]});
      else
        mma_six<2>({&o[mt][0], &o[mt + 1][0]}, {a0, a1}, {b[0], b[0]});
    }
  }
  if constexpr (MODE == LT) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float pa = off[16 * i + gq + 1], pb = off[16 * i + gq + 9];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[i][0][e] = (o[i][0][e] + rest[i][e]) * (e < 2 ? pa : pb);
        rest[i][e] = 0.f;
      }
    }
  }
  // WKV: the norm's weights and the gate, on their way during the last product (a warp has one tile of columns)
  uint32_t gate[MODE == WKV ? 8 : 1];
  float w0 = 0.f, w1 = 0.f;
  if constexpr (MODE == WKV) {
    const int c = n0 + 2 * tq;
    if (c < p.dv) {
      w0 = load_as_float(p.norm_w, p.zb_dtype, (int64_t)h * p.dv + c);
      w1 = load_as_float(p.norm_w, p.zb_dtype, (int64_t)h * p.dv + c + 1);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 8 * i + gq;
      gate[i] = row < rows && c < p.dv ? *reinterpret_cast<const uint32_t*>(p.gate + (int64_t)(t0 + row) * p.ldv + (int64_t)h * p.dv + c) : 0u;
    }
  }
  // ---- the pairs' sums times the values
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    if (16 * ks >= rows) break;
    uint32_t v[NT][2];
    {
      uint32_t t[4];      // (one tile of columns: the rows of the next step come along)
      if constexpr (NT == 2) {
        ldm_x4_trans(t, Vs + (ks * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * LDV + n0 + (lane >> 4) * 8);
        v[1][0] = t[2];
        v[1][1] = t[3];
      } else {
        ldm_x4_trans(t, Vs + (min(ks * 16 + (lane >> 4) * 16, L - 16) + ((lane >> 3) & 1) * 8 + (lane & 7)) * LDV + n0);
      }
      v[0][0] = t[0];
      v[0][1] = t[1];
    }
    uint32_t b[NT][3][2];
    if constexpr (MODE == LT) {
#pragma unroll
      for (int x = 0; x < NT; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const float2 f = unpack(v[x][y]);
          set_b(b[x], y, make_float2(silu(f.x), silu(f.y)));
        }
    }
#pragma unroll
    for (int mt = ks; mt < 4; ++mt) {
      uint32_t w[3][4];
      if (16 * mt >= rows) break;
      planes(w, P, LP, 16 * mt, 16 * ks);
      if constexpr (MODE == LT)
        mma_six<1>({&o[mt][0]}, {&rest[mt]}, {w}, {b[0]});
      else if constexpr (NT == 2)
        mma_three<2>({&o[mt][0], &o[mt][1]}, {w, w}, v);
      else
        mma_three<1>({&o[mt][0]}, {w}, v);
    }
  }
  if constexpr (MODE == LT) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[i][0][e] += rest[i][e];
  }
  float odd = 0.f;                                          // not zero: what zero times a number that is not finite leaves
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int x = 0; x < NT; ++x)
#pragma unroll
      for (int e = 0; e < 4; ++e) odd = fmaf(o[i][x][e], 0.f, odd);
  if (__syncthreads_or(walk || odd != 0.f)) {
    walk_chunk<MODE, VT, NQ>(p, h, c0, t0, rows, reinterpret_cast<float*>(la_smem));
    return;
  }
  if constexpr (MODE == WKV) {
    // o over its root mean square: a row lies with all warps (columns beyond dv are zero; one tile holds the head)
    float* part = reinterpret_cast<float*>(Q);              // [8][L], in the place of the queries
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float sa = 0.f, sb = 0.f;
#pragma unroll
      for (int x = 0; x < NT; ++x) {
        sa = fmaf(o[i][x][0], o[i][x][0], fmaf(o[i][x][1], o[i][x][1], sa));
        sb = fmaf(o[i][x][2], o[i][x][2], fmaf(o[i][x][3], o[i][x][3], sb));
      }
      sa += __shfl_xor_sync(0xffffffffu, sa, 1);
      sa += __shfl_xor_sync(0xffffffffu, sa, 2);
      sb += __shfl_xor_sync(0xffffffffu, sb, 1);
      sb += __shfl_xor_sync(0xffffffffu, sb, 2);
      if (tq == 0) {
        part[warp * L + 16 * i + gq] = sa;
        part[warp * L + 16 * i + gq + 8] = sb;
      }
    }
    __syncthreads();
    const int c = n0 + 2 * tq;
    const bool in = c < p.dv;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int row = 16 * i + gq + 8 * m;
        if (row >= rows || !in) continue;
        float ss = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) ss += part[w * L + row];
        const float f = rsqrtf(ss / (float)p.dv + p.eps);
        const int64_t at = (int64_t)(t0 + row) * p.ldv + (int64_t)h * p.dv + c;
        const float2 gt = unpack(gate[2 * i + m]);
        *reinterpret_cast<uint32_t*>(p.y + at) = pack(o[i][0][2 * m] * f * w0 * silu(gt.x), o[i][0][2 * m + 1] * f * w1 * silu(gt.y));
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int x = 0; x < NT; ++x) {
        const int c = c0 + n0 + 8 * x + 2 * tq;
        if (c >= p.dv) continue;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const int row = 16 * i + gq + 8 * m;
          if (row < rows)
            *reinterpret_cast<float2*>(p.out + ((int64_t)(t0 + row) * p.H + h) * p.dv + c) = make_float2(o[i][x][2 * m], o[i][x][2 * m + 1]);
        }
      }
    }
  }
  }
}

static size_t sum_smem(int mode, int np, int vt) {
  const size_t vp = mode == LT ? 3 : 1;
  return 2 * (3 * (size_t)L * (np + 8) + vp * L * (vt + 8)) + 4 * (mode == LT ? (size_t)L : 4 * (size_t)np);
}
static size_t out_smem(int mode, int np, int vt) {
  const size_t planes = 2 * 3 * (size_t)L * (np + 8), pairs = 2 * 3 * (size_t)L * LP, rows = 4 * (size_t)L * (np + 4);
  const size_t values = 2 * (size_t)L * (vt + 8);
  if (mode == LT) return values + 4 * (L + 4) + planes + (rows > pairs ? rows : pairs);
  const size_t keys = rows + 2 * (size_t)L * (np + 8);
  return values + 4 * 6 * (size_t)np + pairs + (keys > planes ? keys : planes);
}

template <int MODE, int VT, int NQ>
static int launch(const Params& p, int T, cudaStream_t stream) {
  constexpr int TH = MODE != LT && NQ == 2 && VT == 64 ? 128 : THREADS;
  const int np = (p.dk + 15) & ~15;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(la_chunk_sum_kernel<MODE, VT, TH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sum_smem(MODE, 128, VT)) != cudaSuccess ||
        cudaFuncSetAttribute(la_chunk_out_kernel<MODE, VT, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)out_smem(MODE, 32 * NQ, VT)) != cudaSuccess)
      return ATOM_ERR_LAUNCH;
    attr_set = true;
  }
  const dim3 grid((T + L - 1) / L + p.num_seqs, p.H, (p.dv + VT - 1) / VT);
  atom::launch_pdl(la_chunk_sum_kernel<MODE, VT, TH>, grid, dim3(TH), sum_smem(MODE, np, VT), stream, p);
  const int64_t mat = (int64_t)p.dk * p.dv;
  atom::launch_pdl(la_prefix_kernel, dim3(p.num_seqs, p.H, (unsigned)((mat / 4 + 255) / 256)), dim3(256), 0, stream, p);
  atom::launch_pdl(la_chunk_out_kernel<MODE, VT, NQ>, grid, dim3(THREADS), out_smem(MODE, np, VT), stream, p);
  return atom::check_launch();
}
static int sm_count() {
  static const int n = [] {      // (asked once)
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 148;
    return sms;
  }();
  return n;
}

// Values of up to 64 columns a head in one tile of 64, wider ones in tiles of 128; up to 64 key channels or up to 128.
// Wider ones in tiles of 64 too where tiles of 128 are no more than the SMs: a CTA's time is then a chain of loads and
// products with nothing beside it, and half the columns are half of the state's and the values' part of it, while what both
// tiles of a chunk do (decays, pairs' sums) goes to SMs that had nothing to do.  The layer at width 2,048 (16 heads of 128 x
// 128), two requests, in tiles of 128 and of 64: LT 96 rows 81 and 64 us, 256 rows 87 and 74, 512 rows (144 CTAs of 148) 100
// and 78, 600 rows (176) 104 and 106, 1,024 rows 118 and 136; GLA 69 and 62, 75 and 71, 90 and 85, 96 and 105, 110 and 133.  But
// not GLA with up to 64 key channels, whose decays weigh more than half of its values: the three launches, 16 heads of 64 x 128, 200
// rows 31.9 and 34.6, 512 rows 35.6 and 39.1; 2 heads, 2,000 rows 27 and 39 (LT 45 and 38, 46 and 39, 35 and 39).  A column's numbers
// are formed alike in both.
template <int MODE>
static int launch(const Params& p, int T, cudaStream_t stream) {
  const int64_t chunks = ((int64_t)T + (int64_t)(L - 1) * p.num_seqs) / L;      // at most: every request's last one is cut short
  if (p.dv <= 64 || (!(MODE == GLA && p.dk <= 64) && chunks * p.H * ((p.dv + 127) / 128) <= sm_count()))
    return p.dk <= 64 ? launch<MODE, 64, 2>(p, T, stream) : launch<MODE, 64, 4>(p, T, stream);
  if constexpr (MODE != WKV) return p.dk <= 64 ? launch<MODE, 128, 2>(p, T, stream) : launch<MODE, 128, 4>(p, T, stream);
  return ATOM_ERR_ARG;
}

// What all three take: sizes in steps of 8 (rows are read 16 bytes at a time), up to 128 key channels.
static bool sizes_ok(int H, int dk, int dv, int num_seqs) {
  return dk > 0 && dk <= 128 && dk % 8 == 0 && dv > 0 && dv % 8 == 0 && H > 0 && H <= 65535 && num_seqs <= 65535;
}
static bool aligned(const void* a) { return ((uintptr_t)a % 16) == 0; }

}  // namespace latc
}  // namespace atom

ATOM_EXPORT int atom_linear_tc_supports(int dk, int dv) { return atom::latc::sizes_ok(1, dk, dv, 1) ? 1 : 0; }
ATOM_EXPORT int atom_linear_tc_chunk(void) { return atom::latc::L; }

// scratch: the chunks' sums [ceil(T / 64) + num_seqs, H, dk, dv], then their decays [.., H, dk]; 16-byte aligned.
ATOM_EXPORT int atom_lightning_tc(float* out, const void* proj, int64_t ld, const float* decay, float* state, float* scratch,
                                  const int* cu_q, const int* state_slots, int num_seqs, int T, int H, int dk, int dv,
                                  int write_state, cudaStream_t stream) {
  using namespace atom::latc;
  if (T <= 0 || num_seqs <= 0) return ATOM_OK;
  if (!sizes_ok(H, dk, dv, num_seqs) || ld % 8 || !aligned(proj) || !aligned(out) || !aligned(state) || !aligned(scratch) || !scratch)
    return ATOM_ERR_ARG;
  const __nv_bfloat16* x = (const __nv_bfloat16*)proj;
  const int64_t slots = (T + L - 1) / L + num_seqs;
  Params p{};
  p.q = x;
  p.k = x + (int64_t)H * dk;
  p.v = x + 2 * (int64_t)H * dk;
  p.ld = p.ldv = ld;
  p.decay = decay;
  p.out = out;
  p.state = state;
  p.sB = scratch;
  p.sA = scratch + slots * H * dk * dv;
  p.cu_q = cu_q;
  p.state_slots = state_slots;
  p.num_seqs = num_seqs;
  p.H = H;
  p.dk = dk;
  p.dv = dv;
  p.write_state = write_state;
  return launch<LT>(p, T, stream);
}

// scratch_b: the chunks' sums; scratch_a: their decays [ceil(T / 64) + num_seqs, H, dk], then the logarithms' sums [T, H, dk].
ATOM_EXPORT int atom_gla_tc(float* out, const void* q, const void* k, const void* v, int64_t ld, const float* z, int64_t ldz,
                            const void* zb, int zb_dtype, float tau, float q_scale, float* state, float* scratch_b,
                            float* scratch_a, const int* cu_q, const int* state_slots, int num_seqs, int T, int H, int dk,
                            int dv, int write_state, cudaStream_t stream) {
  using namespace atom::latc;
  if (T <= 0 || num_seqs <= 0) return ATOM_OK;
  if (!sizes_ok(H, dk, dv, num_seqs) || ld % 8 || !aligned(q) || !aligned(k) || !aligned(v) || !aligned(out) || !aligned(state) ||
      !aligned(scratch_b) || !aligned(scratch_a) || !scratch_a || !scratch_b || !(tau > 0.f) ||
      (zb_dtype != ATOM_F32 && zb_dtype != ATOM_BF16))
    return ATOM_ERR_ARG;
  const int64_t slots = (T + L - 1) / L + num_seqs;
  Params p{};
  p.q = (const __nv_bfloat16*)q;
  p.k = (const __nv_bfloat16*)k;
  p.v = (const __nv_bfloat16*)v;
  p.ld = p.ldv = ld;
  p.z = z;
  p.ldz = ldz;
  p.zb = zb;
  p.zb_dtype = zb_dtype;
  p.inv_tau = 1.f / tau;
  p.q_scale = q_scale;
  p.out = out;
  p.state = state;
  p.g = scratch_a + slots * H * dk;
  p.sB = scratch_b;
  p.sA = scratch_a;
  p.cu_q = cu_q;
  p.state_slots = state_slots;
  p.num_seqs = num_seqs;
  p.H = H;
  p.dk = dk;
  p.dv = dv;
  p.write_state = write_state;
  return launch<GLA>(p, T, stream);
}

// As atom_wkv for dense bfloat16 rows, d in 32-bit, up to 64 value columns a head; scratch: the chunks' sums, their decays and
// the logarithms' sums one after another.
ATOM_EXPORT int atom_wkv_tc(void* y, const void* r, const void* k, const void* v, const float* d, const void* gate,
                            const void* w0, const void* u, const void* norm_w, int vec_dtype, float* state, float* scratch,
                            const int* cu_q, const int* state_slots, int num_seqs, int T, int H, int dk, int dv, float eps,
                            int write_state, cudaStream_t stream) {
  using namespace atom::latc;
  if (T <= 0 || num_seqs <= 0) return ATOM_OK;
  if (!sizes_ok(H, dk, dv, num_seqs) || dv > 64 || !aligned(r) || !aligned(k) || !aligned(v) || !aligned(gate) || !aligned(y) ||
      !aligned(state) || !aligned(scratch) || !scratch || (vec_dtype != ATOM_F32 && vec_dtype != ATOM_BF16))
    return ATOM_ERR_ARG;
  const int64_t slots = (T + L - 1) / L + num_seqs;
  Params p{};
  p.q = (const __nv_bfloat16*)r;
  p.k = (const __nv_bfloat16*)k;
  p.v = (const __nv_bfloat16*)v;
  p.ld = (int64_t)H * dk;
  p.ldv = (int64_t)H * dv;
  p.z = d;
  p.ldz = (int64_t)H * dk;
  p.zb = w0;
  p.zb_dtype = vec_dtype;
  p.u = u;
  p.norm_w = norm_w;
  p.gate = (const __nv_bfloat16*)gate;
  p.y = (__nv_bfloat16*)y;
  p.eps = eps;
  p.state = state;
  p.sB = scratch;
  p.sA = scratch + slots * H * dk * dv;
  p.g = p.sA + slots * H * dk;
  p.cu_q = cu_q;
  p.state_slots = state_slots;
  p.num_seqs = num_seqs;
  p.H = H;
  p.dk = dk;
  p.dv = dv;
  p.write_state = write_state;
  return launch<WKV>(p, T, stream);
}
