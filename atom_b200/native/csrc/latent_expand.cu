// What attention through a latent needs before keys and values are built per head (bfloat16): the cached rows that a step's
// requests see, one request after another, in one array; and the queries' rotated parts, in place.  One launch: the first CTAs
// copy eight rows each (a warp per row, 16 bytes a lane), the others rotate a token each.
#include "common.cuh"

namespace atom {

// dense [keys, D] <- pages [pages, page_size, D]; request s has rows for the keys from max(0, its first position - window + 1)
// (0 without a window) to its last.  q: [T, heads] vectors of `vec` numbers, rows q_ld apart, whose numbers off .. off + dims - 1
// are rotated (pairs (i, i + dims / 2)) by position * freq, times mag.
__global__ void __launch_bounds__(256)
latent_expand_kernel(__nv_bfloat16* __restrict__ dense, const __nv_bfloat16* __restrict__ pages, int D, int page_size,
                     const int* __restrict__ block_table, int table_width, const int* __restrict__ cu_q, const int* __restrict__ ctx_len,
                     int num_seqs, int window, int64_t keys, int copy_ctas, __nv_bfloat16* __restrict__ q, int64_t q_ld, int heads, int vec,
                     int off, int dims, const float* __restrict__ freq, float mag, const int* __restrict__ positions,
                     const int* __restrict__ seq_of_token) {
  atom::pdl_trigger();
  atom::pdl_wait();
  if ((int)blockIdx.x < copy_ctas) {
    const int lane = threadIdx.x & 31;
    int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= keys) return;
    const int64_t to = row;
    int s = 0, first = 0;
    for (; s < num_seqs; ++s) {
      const int n = cu_q[s + 1] - cu_q[s];
      if (n <= 0) continue;
      const int start = ctx_len[s] - n;
      first = window > 0 ? max(0, start - window + 1) : 0;
      if (row < ctx_len[s] - first) break;
      row -= ctx_len[s] - first;
    }
    if (s == num_seqs) return;
    const int key = first + (int)row;
    const int page = block_table[(int64_t)s * table_width + key / page_size];
    if (page < 0) return;
    const uint4* src = reinterpret_cast<const uint4*>(pages + ((int64_t)page * page_size + key % page_size) * D);
    uint4* dst = reinterpret_cast<uint4*>(dense + to * D);
    for (int i = lane; i < D / 8; i += 32) dst[i] = src[i];
    return;
  }
  const int t = blockIdx.x - copy_ctas;
  if (seq_of_token[t] < 0) return;
  const float pos = (float)positions[t];
  const int half = dims / 2;
  for (int e = threadIdx.x; e < heads * half; e += blockDim.x) {
    const int h = e / half, i = e - h * half;
    __nv_bfloat16* v = q + (int64_t)t * q_ld + (int64_t)h * vec + off + i;
    float s, c;
    sincosf(pos * freq[i], &s, &c);
    s *= mag;
    c *= mag;
    const float a = __bfloat162float(v[0]), b = __bfloat162float(v[half]);
    v[0] = __float2bfloat16_rn(a * c - b * s);
    v[half] = __float2bfloat16_rn(b * c + a * s);
  }
}

}  // namespace atom

ATOM_EXPORT int atom_latent_expand(void* dense, const void* pages, int D, int page_size, const int* block_table, int table_width,
                                   const int* cu_q, const int* ctx_len, int num_seqs, int window, int64_t keys, void* q, int64_t q_ld,
                                   int heads, int vec, int off, int dims, const float* freq, float mag, const int* positions,
                                   const int* seq_of_token, int T, cudaStream_t stream) {
  if (T <= 0 || num_seqs <= 0 || keys <= 0) return ATOM_OK;
  if (D <= 0 || D % 8 || page_size <= 0 || keys > (1LL << 30) || dims < 0 || dims % 2 || off + dims > vec || (((uintptr_t)dense | (uintptr_t)pages) % 16) != 0)
    return ATOM_ERR_ARG;
  const int copy_ctas = (int)((keys + 7) / 8);
  atom::launch_pdl(atom::latent_expand_kernel, dim3(copy_ctas + (dims > 0 ? T : 0)), dim3(256), 0, stream, (__nv_bfloat16*)dense,
                   (const __nv_bfloat16*)pages, D, page_size, block_table, table_width, cu_q, ctx_len, num_seqs, window, keys, copy_ctas,
                   (__nv_bfloat16*)q, q_ld, heads, vec, off, dims, freq, mag, positions, seq_of_token);
  return atom::check_launch();
}
