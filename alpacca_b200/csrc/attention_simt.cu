// Attention over the paged cache, one warp per (token, query head), plain
// 32-bit arithmetic.  It is the attention of the 32-bit path (T = float), for
// prefill and decode alike, and takes every head size up to 256; the bfloat16
// path uses it for head sizes that the tensor-core kernel refuses.
//
// For token t at position p of sequence b, head h reads KV head h / (H/K):
//   score_s = (q . k_s) * scale  for lo <= s <= p   (alpacca/model.py:447-467)
//   out = sum_s softmax(score)_s * v_s
// with lo = 0, or p - window + 1 when a window is given.  The softmax is the
// running (online) form, eight keys at a time in key order; nothing is shared
// between warps, so a token's result does not depend on the rest of the batch.
//
// Bound by latency: a warp's keys follow one another.  One key at a time is five
// dependent shuffles, two exponentials and a load that nothing overlaps; eight at
// a time are eight loads in flight, nine shuffles for their sums and one rescaling.
// 333 tokens, 32 heads of 64 on 8, float32: 281 -> 169 us.
#include "common.cuh"

#define KEYS 8      // keys that a warp takes at a time; the exchanges below are written for 8

__device__ __forceinline__ size_t key_place(const int* bt, int s, int K, int kh, int page_size, int D) {
  return (((size_t)bt[s / page_size] * K + kh) * page_size + s % page_size) * D;
}

// WHOLE: pages hold a multiple of KEYS keys, so that a run of them lies in one page; others look up every key
template <typename T, int DPL, bool WHOLE>
__global__ void attention_simt_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out,
                                      const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                                      const int* __restrict__ block_table, int table_width,
                                      const int* __restrict__ tok_pos, const int* __restrict__ tok_seq,
                                      int n_tokens, int H, int K, int D, int page_size, float scale, int window) {
  const int lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= (long long)n_tokens * H) return;
  const int t = (int)(w / H), h = (int)(w - (long long)t * H);
  const int b = tok_seq[t];
  T* o = out + ((size_t)t * H + h) * D;
  if (b < 0) return;
  const int pos = tok_pos[t];
  const int kh = h / (H / K);
  const T* qv = q + (size_t)t * q_stride + (size_t)h * D;
  float qr[DPL], acc[DPL];
#pragma unroll
  for (int j = 0; j < DPL; ++j) {
    const int d = lane + 32 * j;
    qr[j] = d < D ? to_f32(qv[d]) : 0.f;
    acc[j] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const int* bt = block_table + (size_t)b * table_width;
  // KEYS keys at a time (a run starts at a multiple of KEYS, so it does not depend on where the walk began)
  for (int s0 = lo - lo % KEYS; s0 <= pos; s0 += KEYS) {
    const size_t base = key_place(bt, s0, K, kh, page_size, D);
    const T *k_run = k_pages + base, *v_run = v_pages + base;
    float v[KEYS];
#pragma unroll
    for (int i = 0; i < KEYS; ++i) {
      // a key outside lo .. pos gets no weight
      const T* kv = k_run + (size_t)i * D;
      if constexpr (!WHOLE) kv = k_pages + key_place(bt, min(s0 + i, pos), K, kh, page_size, D);
      float part = 0.f;
#pragma unroll
      for (int j = 0; j < DPL; ++j) {
        const int d = lane + 32 * j;
        if (d < D) part += qr[j] * to_f32(kv[d]);
      }
      v[i] = part;
    }
    // the eight sums over the lanes side by side: each exchange halves the keys that a lane looks after
#pragma unroll
    for (int half = KEYS / 2, o = 16; half >= 1; half >>= 1, o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float give = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    const int mine = s0 + (lane >> 2);               // the key whose score this lane (and three others) holds
    const float score = mine < lo || mine > pos ? -INFINITY : v[0] * scale;
    float m_new = score;
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, o));
    m_new = fmaxf(m, m_new);
    const float corr = expf(m - m_new);              // exp(-inf) = 0 on the first run
    const float p = expf(score - m_new);
    float sum = p;
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    l = l * corr + sum;
#pragma unroll
    for (int j = 0; j < DPL; ++j) acc[j] *= corr;
#pragma unroll
    for (int i = 0; i < KEYS; ++i) {
      const float pi = __shfl_sync(0xffffffffu, p, 4 * i);
      if (s0 + i < lo || s0 + i > pos) continue;     // the same for the whole warp
      if constexpr (!WHOLE) v_run = v_pages + key_place(bt, s0 + i, K, kh, page_size, D) - (size_t)i * D;
#pragma unroll
      for (int j = 0; j < DPL; ++j) {
        const int d = lane + 32 * j;
        if (d < D) acc[j] += pi * to_f32(v_run[(size_t)i * D + d]);
      }
    }
    m = m_new;
  }
  const float inv = 1.0f / l;
#pragma unroll
  for (int j = 0; j < DPL; ++j) {
    const int d = lane + 32 * j;
    if (d < D) o[d] = from_f32<T>(acc[j] * inv);
  }
}

template <typename T>
static int launch(const void* q, int q_stride, void* out, const void* k_pages, const void* v_pages,
                  const int* block_table, int table_width, const int* tok_pos, const int* tok_seq, int n_tokens,
                  int H, int K, int D, int page_size, float scale, int window, cudaStream_t stream) {
  const long long warps = (long long)n_tokens * H;
  const int wpb = 4;
  const unsigned blocks = (unsigned)((warps + wpb - 1) / wpb);
  const bool whole = page_size % KEYS == 0;
#define AB_GO(DPL)                                                                                       \
  (whole ? attention_simt_kernel<T, DPL, true> : attention_simt_kernel<T, DPL, false>)<<<blocks, wpb * 32, 0, stream>>>(                                        \
      (const T*)q, q_stride, (T*)out, (const T*)k_pages, (const T*)v_pages, block_table, table_width,   \
      tok_pos, tok_seq, n_tokens, H, K, D, page_size, scale, window)
  if (D <= 32) AB_GO(1);
  else if (D <= 64) AB_GO(2);
  else if (D <= 128) AB_GO(4);
  else AB_GO(8);
#undef AB_GO
  return ab_launch_status();
}

AB_API int ab_attention_simt(const void* q, int q_stride, void* out, int dtype, const void* k_pages,
                             const void* v_pages, const int* block_table, int table_width, const int* tok_pos,
                             const int* tok_seq, int n_tokens, int H, int K, int D, int page_size, float scale,
                             int window, cudaStream_t stream) {
  if (n_tokens <= 0) return AB_OK;
  if (D <= 0 || D > 256 || H <= 0 || K <= 0 || H % K || page_size <= 0) return AB_BAD_ARG;
  if (dtype == AB_F32)
    return launch<float>(q, q_stride, out, k_pages, v_pages, block_table, table_width, tok_pos, tok_seq,
                         n_tokens, H, K, D, page_size, scale, window, stream);
  if (dtype == AB_BF16)
    return launch<bf16>(q, q_stride, out, k_pages, v_pages, block_table, table_width, tok_pos, tok_seq,
                        n_tokens, H, K, D, page_size, scale, window, stream);
  return AB_BAD_ARG;
}
