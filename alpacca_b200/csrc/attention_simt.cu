// Attention over the paged cache, one warp per (token, query head), plain
// 32-bit arithmetic.  It is the attention of the 32-bit path (T = float), for
// prefill and decode alike, and takes every head size up to 256; the bfloat16
// path uses it for head sizes that the tensor-core kernel refuses.
//
// For token t at position p of sequence b, head h reads KV head h / (H/K):
//   score_s = (q . k_s) * scale  for lo <= s <= p   (alpacca/model.py:447-467)
//   out = sum_s softmax(score)_s * v_s
// with lo = 0, or p - window + 1 when a window is given.  The softmax is the
// running (online) form, eight keys at a time in key order; a token's result
// does not depend on the rest of the batch.
//
// Row by row (attention_simt_kernel): bound by latency, a warp's keys follow one
// another.  One key at a time is five dependent shuffles, two exponentials and a
// load that nothing overlaps; eight at a time are eight loads in flight, nine
// shuffles for their sums and one rescaling.
// 333 tokens, 32 heads of 64 on 8, float32: 281 -> 169 us.
//
// Four heads of a KV head at a time (attention_rows_kernel; float32, heads of 64 or 128 that come in fours per KV head): a warp
// takes four heads of a token, and its block brings 32 keys and values at a time to shared memory by cp.async.  For the
// scores a lane has a key and forms its four products with the heads; the softmax is that of four runs of eight lanes; for
// the values a lane has its dimensions.  Every sum is formed in the order of the other kernel, operation by operation, so a
// row's bits do not depend on which of the two ran.  Bound by instructions (about nine per head and key and 32 lanes) where
// tokens share their keys, else by the chain of one warp.  us row by row / this, 32 heads on 8: 333 tokens, heads of 64
// 156 / 53, of 128 212 / 101; one token each of 1, 8 and 48 sequences, heads of 64, on one key 3.1 / 2.7, 3.2 / 2.8, 3.5 / 3.0,
// on 16 keys 6.7 / 4.5, 6.9 / 4.6, 7.3 / 5.0; of 8 on 2,000 keys 589 / 169, of 48 on 500 keys 271 / 51; of 200 sequences with
// heads of 128 on one key 7.5 / 11.6 (the one case that was seen slower), on 40 keys 39 / 26, on 500 keys 914 / 211.
#include "common.cuh"

#define KEYS 8      // keys that a warp takes at a time; the exchanges below are written for 8

__device__ __forceinline__ size_t key_place(const int* bt, int s, int K, int kh, int page_size, int D) {
  return (((size_t)bt[s / page_size] * K + kh) * page_size + s % page_size) * D;
}

// One row, a query head of a token at position pos, by one warp: q and o its D numbers, bt its sequence's row of the block table.
// WHOLE: pages hold a multiple of KEYS keys, so that a run of them lies in one page; others look up every key
template <typename T, int DPL, bool WHOLE>
__device__ __forceinline__ void walk_row(const T* __restrict__ qv, T* __restrict__ o, const T* __restrict__ k_pages,
                                         const T* __restrict__ v_pages, const int* __restrict__ bt, int pos, int kh, int K, int D,
                                         int page_size, float scale, int window) {
  const int lane = threadIdx.x & 31;
  float qr[DPL], acc[DPL];
#pragma unroll
  for (int j = 0; j < DPL; ++j) {
    const int d = lane + 32 * j;
    qr[j] = d < D ? to_f32(qv[d]) : 0.f;
    acc[j] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
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
    // a run without a score above -inf changes nothing (before the first such score all maxima are -inf)
    const float corr = m == m_new ? 1.f : expf(m - m_new);
    const float p = score == -INFINITY ? 0.f : expf(score - m_new);
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

template <typename T, int DPL, bool WHOLE>
__global__ void attention_simt_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out,
                                      const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                                      const int* __restrict__ block_table, int table_width,
                                      const int* __restrict__ tok_pos, const int* __restrict__ tok_seq,
                                      int n_tokens, int H, int K, int D, int page_size, float scale, int window) {
  const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= (long long)n_tokens * H) return;
  const int t = (int)(w / H), h = (int)(w - (long long)t * H);
  const int b = tok_seq[t];
  if (b < 0) return;
  walk_row<T, DPL, WHOLE>(q + (size_t)t * q_stride + (size_t)h * D, out + ((size_t)t * H + h) * D, k_pages, v_pages,
                          block_table + (size_t)b * table_width, tok_pos[t], h / (H / K), K, D, page_size, scale, window);
}

// float32, D = 32 DPL, pages of a multiple of KEYS keys; see the head of the file.
// TOKENS of a block: 8, a run of its sequence's, each a warp; or 1, of any sequence, whose four heads are one warp's (other
// warps help to load).  A token that sees a single run of KEYS keys goes row by row, without shared memory.
#define ROWS 4             // heads of a warp
#define STEP 32            // keys at a time
template <int DPL, int TOKENS, int WARPS, int BUFFERS> struct RowsShape {
  static constexpr int D = 32 * DPL;
  static constexpr int KP = D + 4;                                   // a lane per key reads 16 bytes of its row: no bank twice
  static constexpr int TILE = STEP * (KP + D);                       // floats of a step's keys and values
  static constexpr int Q = BUFFERS * TILE, P = Q + TOKENS * ROWS * D, SMEM = (P + TOKENS * ROWS * STEP) * 4;
};

template <int DPL, int TOKENS, int WARPS, int BUFFERS>
__global__ void __launch_bounds__(WARPS * 32)
attention_rows_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, const float* __restrict__ k_pages,
                      const float* __restrict__ v_pages, const int* __restrict__ block_table, int table_width,
                      const int* __restrict__ tok_pos, const int* __restrict__ tok_seq, const int* __restrict__ cu_q, int n_seqs,
                      int n_tokens, int H, int K, int page_size, float scale, int window) {
  using S = RowsShape<DPL, TOKENS, WARPS, BUFFERS>;
  constexpr int D = S::D, T = WARPS * 32;
  extern __shared__ __align__(16) float sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int h = blockIdx.y * ROWS, kh = h / (H / K);
  // this block's tokens: one, or the next of its sequence's runs of TOKENS (the last ones, which see most keys, first); a lane
  // per sequence looks for it
  int t0 = blockIdx.x, t_end = t0 + 1;
  if (TOKENS > 1) {
    int tile = gridDim.x - 1 - blockIdx.x;
    t_end = t0 = 0;
    for (int i0 = 0; i0 < n_seqs; i0 += 32) {
      const int i = i0 + lane, begin = i < n_seqs ? cu_q[i] : 0, end = i < n_seqs ? min(cu_q[i + 1], n_tokens) : 0;
      const int tiles = max(0, (end - begin + TOKENS - 1) / TOKENS);
      int upto = tiles;                            // runs of the lanes up to this one
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int before = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += before;
      }
      const unsigned found = __ballot_sync(0xffffffffu, tile < upto);
      if (found) {
        const int at = __ffs(found) - 1;
        const int from = begin + (tile - (upto - tiles)) * TOKENS;
        t0 = __shfl_sync(0xffffffffu, from, at);
        t_end = min(__shfl_sync(0xffffffffu, end, at), t0 + TOKENS);
        break;
      }
      tile -= __shfl_sync(0xffffffffu, upto, 31);
    }
  }
  if (t0 >= t_end) return;                         // more blocks than runs
  const int b = tok_seq[t0];
  if (b < 0) return;                               // rows without a sequence
  const int t = t0 + warp;
  const bool mine = t < t_end;
  const int pos = mine ? tok_pos[t] : -1;
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const int* bt = block_table + (size_t)b * table_width;
  if (TOKENS == 1) {
    const int p = tok_pos[t0];
    if (p < KEYS) {
#pragma unroll 1
      for (int i = h + warp; i < h + ROWS; i += WARPS)
        walk_row<float, DPL, true>(q + (size_t)t0 * q_stride + (size_t)i * D, out + ((size_t)t0 * H + i) * D, k_pages, v_pages, bt, p,
                                   kh, K, D, page_size, scale, window);
      return;
    }
  }
  float* q_s = sm + S::Q + warp * ROWS * D;
  float* p_s = sm + S::P + warp * ROWS * STEP;
  if (mine) {
#pragma unroll
    for (int i = 0; i < ROWS * DPL; ++i) q_s[lane + 32 * i] = q[(size_t)t * q_stride + (size_t)h * D + lane + 32 * i];
  }
  __syncwarp();
  float acc[ROWS][DPL], m[ROWS], l[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int j = 0; j < DPL; ++j) acc[r][j] = 0.f;
  }
  int from = 0x7fffffff, to = -1;                  // what the block's tokens see
  for (int i = t0; i < t_end; ++i) {
    const int p = tok_pos[i];
    to = max(to, p);
    from = min(from, (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0);
  }
  from -= from % KEYS;
  auto stage = [&](int s0, int buf) {
    if (s0 <= to) {
      float* k_t = sm + buf * S::TILE;
      for (int i = threadIdx.x; i < STEP * (D / 4); i += T) {
        const int row = i / (D / 4), c = i % (D / 4) * 4;
        const size_t at = key_place(bt, min(s0 + row, to), K, kh, page_size, D) + c;      // (past the end: no row uses it)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(k_t + row * S::KP + c)), "l"(k_pages + at));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(k_t + STEP * S::KP + row * D + c)), "l"(v_pages + at));
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int buf = 0;
  if (BUFFERS == 2) stage(from, 0);
  for (int s0 = from; s0 <= to; s0 += STEP, buf ^= BUFFERS - 1) {
    stage(BUFFERS == 2 ? s0 + STEP : s0, BUFFERS == 2 ? buf ^ 1 : 0);
    asm volatile("cp.async.wait_group %0;" ::"n"(BUFFERS - 1) : "memory");
    __syncthreads();
    if (mine && s0 <= pos && s0 + STEP > lo) {
      const float *k_row = sm + buf * S::TILE + lane * S::KP, *v_t = sm + buf * S::TILE + STEP * S::KP;
      // the products of dimensions d and d + 32 (.. + 96) first, then a tree over d: 16 apart, 8, 4, 2, 1
      auto part = [&](int a, float4* x) {      // d = 4 a .. 4 a + 3 of the four heads
        float4 kk[DPL];
#pragma unroll
        for (int j = 0; j < DPL; ++j) kk[j] = *reinterpret_cast<const float4*>(k_row + 32 * j + 4 * a);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          x[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int j = 0; j < DPL; ++j) {
            const float4 qq = *reinterpret_cast<const float4*>(q_s + r * D + 32 * j + 4 * a);
            x[r].x = fmaf(qq.x, kk[j].x, x[r].x);
            x[r].y = fmaf(qq.y, kk[j].y, x[r].y);
            x[r].z = fmaf(qq.z, kk[j].z, x[r].z);
            x[r].w = fmaf(qq.w, kk[j].w, x[r].w);
          }
        }
      };
      auto add = [](float4* x, const float4* y) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          x[r] = make_float4(__fadd_rn(x[r].x, y[r].x), __fadd_rn(x[r].y, y[r].y), __fadd_rn(x[r].z, y[r].z), __fadd_rn(x[r].w, y[r].w));
      };
      auto quarter = [&](int a, float4* x) {   // a, a + 4, a + 2, a + 6
        float4 y[ROWS], z[ROWS];
        part(a, x);
        part(a + 4, y);
        add(x, y);
        part(a + 2, y);
        part(a + 6, z);
        add(y, z);
        add(x, y);
      };
      float4 even[ROWS], odd[ROWS];
      quarter(0, even);
      quarter(1, odd);
      add(even, odd);
      // four runs of eight keys: a run's lanes have its scores, and every lane follows the runs before its own
      const int key = s0 + lane, run = lane >> 3;
      float corr[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const float dot = __fadd_rn(__fadd_rn(even[r].x, even[r].z), __fadd_rn(even[r].y, even[r].w));
        const float score = key < lo || key > pos ? -INFINITY : __fmul_rn(dot, scale);
        float top = score;
#pragma unroll
        for (int o = 1; o < KEYS; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        float before = m[r], after = m[r];       // the maximum before and after this lane's run
#pragma unroll
        for (int g = 0; g < STEP / KEYS; ++g) {
          const float run_top = __shfl_sync(0xffffffffu, top, g * KEYS);
          if (g < run) before = fmaxf(before, run_top);
          if (g <= run) after = fmaxf(after, run_top);
          m[r] = fmaxf(m[r], run_top);
        }
        // a run without a visible key changes nothing (before the first one all maxima are -inf)
        corr[r] = after == before ? 1.0f : expf(before - after);
        const float p = score == -INFINITY ? 0.f : expf(score - after);
        float sum = p;
#pragma unroll
        for (int o = 1; o < KEYS; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
        for (int g = 0; g < STEP / KEYS; ++g)
          l[r] = fmaf(l[r], __shfl_sync(0xffffffffu, corr[r], g * KEYS), __shfl_sync(0xffffffffu, sum, g * KEYS));
        p_s[r * STEP + lane] = p;
      }
      __syncwarp();
#pragma unroll
      for (int g = 0; g < STEP / KEYS; ++g) {
        const int g0 = s0 + g * KEYS;
        if (g0 > pos || g0 + KEYS <= lo) continue;             // the same for the whole warp
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const float c = __shfl_sync(0xffffffffu, corr[r], g * KEYS);
#pragma unroll
          for (int j = 0; j < DPL; ++j) acc[r][j] *= c;
        }
        const bool whole = g0 >= lo && g0 + KEYS - 1 <= pos;
#pragma unroll
        for (int i0 = 0; i0 < KEYS; i0 += 4) {
          float4 pr[ROWS];
#pragma unroll
          for (int r = 0; r < ROWS; ++r) pr[r] = *reinterpret_cast<const float4*>(p_s + r * STEP + g * KEYS + i0);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int s = g0 + i0 + i;
            if (!whole && (s < lo || s > pos)) continue;
            const float* v_row = v_t + (g * KEYS + i0 + i) * D + DPL * lane;
            float v[DPL];
            if constexpr (DPL == 2) *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(v_row);
            else *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(v_row);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
              const float p = i == 0 ? pr[r].x : i == 1 ? pr[r].y : i == 2 ? pr[r].z : pr[r].w;
#pragma unroll
              for (int j = 0; j < DPL; ++j) acc[r][j] = fmaf(p, v[j], acc[r][j]);
            }
          }
        }
      }
    }
    __syncthreads();                             // the buffer may be filled again
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (!mine) return;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float inv = 1.0f / l[r];
    float* o = out + ((size_t)t * H + h + r) * D + DPL * lane;
#pragma unroll
    for (int j = 0; j < DPL; ++j) o[j] = acc[r][j] * inv;
  }
}

struct RowsArgs {
  const float* q;
  int q_stride;
  float* out;
  const float *k_pages, *v_pages;
  const int* block_table;
  int table_width;
  const int *tok_pos, *tok_seq, *cu_q;
  int n_seqs, n_tokens, H, K, page_size;
  float scale;
  int window;
  cudaStream_t stream;
};
template <int DPL, int TOKENS, int WARPS, int BUFFERS>
static int launch_rows(const RowsArgs& a) {
  using S = RowsShape<DPL, TOKENS, WARPS, BUFFERS>;
  auto kernel = attention_rows_kernel<DPL, TOKENS, WARPS, BUFFERS>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
  if (e != cudaSuccess) return AB_CUDA_ERR + (int)e;
  // (a sequence's last run may be short: at most n_seqs more than the tokens fill)
  const dim3 grid((unsigned)(TOKENS > 1 ? (a.n_tokens + TOKENS - 1) / TOKENS + a.n_seqs : a.n_tokens), (unsigned)(a.H / ROWS));
  kernel<<<grid, WARPS * 32, S::SMEM, a.stream>>>(a.q, a.q_stride, a.out, a.k_pages, a.v_pages, a.block_table, a.table_width,
                                                     a.tok_pos, a.tok_seq, a.cu_q, a.n_seqs, a.n_tokens, a.H, a.K, a.page_size,
                                                     a.scale, a.window);
  return ab_launch_status();
}
// Runs of eight tokens where sequences bring four or more on average or the runs leave processors idle (32 heads of 128, us in
// runs / token by token: 100 sequences of 3 tokens on 40 keys 76 / 37, 8 of 3 on 700 87 / 97), else a block per token: while
// there is a processor for each, with seven warps that help to load (one token on 4,000 keys, 1 / 4 / 8 warps 626 / 533 /
// 460); up to three blocks a processor, with three (48 tokens of 32 heads on 500 keys 87 / 74 / 181); more, one warp and one
// buffer, twelve a processor (200 tokens 210 / 282 / 660).
template <int DPL>
static int launch_rows(RowsArgs a) {
  if (a.cu_q && (a.n_tokens >= 4LL * a.n_seqs || (long long)a.n_seqs * (a.H / ROWS) <= 148)) return launch_rows<DPL, 8, 8, 2>(a);
  const long long blocks = (long long)a.n_tokens * (a.H / ROWS);
  return blocks <= 148 ? launch_rows<DPL, 1, 8, 2>(a) : blocks <= 444 ? launch_rows<DPL, 1, 4, 2>(a) : launch_rows<DPL, 1, 1, 1>(a);
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

// cu_q (int [n_seqs + 1], or null): where the sequences' tokens begin, in prompts.  `single`: one token per sequence.  With one of
// the two, the kernel of four heads is taken where it can be; the results are the same.
AB_API int ab_attention_simt(const void* q, int q_stride, void* out, int dtype, const void* k_pages, const void* v_pages,
                             const int* block_table, int table_width, const int* tok_pos, const int* tok_seq, const int* cu_q,
                             int n_seqs, int single, int n_tokens, int H, int K, int D, int page_size, float scale, int window,
                             cudaStream_t stream) {
  if (n_tokens <= 0) return AB_OK;
  if (D <= 0 || D > 256 || H <= 0 || K <= 0 || H % K || page_size <= 0) return AB_BAD_ARG;
  if ((cu_q || single) && dtype == AB_F32 && (D == 64 || D == 128) && H / K % ROWS == 0 && H / ROWS <= 65535 && page_size % KEYS == 0 &&
      (((uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0) {
    const RowsArgs a{(const float*)q, q_stride, (float*)out, (const float*)k_pages, (const float*)v_pages, block_table, table_width,
                     tok_pos, tok_seq, single ? nullptr : cu_q, n_seqs, n_tokens, H, K, page_size, scale, window, stream};
    return D == 64 ? launch_rows<2>(a) : launch_rows<4>(a);
  }
  if (dtype == AB_F32)
    return launch<float>(q, q_stride, out, k_pages, v_pages, block_table, table_width, tok_pos, tok_seq,
                         n_tokens, H, K, D, page_size, scale, window, stream);
  if (dtype == AB_BF16)
    return launch<bf16>(q, q_stride, out, k_pages, v_pages, block_table, table_width, tok_pos, tok_seq,
                        n_tokens, H, K, D, page_size, scale, window, stream);
  return AB_BAD_ARG;
}
