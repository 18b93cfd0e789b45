// Causal attention of prompts over a cached latent on the fifth-generation tensor cores (bfloat16): all H heads of a token
// read the same row per position, [c (C dims) | r (R dims)], Dk = C + R up to 256 in steps of 16; a head's value at a
// position is the row's first C dims.
//
// A CTA owns up to 128 query rows: the H heads of floor(128 / H) consecutive tokens of one sequence.  Keys are visited 128 at
// a time (two pages, TMA boxes of 64 rows x 64 dims, 128-byte swizzle).  A tile of rows is brought to shared memory ONCE and
// read twice: as the K-major second operand of S = Q K^T and as the MN-major second operand of O += P V.
//
//   MMA warp      S_j = Q K_j^T     (M 128, N 128, K = Dk)        -> TMEM, two buffers
//   softmax warps S_j from TMEM (a row per thread), scale, mask, maximum and sum, P_j = 2^(s - m) in bfloat16 -> TMEM, over
//                 the first half of its S_j
//   MMA warp      O += P_j V_j      (M 128, N = C up to a multiple of 16, K 128)  -> TMEM
//
// The reference m of a row follows its maximum lazily, as in attention_tc.cu; every mbarrier wait is bounded
// (attention_tc.cuh).  What bounds it: the MMAs and the softmax of a tile take about as long as each other
// (1,024 + 900 clocks of MMA at full rate, 1,024 of the exponentials' unit), and a CTA has two tiles in hand.  16 heads, 224 +
// 32 dims: 2,000 tokens on 1,000 held ones 73 us, 842 TFLOP/s (mma.sync tiles: 437 us); 500 tokens 14 us (37).
#include "attention_tc.cuh"
#include "common.cuh"
#include "launch.cuh"

#define LT_ROWS 128
#define LT_PAGE 64
#define LT_KEYS 128
#define LT_THREADS 192

// Panels of [128 rows][64 dims] = 128-byte rows, 1024-byte aligned: PANELS of them for Q, then STAGES tiles of keys.  TMEM:
// S at columns 0 and 128 (P over the first half of each), O from column 256: all 512, one CTA per SM.
template <int PANELS> struct LtShape {
  static constexpr int STAGES = PANELS == 4 ? 2 : (PANELS == 3 ? 3 : 4);
  static constexpr int PANEL = 128 * 128;
  static constexpr int TILE = PANELS * PANEL;
  static constexpr int BAR_OFF = TILE * (1 + STAGES);
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

template <int PANELS>
__global__ void __launch_bounds__(LT_THREADS, 1)
attention_latent_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           bf16* __restrict__ out, const int* __restrict__ block_table, int table_width,
                           const int* __restrict__ tok_pos, const int* __restrict__ cu_q,
                           const int* __restrict__ tile_seq, const int* __restrict__ tile_q0, int H, int Dk, int C,
                           float scale_log2, int window, int tokens_per_tile, int* __restrict__ status,
                           const float* __restrict__ sink) {
  using Sh = LtShape<PANELS>;
  constexpr int STAGES = Sh::STAGES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* q_full = reinterpret_cast<uint64_t*>(base + Sh::BAR_OFF);      // 1
  uint64_t* k_full = q_full + 1;                 // STAGES
  uint64_t* k_empty = k_full + STAGES;           // STAGES
  uint64_t* s_full = k_empty + STAGES;           // 2
  uint64_t* p_full = s_full + 2;                 // 2
  // 2, for even and odd j: completes once per product O += P_j V_j (a warp that waits for product j may come when product
  // j - 1 is not done yet, which one barrier could not tell from product j)
  uint64_t* o_done = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    at_bar_init(q_full, 1);
    for (int s = 0; s < STAGES; ++s) { at_bar_init(k_full + s, 1); at_bar_init(k_empty + s, 1); }
    for (int i = 0; i < 2; ++i) { at_bar_init(s_full + i, 1); at_bar_init(p_full + i, 128); at_bar_init(o_done + i, 1); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t o_col = 256;
  pdl_wait();
  pdl_trigger();

  const int tile = blockIdx.x;
  const int b = tile_seq[tile], q0 = tile_q0[tile];
  const int n_tok = min(tokens_per_tile, cu_q[b + 1] - q0);
  const int n_rows = n_tok * H;
  const int pos_first = tok_pos[q0], pos_last = tok_pos[q0 + n_tok - 1];
  const int page_begin = (window > 0 && pos_first - window + 1 > 0) ? (pos_first - window + 1) / LT_PAGE : 0;
  const int page_end = pos_last / LT_PAGE + 1;
  const int n_tiles = (page_end - page_begin + 1) / 2;
  const int* bt = block_table + (size_t)b * table_width;

  if (warp == 0) {
    if (lane == 0) {
      // the box holds tokens_per_tile x H rows (all counted, also where they lie past the sequence's end and become zeros);
      // rows of the tile past the box are never written and stay in their own rows of S, P and O, which nobody stores
      at_expect_tx(q_full, PANELS * tokens_per_tile * H * 128);
      for (int p = 0; p < PANELS; ++p) at_tma_3d(base + p * Sh::PANEL, &map_q, p * 64, 0, q0, q_full);
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % STAGES;
        if (j >= STAGES && !at_wait(k_empty + s, ((j / STAGES) - 1) & 1)) { atomicExch(status, 21); break; }
        const int i0 = page_begin + 2 * j, i1 = min(i0 + 1, page_end - 1);      // an odd last page stands twice; its copy is masked
        const int r0 = bt[i0] * LT_PAGE, r1 = bt[i1] * LT_PAGE;
        unsigned char* dst = base + Sh::TILE * (1 + s);
        at_expect_tx(k_full + s, Sh::TILE);
        for (int p = 0; p < PANELS; ++p) {
          at_tma_2d(dst + p * Sh::PANEL, &map_k, p * 64, r0, k_full + s);
          at_tma_2d(dst + p * Sh::PANEL + LT_PAGE * 128, &map_k, p * 64, r1, k_full + s);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // S = Q K^T: both operands K-major, N = 128;  O += P V: P from TMEM, V = the tile's first dims, MN-major
      constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_KEYS >> 3) << 17) |
                                   ((uint32_t)(LT_ROWS >> 4) << 24);
      const uint32_t n_v = (uint32_t)(C + 15) / 16 * 16;
      const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((n_v >> 3) << 17) |
                               ((uint32_t)(LT_ROWS >> 4) << 24);
      const uint32_t q_addr = at_smem(base);
      const int steps = Dk / 16;
      bool ok = at_wait(q_full, 0);
      if (!ok) atomicExch(status, 22);
      auto issue_s = [&](int j) {
        const int s = j % STAGES;
        if (!at_wait(k_full + s, (j / STAGES) & 1)) { atomicExch(status, 23); ok = false; return; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t k_addr = at_smem(base + Sh::TILE * (1 + s));
        for (int k = 0; k < steps; ++k)      // 16 dims per MMA: 32 bytes along a panel's rows
          at_mma(tmem + (j & 1) * 128, at_desc(q_addr + (k >> 2) * Sh::PANEL + (k & 3) * 32),
                 at_desc(k_addr + (k >> 2) * Sh::PANEL + (k & 3) * 32), idesc_s, k > 0 ? 1u : 0u);
        at_commit(s_full + (j & 1));
      };
      if (ok) issue_s(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) issue_s(j + 1);        // the next tile's scores run while this tile's softmax does
        if (!ok) break;
        if (!at_wait(p_full + (j & 1), (j >> 1) & 1)) { atomicExch(status, 24); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int s = j % STAGES;
        const uint32_t v_addr = at_smem(base + Sh::TILE * (1 + s));
#pragma unroll
        for (int k = 0; k < LT_KEYS / 16; ++k)     // 16 keys per MMA: 8 columns of P, 2 groups of 8 rows of the tile
          at_mma_ts(tmem + o_col, tmem + (j & 1) * 128 + k * 8, at_desc_mn(v_addr + k * 2048, Sh::PANEL), idesc_o,
                    (j > 0 || k > 0) ? 1u : 0u);
        at_commit(o_done + (j & 1));
        at_commit(k_empty + s);
      }
    }
  } else {
    // softmax warps 2..5: TMEM lanes 32 * (warp % 4) ..; thread = query row
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const bool row_ok = r < n_rows;
    int pos = 0x3fffffff, lo = 0;
    if (row_ok) {
      pos = tok_pos[q0 + r / H];
      lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    }
    float m_ref = -INFINITY, l_run = 0.f;       // the row's reference and its sum of 2^(s - m_ref)
    bool ok = true;
    for (int j = 0; j < n_tiles && ok; ++j) {
      if (!at_wait(s_full + (j & 1), (j >> 1) & 1)) { atomicExch(status, 26); ok = false; }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float sc[LT_KEYS];
      const uint32_t s_col = tmem + lane_base + (j & 1) * 128;
#pragma unroll
      for (int c0 = 0; c0 < LT_KEYS; c0 += 16) at_ld16(s_col + c0, sc + c0);
      at_ld_wait();
      const int key0 = (page_begin + 2 * j) * LT_PAGE;
      if (key0 + LT_KEYS - 1 > pos_first || window > 0) {
#pragma unroll
        for (int c = 0; c < LT_KEYS; ++c)
          if (key0 + c > pos || key0 + c < lo) sc[c] = -INFINITY;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < LT_KEYS; c += 4) {
        mx4[0] = fmaxf(mx4[0], sc[c]);
        mx4[1] = fmaxf(mx4[1], sc[c + 1]);
        mx4[2] = fmaxf(mx4[2], sc[c + 2]);
        mx4[3] = fmaxf(mx4[3], sc[c + 3]);
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
      const bool move = (mx > m_ref + AT_LAZY) || (m_ref == -INFINITY && mx > -INFINITY);
      float corr = 1.f;
      if (move) {
        corr = (m_ref == -INFINITY) ? 0.f : at_exp2(m_ref - mx);
        m_ref = mx;
        l_run *= corr;
      }
      const float sub = (m_ref == -INFINITY) ? 0.f : m_ref;
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c0 = 0; c0 < LT_KEYS; c0 += 32) {
        uint32_t packed[16];
#pragma unroll
        for (int c = c0; c < c0 + 32; c += 4) {
          const float p0 = at_exp2(fmaf(sc[c], scale_log2, -sub)), p1 = at_exp2(fmaf(sc[c + 1], scale_log2, -sub));
          const float p2 = at_exp2(fmaf(sc[c + 2], scale_log2, -sub)), p3 = at_exp2(fmaf(sc[c + 3], scale_log2, -sub));
          sum4[0] += p0; sum4[1] += p1; sum4[2] += p2; sum4[3] += p3;
          __nv_bfloat162 pa = __floats2bfloat162_rn(p0, p1), pb = __floats2bfloat162_rn(p2, p3);
          packed[(c - c0) >> 1] = *reinterpret_cast<uint32_t*>(&pa);
          packed[((c - c0) >> 1) + 1] = *reinterpret_cast<uint32_t*>(&pb);
        }
        at_st16u(s_col + c0 / 2, packed);        // P row: two keys per column of this thread's lane
      }
      l_run += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
      if (j > 0 && __any_sync(0xffffffffu, move)) {
        // rescale this warp's rows of O in TMEM, after the product before this tile has landed there
        if (!at_wait(o_done + ((j - 1) & 1), ((j - 1) >> 1) & 1)) { atomicExch(status, 25); ok = false; }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int c0 = 0; c0 < C; c0 += 16) {
          float t[16];
          at_ld16(tmem + lane_base + o_col + c0, t);
          at_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c) t[c] *= corr;
          at_st16(tmem + lane_base + o_col + c0, t);
        }
      }
      at_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      at_arrive(p_full + (j & 1));
    }
    if (ok) {
      if (!at_wait(o_done + ((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1)) { atomicExch(status, 27); ok = false; }
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // the sink: one more term of the denominator, without a value
      if (sink != nullptr && row_ok && m_ref > -INFINITY) l_run += exp2f(sink[r % H] * AT_LOG2E - m_ref);
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      bf16* dst = out + ((size_t)(q0 + r / H) * H + r % H) * Dk;
      for (int c0 = 0; c0 < C; c0 += 16) {       // up to a multiple of 16, which the row has
        float t[16];
        at_ld16(tmem + lane_base + o_col + c0, t);
        at_ld_wait();
        if (row_ok) {
          uint32_t w[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            __nv_bfloat162 pr = __floats2bfloat162_rn(t[2 * e] * inv, t[2 * e + 1] * inv);
            w[e] = *reinterpret_cast<uint32_t*>(&pr);
          }
          *reinterpret_cast<uint4*>(dst + c0) = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4*>(dst + c0 + 8) = make_uint4(w[4], w[5], w[6], w[7]);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

static int* lt_status_word() {
  static int* p[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!p[dev]) {
    if (cudaMalloc(&p[dev], sizeof(int)) != cudaSuccess) return nullptr;
    cudaMemset(p[dev], 0, sizeof(int));
  }
  return p[dev];
}
AB_API int ab_attention_latent_tc_status() {
  int* p = lt_status_word();
  if (!p) return -1;
  int v = 0;
  if (cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (v) cudaMemset(p, 0, sizeof(int));
  return v;
}

// 1 if this kernel takes the sizes: rows of Dk = C + R dims in steps of 16 up to 256, up to 128 heads
AB_API int ab_attention_latent_tc_supports(int H, int C, int R) {
  return H > 0 && H <= LT_ROWS && C > 0 && R >= 0 && (C + R) % 16 == 0 && C + R <= 256;
}

// q, out [n_tokens, H, C + R] (16-byte aligned; of out's rows the first C dims up to a multiple of 16 are written); pages
// [n_pages, 64, C + R]; tile_seq / tile_q0: the tiles of floor(128 / H) tokens (sequence, first packed token); sink: float
// [H] or null
AB_API int ab_attention_latent_tc(const void* q, int n_tokens, void* out, const void* pages, int n_pages,
                                  const int* block_table, int table_width, const int* tok_pos, const int* cu_q,
                                  const int* tile_seq, const int* tile_q0, int n_tiles, int H, int C, int R, float scale,
                                  int window, const float* sink, cudaStream_t stream) {
  if (n_tiles <= 0) return AB_OK;
  if (!ab_attention_latent_tc_supports(H, C, R) || ((uintptr_t)out & 15)) return AB_BAD_ARG;
  AtEncodeFn enc = at_encode_fn();
  int* status = lt_status_word();
  if (!enc || !status) return AB_BAD_ARG;
  const int Dk = C + R, tpt = LT_ROWS / H;
  CUtensorMap mq, mk;
  {
    cuuint64_t dims[3] = {(cuuint64_t)Dk, (cuuint64_t)H, (cuuint64_t)n_tokens};
    cuuint64_t strides[2] = {(cuuint64_t)Dk * 2, (cuuint64_t)H * Dk * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)H, (cuuint32_t)tpt};          // one panel: 64 dims; zeros past Dk
    cuuint32_t elem[3] = {1, 1, 1};
    if (enc(&mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return AB_BAD_ARG;
  }
  {
    cuuint64_t dims[2] = {(cuuint64_t)Dk, (cuuint64_t)n_pages * LT_PAGE};
    cuuint64_t strides[1] = {(cuuint64_t)Dk * 2};
    cuuint32_t box[2] = {64, LT_PAGE};
    cuuint32_t elem[2] = {1, 1};
    if (enc(&mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(pages), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return AB_BAD_ARG;
  }
  cudaError_t e;
#define LT_GO(P)                                                                                                        \
  {                                                                                                                     \
    e = cudaFuncSetAttribute(attention_latent_tc_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize,                \
                             LtShape<P>::TOTAL);                                                                        \
    if (e != cudaSuccess) return AB_CUDA_ERR + (int)e;                                                                  \
    e = ab_launch(attention_latent_tc_kernel<P>, dim3((unsigned)n_tiles), dim3(LT_THREADS), LtShape<P>::TOTAL, stream,  \
                  mq, mk, (bf16*)out, block_table, table_width, tok_pos, cu_q, tile_seq, tile_q0, H, Dk, C,             \
                  scale * AT_LOG2E, window, tpt, status, sink);                                                         \
  }
  switch ((Dk + 63) / 64) {
    case 1: LT_GO(1) break;
    case 2: LT_GO(2) break;
    case 3: LT_GO(3) break;
    default: LT_GO(4) break;
  }
#undef LT_GO
  if (e != cudaSuccess) return AB_CUDA_ERR + (int)e;
  return ab_launch_status();
}
