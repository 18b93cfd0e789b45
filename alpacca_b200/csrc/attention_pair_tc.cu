// Causal grouped-query attention of long prompts on the fifth-generation tensor cores (bfloat16, head size 128), two tiles
// of query rows per CTA.
//
// A CTA owns two tiles of up to 128 query rows of one KV head, each the G query heads of the group for floor(128 / G)
// consecutive tokens of one sequence, the second tile's tokens right behind the first one's.  Keys are visited 128 at a time
// (two pages, TMA boxes of 64 rows x 64 dims, 128-byte swizzle); a tile of keys and values serves both.  For key tile j and
// query tile x:
//
//   MMA warp            S_x = Q_x K_j^T   (M 128, N 128, K = head size)         -> TMEM
//   softmax warps of x  S_x from TMEM (a row per thread), scale, mask, maximum and sum, P_x = 2^(s - m) in bfloat16 -> TMEM,
//                       over the first half of S_x
//   MMA warp            O_x += P_x V_j    (M 128, N = head size, K 128)         -> TMEM, then S_x of tile j + 1
//
// The softmax of one query tile runs while the tensor cores work for the other.  Everything else is as in attention_tc.cu
// (lazy reference m, P read from TMEM, bounded waits); that kernel has 64 keys per tile, two buffers of S and two CTAs per SM.
// That one's MMAs of 64 columns cost more than half of those of 128, and its chain of products and softmax is met more often:
// 8,192 tokens, 32 heads on 8, 614 -> 507 us (1.09 PFLOP/s), on 32 666 -> 525; 1,000 tokens on 3,000 held ones 89 -> 75.  Bound by
// the softmax warps (two per scheduler), whose exponentials alone are half of the time.  Head size 64 has half the MMAs for the
// same softmax and lost (397 -> 443 us), as did two threads per row (576 us).
#include "attention_tc.cuh"
#include "common.cuh"
#include "launch.cuh"

#define AP_ROWS 128
#define AP_PAGE 64
#define AP_KEYS 128
#define AP_THREADS 320      // TMA, MMA, four softmax warps per query tile

// Panels of [128 rows][64 dims] = 128-byte rows, 1024-byte aligned: the query tiles', then STAGES of keys and values.  TMEM: S
// at columns 0 and 128, O from 256; one CTA per SM.
template <int HD> struct ApShape {
  static constexpr int PANELS = HD / 64;
  static constexpr int STAGES = 2;
  static constexpr int PANEL = 128 * 128;
  static constexpr int TILE = PANELS * PANEL;
  static constexpr int KV_OFF = 2 * TILE;
  static constexpr int BAR_OFF = KV_OFF + STAGES * 2 * TILE;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

template <int HD>
__global__ void __launch_bounds__(AP_THREADS, 1)
attention_pair_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, bf16* __restrict__ out, const int* __restrict__ block_table,
                         int table_width, const int* __restrict__ tok_pos, const int* __restrict__ cu_q,
                         const int* __restrict__ tile_seq, const int* __restrict__ tile_q0, int H, int K, float scale_log2,
                         int window, int tokens_per_tile, int* __restrict__ status, const float* __restrict__ sink) {
  using Sh = ApShape<HD>;
  constexpr int STAGES = Sh::STAGES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* q_full = reinterpret_cast<uint64_t*>(base + Sh::BAR_OFF);      // 1
  uint64_t* kv_full = q_full + 1;                // STAGES
  uint64_t* kv_empty = kv_full + STAGES;         // STAGES
  uint64_t* s_full = kv_empty + STAGES;          // a query tile each: completes once per key tile, as the next two do
  uint64_t* p_full = s_full + 2;
  uint64_t* o_done = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = H / K;
  const int tile = blockIdx.x / K, kh = blockIdx.x - tile * K;
  if (threadIdx.x == 0) {
    at_bar_init(q_full, 1);
    for (int s = 0; s < STAGES; ++s) { at_bar_init(kv_full + s, 1); at_bar_init(kv_empty + s, 1); }
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
  pdl_wait();
  pdl_trigger();

  const int b = tile_seq[tile], q0 = tile_q0[tile];
  const int n_tok = min(2 * tokens_per_tile, cu_q[b + 1] - q0);
  const int pos_first = tok_pos[q0], pos_last = tok_pos[q0 + n_tok - 1];
  const int page_begin = (window > 0 && pos_first - window + 1 > 0) ? (pos_first - window + 1) / AP_PAGE : 0;
  const int page_end = pos_last / AP_PAGE + 1;
  const int n_tiles = (page_end - page_begin + 1) / 2;
  const int* bt = block_table + (size_t)b * table_width;

  if (warp == 0) {
    if (lane == 0) {
      // a box holds tokens_per_tile x G rows (all counted, also where they lie past the step's end and become zeros); a second
      // tile that lies past it altogether is all zeros
      at_expect_tx(q_full, 2 * Sh::PANELS * tokens_per_tile * G * 128);
      for (int x = 0; x < 2; ++x)
        for (int p = 0; p < Sh::PANELS; ++p)
          at_tma_3d(base + x * Sh::TILE + p * Sh::PANEL, &map_q, p * 64, kh * G, q0 + x * tokens_per_tile, q_full);
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % STAGES;
        if (j >= STAGES && !at_wait(kv_empty + s, ((j / STAGES) - 1) & 1)) { atomicExch(status, 31); break; }
        const int i0 = page_begin + 2 * j, i1 = min(i0 + 1, page_end - 1);      // an odd last page stands twice; its copy is masked
        const int r0 = (bt[i0] * K + kh) * AP_PAGE, r1 = (bt[i1] * K + kh) * AP_PAGE;
        unsigned char* dst = base + Sh::KV_OFF + s * 2 * Sh::TILE;
        at_expect_tx(kv_full + s, 2 * Sh::TILE);
        for (int p = 0; p < Sh::PANELS; ++p) {
          at_tma_2d(dst + p * Sh::PANEL, &map_k, p * 64, r0, kv_full + s);
          at_tma_2d(dst + p * Sh::PANEL + AP_PAGE * 128, &map_k, p * 64, r1, kv_full + s);
          at_tma_2d(dst + Sh::TILE + p * Sh::PANEL, &map_v, p * 64, r0, kv_full + s);
          at_tma_2d(dst + Sh::TILE + p * Sh::PANEL + AP_PAGE * 128, &map_v, p * 64, r1, kv_full + s);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // S = Q K^T: both operands K-major, N = 128;  O += P V: P from TMEM, V [key][dim] = MN-major, N = head size
      constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AP_KEYS >> 3) << 17) |
                                   ((uint32_t)(AP_ROWS >> 4) << 24);
      constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) |
                                   ((uint32_t)(AP_ROWS >> 4) << 24);
      bool ok = at_wait(q_full, 0);
      if (!ok) atomicExch(status, 32);
      auto keys = [&](int j) {
        if (!at_wait(kv_full + j % STAGES, (j / STAGES) & 1)) { atomicExch(status, 33); ok = false; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      };
      auto issue_s = [&](int j, int x) {
        const uint32_t q_addr = at_smem(base + x * Sh::TILE);
        const uint32_t k_addr = at_smem(base + Sh::KV_OFF + j % STAGES * 2 * Sh::TILE);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k)      // 16 dims per MMA: 32 bytes along a panel's rows
          at_mma(tmem + x * 128, at_desc(q_addr + (k >> 2) * Sh::PANEL + (k & 3) * 32),
                 at_desc(k_addr + (k >> 2) * Sh::PANEL + (k & 3) * 32), idesc_s, k > 0 ? 1u : 0u);
        at_commit(s_full + x);
      };
      if (ok) keys(0);
      if (ok) { issue_s(0, 0); issue_s(0, 1); }
      for (int j = 0; j < n_tiles && ok; ++j) {
        const uint32_t v_addr = at_smem(base + Sh::KV_OFF + j % STAGES * 2 * Sh::TILE + Sh::TILE);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          if (!ok) break;
          if (!at_wait(p_full + x, j & 1)) { atomicExch(status, 34); ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int k = 0; k < AP_KEYS / 16; ++k)     // 16 keys per MMA: 8 columns of P, 2 groups of 8 rows of V
            at_mma_ts(tmem + 256 + x * HD, tmem + x * 128 + k * 8, at_desc_mn(v_addr + k * 2048, Sh::PANEL), idesc_o,
                      (j > 0 || k > 0) ? 1u : 0u);
          at_commit(o_done + x);
          if (x == 1) at_commit(kv_empty + j % STAGES);
          if (j + 1 < n_tiles) {
            if (x == 0) keys(j + 1);
            if (ok) issue_s(j + 1, x);      // over P_x, behind the product that reads it
          }
        }
      }
    }
  } else {
    // softmax warps: TMEM lanes 32 * (warp % 4) ..; thread = query row of tile x
    const int x = warp >= 6 ? 1 : 0, quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_col = tmem + lane_base + x * 128, o_col = tmem + lane_base + 256 + x * HD;
    const int t0 = q0 + x * tokens_per_tile;                 // this tile's first token
    const int t = t0 + r / G;
    const bool row_ok = r < tokens_per_tile * G && t < q0 + n_tok;
    int pos = 0x3fffffff, lo = 0;
    if (row_ok) {
      pos = tok_pos[t];
      lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    }
    const int mask_from = pos_first + x * tokens_per_tile;   // keys up to here are seen by all of the tile's rows
    float m_ref = -INFINITY, l_run = 0.f;       // the row's reference and its sum of 2^(s - m_ref)
    bool ok = true;
    for (int j = 0; j < n_tiles && ok; ++j) {
      if (!at_wait(s_full + x, j & 1)) { atomicExch(status, 36); ok = false; }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float sc[AP_KEYS];
#pragma unroll
      for (int c0 = 0; c0 < AP_KEYS; c0 += 16) at_ld16(s_col + c0, sc + c0);
      at_ld_wait();
      const int key0 = (page_begin + 2 * j) * AP_PAGE;
      if (key0 + AP_KEYS - 1 > mask_from || window > 0) {
#pragma unroll
        for (int c = 0; c < AP_KEYS; ++c)
          if (key0 + c > pos || key0 + c < lo) sc[c] = -INFINITY;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < AP_KEYS; c += 4) {
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
      for (int c0 = 0; c0 < AP_KEYS; c0 += 32) {
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
        if (!at_wait(o_done + x, (j - 1) & 1)) { atomicExch(status, 35); ok = false; }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c0 = 0; c0 < HD; c0 += 16) {
          float o[16];
          at_ld16(o_col + c0, o);
          at_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c) o[c] *= corr;
          at_st16(o_col + c0, o);
        }
      }
      at_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      at_arrive(p_full + x);
    }
    if (ok) {
      if (!at_wait(o_done + x, (n_tiles - 1) & 1)) { atomicExch(status, 37); ok = false; }
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // a sink: a learned logit per head whose exp joins the denominator and which has no value
      if (sink != nullptr && row_ok && m_ref > -INFINITY) l_run += exp2f(sink[kh * G + r % G] * AT_LOG2E - m_ref);
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      bf16* dst = out + ((size_t)t * H + kh * G + r % G) * HD;
#pragma unroll
      for (int c0 = 0; c0 < HD; c0 += 16) {
        float o[16];
        at_ld16(o_col + c0, o);
        at_ld_wait();
        if (row_ok) {
          uint32_t w[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            __nv_bfloat162 pr = __floats2bfloat162_rn(o[2 * e] * inv, o[2 * e + 1] * inv);
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

static int* ap_status_word() {
  static int* p[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!p[dev]) {
    if (cudaMalloc(&p[dev], sizeof(int)) != cudaSuccess) return nullptr;
    cudaMemset(p[dev], 0, sizeof(int));
  }
  return p[dev];
}
AB_API int ab_attention_pair_tc_status() {
  int* p = ap_status_word();
  if (!p) return -1;
  int v = 0;
  if (cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (v) cudaMemset(p, 0, sizeof(int));
  return v;
}

// Arguments as ab_attention_prefill_tc_dist's without a change of the scores; tile_seq / tile_q0: tiles of 2 * floor(128 / G) tokens (sequence, first packed
// token).  out 16-byte aligned.
AB_API int ab_attention_pair_tc(const void* qkv, int row_heads, int n_tokens, void* out, const void* k_pages,
                                const void* v_pages, int n_pages, const int* block_table, int table_width, const int* tok_pos,
                                const int* cu_q, const int* tile_seq, const int* tile_q0, int n_tiles, int H, int K, int D,
                                float scale, int window, const float* sink, cudaStream_t stream) {
  if (n_tiles <= 0) return AB_OK;
  if (D != 128 || K <= 0 || H % K || H / K > AP_ROWS || (long long)n_tiles * K > 0x7fffffffLL || row_heads < H ||
      ((uintptr_t)out & 15))
    return AB_BAD_ARG;
  AtEncodeFn enc = at_encode_fn();
  int* status = ap_status_word();
  if (!enc || !status) return AB_BAD_ARG;
  const int G = H / K, tpt = AP_ROWS / G;
  CUtensorMap mq, mk, mv;
  {
    cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)row_heads, (cuuint64_t)n_tokens};
    cuuint64_t strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)row_heads * D * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)tpt};          // one panel: 64 elements of the head
    cuuint32_t elem[3] = {1, 1, 1};
    if (enc(&mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(qkv), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return AB_BAD_ARG;
  }
  for (int which = 0; which < 2; ++which) {
    cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)n_pages * K * AP_PAGE};
    cuuint64_t strides[1] = {(cuuint64_t)D * 2};
    cuuint32_t box[2] = {64, AP_PAGE};
    cuuint32_t elem[2] = {1, 1};
    if (enc(which ? &mv : &mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(which ? v_pages : k_pages), dims,
            strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return AB_BAD_ARG;
  }
  cudaError_t e = cudaFuncSetAttribute(attention_pair_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ApShape<128>::TOTAL);
  if (e != cudaSuccess) return AB_CUDA_ERR + (int)e;
  e = ab_launch(attention_pair_tc_kernel<128>, dim3((unsigned)n_tiles * K), dim3(AP_THREADS), ApShape<128>::TOTAL, stream, mq,
                mk, mv, (bf16*)out, block_table, table_width, tok_pos, cu_q, tile_seq, tile_q0, H, K, scale * AT_LOG2E, window,
                tpt, status, sink);
  if (e != cudaSuccess) return AB_CUDA_ERR + (int)e;
  return ab_launch_status();
}
