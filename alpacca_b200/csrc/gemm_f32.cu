// C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]) with the precision of 32-bit sums, on the tensor cores.
//
// Every 32-bit number is split into three bfloat16 numbers that add up to it exactly (x = h + m + l: h is x rounded,
// m the rest rounded, l what is then left, at most eight bits).  A product needs six of the nine partial products,
//   a w = ah wh + (ah wm + am wh) + (ah wl + am wm + al wh)
// each exact in 32 bits.  (|m| is up to 2^-8 |x|, |l| up to 2^-17 |x|, so the other three are up to about 2^-24 of |a w|, of
// either sign.)  They are summed by tcgen05.mma in three 32-bit accumulators in tensor memory, one per bracket.  The sums
// of the tensor cores cut off instead of rounding, so the leading accumulator holds 32 k only: adding warps then add it to
// a rounded 32-bit sum in registers.  The two others are 2^-8 smaller and run to the end of a run of k.
// Error against 64 bits, root mean square over |a| |w| (before: multiply-adds in 32 bits): normal numbers 2.0e-9 at 2,048 k
// (4.7e-9), 1.4e-9 at 8,192 (4.5e-9), 5.5e-9 at 128 (1.3e-8), 7.4e-9 at 48 (1.4e-8); all of one sign 3.8e-8 at 2,048
// (4.3e-8), 3.5e-8 at 48 (3.9e-8).  A layer of the 1B shape 2.5e-7 (5.4e-7).  Below 48 k the roundings weigh more than those
// of multiply-adds, which are taken there (`gemm_f32_short_kernel`).
//
// The order of an output's sum depends on K alone: the k range is cut into up to GROUPS runs (of a multiple of BK, at
// least SHORTEST), a run into stages of 32; the first four runs are added in ascending order, the others too, then both.
// So a value does not depend on M, on the tile it falls into, on whether the runs of a tile are computed by one CTA or by
// a cluster of CTAs, or on what other rows are in the batch: the same token gives the same bits alone and in any batch.
// This is the matrix product of the 32-bit path (the reference's float32 path uses BLAS SGEMM, alpacca/tensor.py:91-97).
//
// The parts are those of 2^16 times a number, so that the smallest number's last bit is one of a bfloat16 too, and outputs
// are multiplied by 2^-32: powers of two, which change no other bit.  A number of 2^112 or more splits into infinities and
// NaNs, an output of 2^96 or more overflows.  An output that comes out not finite is therefore formed again by plain
// multiply-adds (`plain_rows`): what the sum gives in 32 bits, infinities included.
//
// A tile is 128 rows of W (the 128 rows of an MMA) by n <= 128 rows of A.  Splitting warps bring both operands' 32-bit rows
// by cp.async into a ring in shared memory (each thread only what it splits itself, so nobody waits for anybody), split
// them and store the parts in the swizzled form that the MMA reads; adding warps move the leading accumulator; one lane of
// another warp issues the MMAs, four per 16 k: [wm|wl] and [wh|wm] lie side by side, so that two MMAs do the work of four.
// What bounds it: for many rows the splitting and adding instructions (some 1,400 clocks a stage at n = 128, the tensor
// cores 768); for few rows the latency of a stage, hidden by two CTAs per processor, and HBM.
// us multiply-adds on the FMA pipes (before) / this: 333 rows of q|k|v, o, gate|up and down of the 1B shape 123 / 45, 87 / 45,
// 571 / 266, 315 / 145; 64 rows 34 / 25, 24 / 24, 114 / 63, 81 / 61; 17 rows 22 / 16, 15 / 15, 67 / 49, 50 / 43; one row
// 11.6 / 12.3, 11.0 / 11.2, 35.9 / 33.6, 35.5 / 30.5.  2,048 rows of 16384x2048: 2,960 / 1,314 (105 TFLOP/s, 46 before).
// Its chain of steps (copy, split, multiply, add, store) is longer than that of multiply-adds: few rows of small matrices
// take 0.5 to 1.8 us more (one row of 2048x128 3.8 / 5.6, of 512x1024 4.7 / 6.2; 333 rows of 2048x128 11.9 / 8.4).
// Tried: 16 warps that split and add in turn (333 rows of gate|up 243, one row of q|k|v 15.8); rounding in integers in place
// of the conversion instruction (the same); two leading accumulators (one row 0.8 us slower a product), four of them where a
// CTA has four stages (one row of 2048x128 0.2 us faster, 333 rows of 16384x128 1 us slower).
//
// Every wait on an mbarrier is bounded; a thread that gives up leaves a code in `gemm_f32_stuck`, all roles fall through
// to the end, where TMEM is given back, and the outputs are NaN until `plain_rows` has formed them.
#include "attention_tc.cuh"
#include "common.cuh"
#include "launch.cuh"

#define BK 32            // k of a stage: 64 bytes of a split row, the width of the swizzle
#define GROUPS 8         // runs of k; also the CTAs of a cluster that share a tile
#define SHORTEST 128     // a run's k at least
#define EARLY 256        // k of W that are fetched to the L2 before the kernel before this one has ended
#define W_PART (128 * 64)          // bytes of one part of the weights' rows in a stage

__device__ int gemm_f32_stuck;     // 0, or the code of a wait that was given up

__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
// A product of K-major operand rows of 64 bytes with the 64-byte swizzle (groups of 8 rows are 512 bytes apart), by the
// lower words of their descriptors: the upper ones are the same, and one thread issues all of them, so every
// instruction around them counts.
#define SPLIT_DESC_LO(addr) (((addr) >> 4) | (1u << 16))
__device__ __forceinline__ void split_mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 x, y;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 x, {%1, %5};\n\tmov.b64 y, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, p;\n\t}"
      ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"((uint32_t)accumulate), "r"(32u | (1u << 14) | (4u << 29)) : "memory");
}
__device__ __forceinline__ void lds16(uint32_t a, uint32_t* x) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t a, const uint32_t* x) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]) : "memory");
}
__device__ __forceinline__ void ld8(uint32_t taddr, float2* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
__device__ __forceinline__ void add8(float2* a, const float2* v) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\t"
        "mov.b64 {%0, %1}, x;\n\t}" : "+f"(a[i].x), "+f"(a[i].y) : "f"(v[i].x), "f"(v[i].y));
}
__device__ __forceinline__ void fma2(float2& s, float ax, float ay, float bx, float by) {      // s += (ax bx, ay by)
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%0, %1};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}" : "+f"(s.x), "+f"(s.y) : "f"(ax), "f"(ay), "f"(bx), "f"(by));
}
__device__ __forceinline__ void st8(uint32_t taddr, const float2* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(__float_as_uint(v[0].x)),
               "r"(__float_as_uint(v[0].y)), "r"(__float_as_uint(v[1].x)), "r"(__float_as_uint(v[1].y)),
               "r"(__float_as_uint(v[2].x)), "r"(__float_as_uint(v[2].y)), "r"(__float_as_uint(v[3].x)),
               "r"(__float_as_uint(v[3].y)) : "memory");
}
__device__ __forceinline__ void less(uint32_t& a, uint32_t& b, uint32_t pa, uint32_t pb) {      // (a, b) -= (pa, pb), exact
  asm("{\n\t.reg .b64 x, p;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 p, {%2, %3};\n\t"
      "fma.rn.f32x2 x, p, %4, x;\n\tmov.b64 {%0, %1}, x;\n\t}" : "+r"(a), "+r"(b) : "r"(pa), "r"(pb), "l"(0xbf800000bf800000ull));
}
// Two numbers (their bits) to two words of parts of 2^16 times them, the first in the lower half.  Rounded, so that the rest
// has either sign and the three products left out cancel; what is left for l is at most eight bits.  Below 2^-110 a number's
// last bits would lie under 2^-133, the last bit of bfloat16: times 2^16 the smallest number's last bit lies on it.
#define SCALE_BITS 0x4780000047800000ull      // 2^16, twice
#define UNSCALE 0x1p-32f                      // what a product is multiplied by in the end
__device__ __forceinline__ void split2(uint32_t a, uint32_t b, uint32_t& h, uint32_t& m, uint32_t& l) {
  asm("{\n\t.reg .b64 x;\n\tmov.b64 x, {%0, %1};\n\tmul.rn.f32x2 x, x, %2;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+r"(a), "+r"(b) : "l"(SCALE_BITS));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(__uint_as_float(b)), "f"(__uint_as_float(a)));
  less(a, b, h << 16, h & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(m) : "f"(__uint_as_float(b)), "f"(__uint_as_float(a)));
  less(a, b, m << 16, m & 0xffff0000u);
  l = __byte_perm(a, b, 0x7632);
}

// the product's last step: z (bias included), or with inv_tau > 0 a decay, sigmoid(z)^inv_tau
__device__ __forceinline__ float finish(float z, float inv_tau) {
  if (inv_tau <= 0.f) return z;
  const float sp = -z > 20.f ? -z : log1pf(expf(-z));      // -log sigmoid(z)
  return expf(-sp * inv_tau);
}
__device__ __forceinline__ bool is_finite(float z) { return (__float_as_uint(z) & 0x7f800000u) != 0x7f800000u; }

// Outputs that the split numbers cannot form, those marked by a number that is not finite in `part` ([n][128], rows of A by
// rows of W), by plain multiply-adds: rows row .. row_end of A from `a`, the `cols` rows of W from `w`, the runs of k in
// ascending order.  T threads (a thread has a column and FALL rows at a time), 32 k after the other by cp.async into `room`.
// A function of its own with few rows a thread: inlined, or with eight rows, it took registers from the loops before it
// (333 rows of 16384x2048 without such outputs 267 -> 272 us).  us with a thread per output that reads both rows from global
// memory / this / the multiply-adds of before: one row of 16384x2048 with a NaN 321 / 115 / 38, one such row of 333
// 516 / 354 / 572, all of 48 11,500 / 426 / 119, all of 333 47,000 / 2,630 / 574; a row of W with a NaN 819 / 444 / 572, of
// 2048x8192 (half the runs in a CTA: every row of the tile again) 726 / 1,155 / 315.
#define FALL 4
#define FALL_BUFFERS 4
template <int T> struct Fall {
  static constexpr int PASS = T / 128 * FALL;                       // rows at a time
  static constexpr int KP = BK + 4;                                 // eight neighbouring threads' 16 bytes meet every bank once
  static constexpr int BUFFER = (128 + PASS) * KP;                  // floats
};
template <int T, bool VEC>
__device__ __noinline__ void plain_rows(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw,
                                           const float* __restrict__ bias, float* __restrict__ c, int ldc, int row, int row_end,
                                           int cols, int K, int run, float inv_tau, const float* part, float* room) {
  using F = Fall<T>;
  const int col = threadIdx.x & 127, first = (threadIdx.x >> 7) * FALL;
#pragma unroll 1
  for (; row < row_end; row += F::PASS) {
    uint32_t bad = 0;
#pragma unroll
    for (int i = 0; i < FALL; ++i)
      if (first < F::PASS && row + first + i < row_end && col < cols && !is_finite(part[(row + first + i) * 128 + col])) bad |= 1u << i;
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.or.pred p, 1, %2, q;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(any) : "r"(bad), "n"(T) : "memory");
    if (!any) continue;
    auto stage = [&](int t) {                      // 32 k from t * BK on, an empty group past the end
      if (t * BK < K) {
        float* to = room + t % FALL_BUFFERS * F::BUFFER;
        constexpr int E = VEC ? 4 : 1;
#pragma unroll 1
        for (int i = threadIdx.x; i < (128 + F::PASS) * (BK / E); i += T) {
          const int r = i / (BK / E), k = t * BK + i % (BK / E) * E;
          const bool in = k < K && (r < 128 ? r < cols : row + r - 128 < row_end);
          const float* from = !in ? a : (r < 128 ? w + (size_t)r * ldw : a + (size_t)(row + r - 128) * lda) + k;
          const uint32_t at = at_smem(to + r * F::KP + i % (BK / E) * E);
          if (VEC) cp_async16(at, from, in ? 16 : 0);
          else cp_async4(at, from, in ? 4 : 0);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float sum[FALL], tot[FALL];
#pragma unroll
    for (int i = 0; i < FALL; ++i) sum[i] = tot[i] = 0.f;
#pragma unroll 1
    for (int t = 0; t < FALL_BUFFERS - 1; ++t) stage(t);
#pragma unroll 1
    for (int t = 0, k0 = 0; k0 < K; ++t, k0 += BK) {
      asm volatile("cp.async.wait_group %0;" ::"n"(FALL_BUFFERS - 2) : "memory");
      asm volatile("barrier.cta.sync 1, %0;" ::"n"(T) : "memory");      // these k are there for all, those before are read by all
      stage(t + FALL_BUFFERS - 1);
      if (__any_sync(0xffffffffu, bad)) {
        const float* from = room + t % FALL_BUFFERS * F::BUFFER;
#pragma unroll 2
        for (int k = 0; k < BK; k += 4) {
          const float4 y = *reinterpret_cast<const float4*>(from + col * F::KP + k);
#pragma unroll
          for (int i = 0; i < FALL; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(from + (128 + first + i) * F::KP + k);
            sum[i] = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, sum[i]))));
          }
        }
        if ((k0 + BK) % run == 0 || k0 + BK >= K) {
#pragma unroll
          for (int i = 0; i < FALL; ++i) {
            tot[i] = k0 < run ? sum[i] : tot[i] + sum[i];
            sum[i] = 0.f;
          }
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("barrier.cta.sync 1, %0;" ::"n"(T) : "memory");        // the buffers may be filled again
#pragma unroll
    for (int i = 0; i < FALL; ++i)
      if (bad >> i & 1) c[(size_t)(row + first + i) * ldc + col] = finish(tot[i] + (bias ? bias[col] : 0.f), inv_tau);
  }
}

// NT: the most rows of A that a tile can hold; `n` of them are this launch's (a multiple of 16).
template <int NT> struct F32Shape {
  static constexpr int SPLITTERS = NT >= 64 ? 12 : NT >= 32 ? 10 : 9;      // warps that split, ..
  static constexpr int ADDERS = NT >= 64 ? 8 : 4;                   // that add up, and the one that issues the MMAs
  static constexpr bool UNEQUAL = NT > 64;                          // registers by role (a warpgroup for the MMAs then)
  static constexpr int WARPS = SPLITTERS + ADDERS;
  static constexpr int THREADS = 32 * (WARPS + (UNEQUAL ? 4 : 1));
  static constexpr int BLOCKS = NT / (2 * ADDERS);                  // blocks of 8 columns that a warp adds up
  static constexpr int ROWS = 128 + NT;                             // of W, then of A
  static constexpr int PASS = 8 * SPLITTERS;                        // rows that the splitting threads take at a time
  static constexpr int PASSES = (ROWS + PASS - 1) / PASS;
  static constexpr int LAST = ROWS - (PASSES - 1) * PASS;           // rows of the last pass
  static constexpr int SLOTS = NT == 64 ? 3 : 2;     // stages of split rows
  static constexpr int RAW = NT == 32 ? 2 : NT == 64 ? 4 : 3;          // stages of 32-bit rows in flight
  static constexpr int RAW_STAGE = ROWS * 128;
  static constexpr int SPLIT_STAGE = 3 * ROWS * 64;
  static constexpr int BAR_OFF = RAW * RAW_STAGE + SLOTS * SPLIT_STAGE;
  static constexpr int SMEM = BAR_OFF + 128 + 1024 /*alignment*/;
  static constexpr int CTAS = NT <= 32 ? 2 : 1;                     // per processor
  static constexpr int TMEM_COLS = NT <= 16 ? 128 : NT <= 32 ? 256 : 512;      // four times n of them used, or five times
  static_assert(BAR_OFF >= 128 * NT * 4 + FALL_BUFFERS * Fall<32 * WARPS>::BUFFER * 4, "the partial sums take the tiles' place");
  static_assert(!UNEQUAL || (THREADS * 80 == 128 * 40 + 32 * SPLITTERS * 72 + 32 * ADDERS * 112), "registers by role");
  static_assert(CTAS * (SMEM + 1024) <= 233472, "what a CTA may have");
};

// PER: the runs of a CTA: all of them, half of GROUPS or one.  `cs` CTAs then share a tile as a cluster, and each adds up
// its part of the tile through distributed shared memory.  VEC: both operands' rows can be copied 16 bytes at a time.
template <int NT, bool VEC, int PER>
__global__ void __launch_bounds__(F32Shape<NT>::THREADS, F32Shape<NT>::CTAS)
gemm_f32_nt_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                   const float* __restrict__ bias, float* __restrict__ C, int ldc, int M, int N, int K, int run,
                   float inv_tau, int n, int cs) {
  using S = F32Shape<NT>;
  constexpr int BLOCKS = S::BLOCKS, RAW = S::RAW, SLOTS = S::SLOTS, PASSES = S::PASSES, STEP = S::ADDERS / 4;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* split_base = base;              // [SLOTS][wh | wm | wl | ah | am | al], rows of 64 bytes
  unsigned char* raw_base = base + SLOTS * S::SPLIT_STAGE;
  uint64_t* full = reinterpret_cast<uint64_t*>(base + S::BAR_OFF);      // SLOTS: a stage is stored
  uint64_t* done = full + SLOTS;                 // SLOTS: a stage is multiplied
  uint64_t* lead_read = done + SLOTS;            // a stage's leading sums have been read
  uint64_t* rest_read = lead_read + 1;           // a run's other sums have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rest_read + 1);
  volatile uint32_t* marked = tmem_slot + 1;     // whether this CTA's part of the outputs has some to be formed again

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr bool ALONE = PER == GROUPS;
  const int rank = ALONE ? 0 : (int)(blockIdx.x % (unsigned)cs);      // the cluster lies along x
  const int share_k = run * PER;
  const int m0 = blockIdx.y * n, n0 = (ALONE ? blockIdx.x : blockIdx.x / (unsigned)cs) * 128;
  const int kbegin = min(K, rank * share_k), kend = min(K, kbegin + share_k);
  const int tiles = (kend - kbegin + BK - 1) / BK, per_run = run / BK;

  // W's first stages on their way to the L2 while the kernel before this one ends: a hint, which reads nothing that it writes
  if (warp < S::SPLITTERS && n <= 64) {
    for (int x = threadIdx.x >> 2; x < 128 && n0 + x < N; x += S::PASS)
      for (int k = kbegin + (threadIdx.x & 3) * 32; k < min(kend, kbegin + EARLY); k += 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (size_t)(n0 + x) * ldw + k));
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < SLOTS; ++i) { at_bar_init(full + i, S::SPLITTERS); at_bar_init(done + i, 1); }
    at_bar_init(lead_read, S::ADDERS);
    at_bar_init(rest_read, S::ADDERS);
    *marked = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == S::WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(tmem_slot)), "r"(S::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;              // columns: n of a stage's leading sums, 2n of a run's others, n or 2n of runs
  pdl_wait();
  pdl_trigger();

  bool ok = true;
  // an adding warp's columns (rows of A): blocks first, first + STEP, ..
  const int first = STEP == 2 ? (warp >> 2) & 1 : 0, blocks = n / 8;
  // In the end every warp has the registers of the launch again, the others behind this barrier only: the adding warps have
  // then taken and given back theirs (warps that took theirs back before would leave too few for them, and all would wait).
  auto roles_end = [] { asm volatile("barrier.cta.sync 2, %0;" ::"n"(S::THREADS) : "memory"); };
  float* part = reinterpret_cast<float*>(base);  // [n][128]: the sums, once nothing reads or writes the stages any more
  if (warp >= S::WARPS) {
    if (S::UNEQUAL) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == S::WARPS && lane == 0) {
      constexpr uint32_t kind = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);
      const uint32_t one = kind | ((uint32_t)(n >> 3) << 17), two = kind | ((uint32_t)(n >> 2) << 17);
      const uint32_t rest = tmem + n, part = (uint32_t)n * 4, lo = SPLIT_DESC_LO(at_smem(split_base));
      int in_run = 0, s = 0;
      uint32_t phase = 0, run_phase = 1;
      for (int t = 0; t < tiles; ++t) {
        if (!at_wait(full + s, phase)) { ok = false; break; }
        if (in_run == 0 && t > 0 && !at_wait(rest_read, run_phase)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t w = lo + s * (S::SPLIT_STAGE >> 4), a = w + (3 * W_PART >> 4);
        constexpr uint32_t wpart = W_PART >> 4;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          split_mma(rest, w + 2 * k, a + part + 2 * k, two, in_run > 0 || k > 0);      // wh am | wh al
          split_mma(rest, w + wpart + 2 * k, a + 2 * k, two, true);                    // wm ah | wm am
          split_mma(rest + n, w + 2 * wpart + 2 * k, a + 2 * k, one, true);            // wl ah
        }
        // The leading products last: meanwhile the sums of the stage before have been read
        if (t > 0 && !at_wait(lead_read, (t - 1) & 1)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) split_mma(tmem, w + 2 * k, a + 2 * k, one, k > 0);
        at_commit(done + s);
        if (++in_run == per_run) { in_run = 0; run_phase ^= 1; }
        if (++s == SLOTS) { s = 0; phase ^= 1; }
      }
      if (!ok) atomicExch(&gemm_f32_stuck, 41);
    }
    if (S::UNEQUAL) {
      __syncwarp();
      roles_end();
      asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
    }
  } else if (warp < S::SPLITTERS) {
    if (S::UNEQUAL) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    // Thread q of a row's four takes the 16-byte pieces q and q + 4 of its 32 numbers (a warp's copy then reads whole
    // sectors) and stores their parts as the row's 16-byte piece q: both operands' k are permuted the same way.
    // Rows past A's end keep whatever is there, rows past W's end read its last one: their outputs are not stored.  (All
    // sixteen rows of a tile reading one row of A cost a single row of 16384x2048 4 us: every CTA asks for the same lines.)
    const int q = threadIdx.x & 3, row = threadIdx.x >> 2;
    const float* src[PASSES];
    bool mine[PASSES];
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
      const int x = row + S::PASS * p;
      mine[p] = x < 128 + min(n, M - m0);
      src[p] = (x < 128 ? W + (size_t)min(n0 + x, N - 1) * ldw : A + (size_t)(mine[p] ? m0 + x - 128 : 0) * lda) + kbegin + q * 4;
    }
    const uint32_t raw = at_smem(raw_base) + threadIdx.x * 16;
    constexpr int PIECES = S::PASS * 64, LAST_PIECES = S::LAST * 64;      // bytes of a pass's first pieces
    int left = kend - kbegin - q * 4;              // k from this thread's first piece of the next stage to the end
    uint32_t slot = raw;
    auto fetch = [&]() {                           // the next stage into the next slot
      if (VEC && left >= 20) {
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
          if (S::PASS * (p + 1) > 128 && !mine[p]) continue;
          cp_async16(slot + p * 2 * PIECES, src[p], 16);
          cp_async16(slot + p * 2 * PIECES + (p < PASSES - 1 ? PIECES : LAST_PIECES), src[p] + 16, 16);
        }
      } else if (left > -q * 4) {
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
          if (!mine[p]) continue;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int e = 0; e < 4; e += VEC ? 4 : 1) {
              const bool in = h * 16 + e < left;
              const float* from = in ? src[p] + h * 16 + e : A;
              const uint32_t to = slot + p * 2 * PIECES + h * (p < PASSES - 1 ? PIECES : LAST_PIECES) + 4 * e;
              if (VEC) cp_async16(to, from, in ? 16 : 0);
              else cp_async4(to, from, in ? 4 : 0);
            }
          }
        }
      }
      left -= BK;
#pragma unroll
      for (int p = 0; p < PASSES; ++p) src[p] += BK;
      slot = slot == raw + (RAW - 1) * S::RAW_STAGE ? raw : slot + S::RAW_STAGE;
      asm volatile("cp.async.commit_group;" ::: "memory");       // an empty group past the end keeps the count
    };
#pragma unroll 1
    for (int t = 0; t < RAW; ++t) fetch();
    const uint32_t to = at_smem(split_base) + ((q ^ ((row >> 1) & 3)) << 4);
    int s = 0;
    uint32_t phase = 1;
#pragma unroll 1
    for (int t = 0; t < tiles; ++t) {
      asm volatile("cp.async.wait_group %0;" ::"n"(RAW - 1) : "memory");
      if (t >= SLOTS && !at_wait(done + s, phase)) ok = false;
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      uint32_t x[PASSES][8];
#pragma unroll
      for (int p = 0; p < PASSES; ++p) {
        if (S::PASS * (p + 1) > 128 && !mine[p]) continue;
        lds16(slot + p * 2 * PIECES, x[p]);
        lds16(slot + p * 2 * PIECES + (p < PASSES - 1 ? PIECES : LAST_PIECES), x[p] + 4);
      }
#pragma unroll
      for (int p = 0; p < PASSES; ++p) {
        if (S::PASS * (p + 1) > 128 && !mine[p]) continue;
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split2(x[p][2 * e], x[p][2 * e + 1], h[e], m[e], l[e]);
        const int x = row + S::PASS * p;           // (PASS is a multiple of 8: the swizzle is the same in all passes)
        const bool a = S::PASS * (p + 1) > 128 && x >= 128;
        const uint32_t o = to + s * S::SPLIT_STAGE + x * 64 + (a ? 2 * W_PART : 0), part = a ? (uint32_t)n * 64 : W_PART;
        sts16(o, h);
        sts16(o + part, m);
        sts16(o + 2 * part, l);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) at_arrive(full + s);
      fetch();                                     // into the pieces that this thread has just read
      if (++s == SLOTS) { s = 0; phase ^= 1; }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!ok && lane == 0) atomicExch(&gemm_f32_stuck, 42);
    if (S::UNEQUAL) {
      __syncwarp();
      roles_end();
      asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
    }
  } else {
    if (S::UNEQUAL) asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + first * 8;     // its lanes of TMEM: rows of W
    float2 acc[BLOCKS][4];                       // the run's sums, in the end all runs'
#pragma unroll
    for (int i = 0; i < BLOCKS; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] = make_float2(0.f, 0.f);
    int in_run = 0, run_index = 0, s = 0;
    uint32_t phase = 0;
#pragma unroll 1
    for (int t = 0; t < tiles; ++t) {
      if (!at_wait(done + s, phase)) ok = false;
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int i = 0; i < BLOCKS; i += 2) {
        float2 v[2][4];
        const bool one = first + STEP * i < blocks, two = i + 1 < BLOCKS && first + STEP * (i + 1) < blocks;
        if (one) ld8(at + STEP * 8 * i, v[0]);
        if (two) ld8(at + STEP * 8 * (i + 1), v[1]);
        at_ld_wait();
        if (one) add8(acc[i], v[0]);
        if (two) add8(acc[i + 1 < BLOCKS ? i + 1 : i], v[1]);
      }
      const bool last = t == tiles - 1, close = ++in_run == per_run || last;
      if (close) {                                 // the run's sum; the sums of the runs before wait in TMEM
        const bool more = run_index % (GROUPS / 2) != 0;
#pragma unroll
        for (int i = 0; i < BLOCKS; ++i) {
          if (first + STEP * i >= blocks) continue;
          const uint32_t col = at + STEP * 8 * i;
          float2 d[4], d2[4];
          ld8(col + n, d);
          ld8(col + 2 * n, d2);
          at_ld_wait();
          add8(d, d2);
          add8(acc[i], d);
          if (more) {
            ld8(col + 3 * n, d);
            at_ld_wait();
            add8(acc[i], d);
          }
          if (ALONE && last && run_index >= GROUPS / 2) {
            ld8(col + 4 * n, d);
            at_ld_wait();
            add8(acc[i], d);
          }
          if (!last) {
            st8(col + (3 + (ALONE && run_index == GROUPS / 2 - 1)) * n, acc[i]);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] = make_float2(0.f, 0.f);
          }
        }
        ++run_index;
        at_st_wait();
        in_run = 0;
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        at_arrive(lead_read);
        if (close) at_arrive(rest_read);
      }
      if (++s == SLOTS) { s = 0; phase ^= 1; }
    }
    if (!ok && lane == 0) atomicExch(&gemm_f32_stuck, 43);
    // The sums go through shared memory (the last stage is multiplied: nothing reads or writes the stages any more) and are
    // finished in a loop: 64 of them a thread in straight line took 9 us, most of it to fetch the instructions.
    float* mine = part + first * 8 * 128 + (warp & 3) * 32 + lane;
    const float spoilt = ok ? 0.f : __uint_as_float(0x7fc00000u);
#pragma unroll
    for (int i = 0; i < BLOCKS; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (first + STEP * i < blocks) {
          mine[(STEP * 8 * i + 2 * e) * 128] = ok ? acc[i][e].x : spoilt;
          mine[(STEP * 8 * i + 2 * e + 1) * 128] = ok ? acc[i][e].y : spoilt;
        }
    if (S::UNEQUAL) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
      roles_end();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == S::WARPS)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::TMEM_COLS));
  if (!ALONE) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const uint32_t own = at_smem(part);
  // this CTA's rows of A (the MMA's warps stay out)
  uint32_t bad = 0;
  const int row_end = (rank + 1) * n / cs, end = warp < S::WARPS ? row_end * 128 : 0;
#pragma unroll 1
  for (int e = rank * n / cs * 128 + threadIdx.x; e < end; e += 32 * S::WARPS) {
    const int m = m0 + e / 128, nn = n0 + e % 128;
    if (m >= M || nn >= N) continue;
    float z = part[e];
    if (!ALONE) {
      constexpr int MOST = GROUPS / PER;           // CTAs; the first MOST / 2 have the first four runs
      float v[MOST];
#pragma unroll
      for (int g = 0; g < MOST; ++g) {
        if (g >= cs) continue;
        uint32_t far;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(own + 4u * e), "r"(g));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[g]) : "r"(far));
      }
      float lo = v[0], hi = v[MOST / 2];
#pragma unroll
      for (int g = 1; g < MOST / 2; ++g) {
        if (g < cs) lo += v[g];
        if (MOST / 2 + g < cs) hi += v[MOST / 2 + g];
      }
      z = cs > MOST / 2 ? lo + hi : lo;
    }
    z *= UNSCALE;
    if (is_finite(z)) {
      C[(size_t)m * ldc + nn] = finish(z + (bias ? bias[nn] : 0.f), inv_tau);
    } else {
      part[e] = z;                                 // a mark (nobody else reads this CTA's own part of its sums)
      bad = 1;
    }
  }
  bool again;
  if (ALONE) {
    if (warp >= S::WARPS) return;
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.or.pred p, 1, %2, q;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(any) : "r"(bad), "n"(32 * S::WARPS) : "memory");
    again = any;
  } else {
    if (bad) *marked = 1;
    // nobody leaves while its partial sums may still be read
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    again = *marked && warp < S::WARPS;
  }
  if (again)
    plain_rows<32 * S::WARPS, VEC>(A + (size_t)m0 * lda, lda, W + (size_t)n0 * ldw, ldw, bias ? bias + n0 : nullptr,
                                             C + (size_t)m0 * ldc + n0, ldc, rank * n / cs, min(row_end, M - m0), min(128, N - n0),
                                             K, run, inv_tau, part, part + n * 128);
}

// Products of few k, by plain multiply-adds: two chains per output, over its even and its odd k, added at the end.  Below
// SHORT_K the several roundings and the parts left out weigh more than the few roundings of the chains, so these take no
// tensor core.  Error against 64 bits, root mean square over the result's, split / chains, x 1e-9: one k 26.0 / 25.4, numbers
// of very unlike sizes 16 k 64.8 / 46.6, 32 k 74.0 / 64.7, 48 k 74.2 / 74.5; largest over the sum of |a| |w|, one k 88 / 60.
// All k of a tile lie in shared memory at once, [row][k], KP floats apart (eight neighbouring threads' 16 bytes meet every
// bank once); two k side by side are one fma.rn.f32x2.  Bound by the latency of its few steps.  us split / chains: one row of
// 2048x16 3.2 / 1.9, 48 rows 5.1 / 2.9, 333 rows 5.7 / 3.6; of 16384x32 3.3 / 2.4, 5.4 / 4.8, 24.6 / 14.7; of 2048x47
// 4.8 / 3.2, 7.0 / 5.0, 7.9 / 7.2.
#define SHORT_K 48
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_short_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, const float* __restrict__ bias,
                      float* __restrict__ C, int ldc, int M, int N, int K, float inv_tau, bool vec) {
  constexpr int NX = BN / TN, NY = BM / TM, T = NX * NY, KP = SHORT_K + 4;
  __shared__ __align__(16) float smem[(BM + BN) * KP];
  pdl_wait();
  pdl_trigger();
  const int tx = threadIdx.x % NX, ty = threadIdx.x / NX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // rows of A, then of W, in pieces of four k, zeros past the matrices: 4, 8 or 16 threads to a row (a division per piece
  // cost 0.7 us)
  const int shift = K <= 16 ? 2 : K <= 32 ? 3 : 4, k0 = (threadIdx.x & ((1 << shift) - 1)) * 4;
  if (k0 < K) {
#pragma unroll 4
    for (int r = threadIdx.x >> shift; r < BM + BN; r += T >> shift) {
      const bool in = r < BM ? m0 + r < M : n0 + r - BM < N;
      const float* src = !in ? A : (r < BM ? A + (size_t)(m0 + r) * lda : W + (size_t)(n0 + r - BM) * ldw) + k0;
      const uint32_t dst = at_smem(smem + r * KP + k0);
      if (vec) {
        cp_async16(dst, src, in ? 16 : 0);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) cp_async4(dst + 4 * e, in && k0 + e < K ? src + e : A, in && k0 + e < K ? 4 : 0);
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float2 acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float4 a[TM], w[TN];
#pragma unroll
    for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(smem + (ty + NY * i) * KP + k);
#pragma unroll
    for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(smem + (BM + tx + NX * j) * KP + k);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        fma2(acc[i][j], a[i].x, a[i].y, w[j].x, w[j].y);
        fma2(acc[i][j], a[i].z, a[i].w, w[j].z, w[j].w);
      }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + NY * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int nn = n0 + tx + NX * j;
      if (nn < N) C[(size_t)m * ldc + nn] = finish(acc[i][j].x + acc[i][j].y + (bias ? bias[nn] : 0.f), inv_tau);
    }
  }
}

struct F32Problem {
  const float *A, *W, *bias;
  float* C;
  int lda, ldw, ldc, M, N, K, run;
  float inv_tau;
  int n, cs;
  cudaStream_t stream;
};

template <int NT, bool VEC, int PER>
static int launch_f32(const F32Problem& p) {
  constexpr int smem = F32Shape<NT>::SMEM;
  auto kernel = gemm_f32_nt_kernel<NT, VEC, PER>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return AB_CUDA_ERR + (int)e;
  if (F32Shape<NT>::UNEQUAL) {                     // the roles' registers are shares of the launch's: with fewer they would wait
    static const int regs = [&] { cudaFuncAttributes a; return cudaFuncGetAttributes(&a, kernel) == cudaSuccess ? a.numRegs : 0; }();
    if (regs != 80) return AB_BAD_ARG;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + 127) / 128 * p.cs, (p.M + p.n - 1) / p.n);
  cfg.blockDim = dim3(F32Shape<NT>::THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = p.stream;
  cudaLaunchAttribute attr[2];
  if (PER < GROUPS) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = p.cs;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (ab_pdl_enabled() && !ab_pdl_held) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  cfg.attrs = attr;
  e = cudaLaunchKernelEx(&cfg, kernel, p.A, p.lda, p.W, p.ldw, p.bias, p.C, p.ldc, p.M, p.N, p.K, p.run, p.inv_tau, p.n, p.cs);
  return e == cudaSuccess ? AB_OK : AB_CUDA_ERR + (int)e;
}

template <int NT, bool VEC>
static int launch_f32(const F32Problem& p, int per) {
  return per == GROUPS ? launch_f32<NT, VEC, GROUPS>(p) : per == 1 ? launch_f32<NT, VEC, 1>(p) : launch_f32<NT, VEC, GROUPS / 2>(p);
}
template <int NT>
static int launch_f32(const F32Problem& p, bool vec, int per) {
  return vec ? launch_f32<NT, true>(p, per) : launch_f32<NT, false>(p, per);
}

// How a product is cut: k of a run, rows of a tile, the runs of a CTA and the CTAs that share a tile.
struct F32Plan {
  int run, n, per, cs;
};
static F32Plan plan_f32(int M, int N, int K, int sms) {
  F32Plan p;
  p.run = ((K + GROUPS - 1) / GROUPS + BK - 1) / BK * BK;
  if (p.run < SHORTEST) p.run = SHORTEST;
  // as few tiles of rows as 128 allow, then as low as they can be
  // (where a tile is one short run and 64 rows leave processors idle, by 64: 200 rows of 2048x128 11.4 -> 8.7 us)
  const int top = K <= SHORTEST && (long long)((N + 127) / 128) * ((M + 63) / 64) <= sms ? 64 : 128;
  const int row_tiles = (M + top - 1) / top;
  p.n = ((M + row_tiles - 1) / row_tiles + 15) / 16 * 16;
  const long long tiles = (long long)((N + 127) / 128) * row_tiles;
  // CTAs of a cluster of 1, 2, .. 8 that run at once on 148 processors, one per processor (what the runtime says)
  static const int together[GROUPS + 1] = {0, 148, 148, 135, 132, 130, 132, 105, 120};
  // Runs of a CTA: rounds of CTAs times what one takes.  It starts and ends in about four stages, and in one more with a
  // cluster or more than 64 rows; where two share a processor, each takes a third longer.  A cluster has as many CTAs as have
  // a run.  us with all runs / half of them / one in a CTA: one row of 2048x768 20.3 / 15.1 / 6.4, of 512x384 11.3 / - /
  // 6.4, of 16384x768 20.9 / 20.3 / 24.7; 200 rows of 2048x768 - / 27.7 / 22.2, of 16384x384 43 / - / 74; 333 rows of
  // 2048x2048 - / 44 / 60.  Of 480 products of 160 to 8,192 k none is more than a tenth slower than with the best of the
  // three.  (Clusters of two or eight alone, whether or not their CTAs had a run: one row of 2048x768 15.3.)
  const int runs = (K + p.run - 1) / p.run;
  p.per = GROUPS;
  p.cs = 1;
  long long best = 0;
  for (int per : {GROUPS, GROUPS / 2, 1}) {
    if (per == GROUPS && p.n > 96 && runs > GROUPS / 2) continue;      // no room for the second sum of runs
    const int cs = (runs + per - 1) / per;
    if (per < GROUPS && cs < 2) continue;                              // nothing to share
    const long long ctas = tiles * cs, alone = (long long)together[cs ? cs : 1] * sms / 148, at_once = p.n <= 32 ? 2 * alone : alone;
    const int k = K < p.run * per ? K : p.run * per;
    long long cost = (ctas + at_once - 1) / at_once * ((k + BK - 1) / BK + (p.n > 64 || cs > 1 ? 5 : 4)) * 10;
    if (p.n <= 32 && ctas > alone) cost = cost * 13 / 10;
    if (!best || cost < best) { best = cost; p.per = per; p.cs = cs > 1 ? cs : 1; }
  }
  return p;
}

template <int BM, int BN, int TM, int TN>
static int launch_short(const F32Problem& p, bool vec) {
  const cudaError_t e = ab_launch(gemm_f32_short_kernel<BM, BN, TM, TN>, dim3((p.N + BN - 1) / BN, (p.M + BM - 1) / BM),
                                  dim3((BM / TM) * (BN / TN)), 0, p.stream, p.A, p.lda, p.W, p.ldw, p.bias, p.C, p.ldc, p.M, p.N, p.K,
                                  p.inv_tau, vec);
  return e == cudaSuccess ? AB_OK : AB_CUDA_ERR + (int)e;
}

static int gemm_f32(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc, int M, int N,
                    int K, float inv_tau, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return AB_OK;
  if (K < 0) return AB_BAD_ARG;
  if ((M + 63) / 64 > 65535) return AB_BAD_ARG;
  // 16-byte copies where every row of both operands starts on a 16-byte boundary and ends on one
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
  int sms = 148, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  F32Problem p{A, W, bias, C, lda, ldw, ldc, M, N, K, 0, inv_tau, 0, 0, stream};
  if (K < SHORT_K) {
    // few rows: as low a tile as holds them; more: the tile that pads fewer, of equals the square one
    if (M <= 8) return launch_short<8, 128, 8, 1>(p, vec);
    if (M <= 16 || (M <= 32 && N <= 8192)) return launch_short<16, 128, 8, 2>(p, vec);
    const long long low = (M + 31) / 32 * 32LL, square = (M + 63) / 64 * 64LL;
    return low < square * 0.97 && low / 32 <= 65535 ? launch_short<32, 128, 8, 4>(p, vec) : launch_short<64, 64, 8, 4>(p, vec);
  }
  const F32Plan c = plan_f32(M, N, K, sms);
  p.run = c.run;
  p.n = c.n;
  p.cs = c.cs;
  if (c.n <= 16) return launch_f32<16>(p, vec, c.per);
  if (c.n <= 32) return launch_f32<32>(p, vec, c.per);
  if (c.n <= 64) return launch_f32<64>(p, vec, c.per);
  return launch_f32<128>(p, vec, c.per);
}

// The plan of a product on 148 processors: k of a run, rows of a tile, runs of a CTA, CTAs of a cluster
AB_API void ab_gemm_f32_plan(int M, int N, int K, int* out) {
  const F32Plan p = plan_f32(M, N, K, 148);
  out[0] = p.run;
  out[1] = p.n;
  out[2] = p.per;
  out[3] = p.cs;
}

AB_API int ab_gemm_f32_nt(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc,
                          int M, int N, int K, cudaStream_t stream) {
  return gemm_f32(A, lda, W, ldw, bias, C, ldc, M, N, K, 0.f, stream);
}

// C = sigmoid(A . W^T + bias)^(1 / tau): the decays of a gated linear attention from its low-rank projection
AB_API int ab_gemm_f32_decay(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc,
                             int M, int N, int K, float tau, cudaStream_t stream) {
  if (!(tau > 0.f)) return AB_BAD_ARG;
  return gemm_f32(A, lda, W, ldw, bias, C, ldc, M, N, K, 1.0f / tau, stream);
}

AB_API int ab_gemm_f32_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, gemm_f32_stuck, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(gemm_f32_stuck, &zero, sizeof(int));
  return v;
}
