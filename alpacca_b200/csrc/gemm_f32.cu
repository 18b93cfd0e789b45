// C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]) in true 32-bit: plain FMA on the CUDA
// cores, no tensor-core mode of reduced precision anywhere.
//
// The order of an output's sum depends on K alone: the k range is cut into up to GROUPS runs (of a
// multiple of BK, at least SHORTEST); a run is two chains of fused multiply-adds in ascending order, one over
// its even k and one over its odd k, added at its end; the runs are added in ascending order.  So a value does
// not depend on M, on the tile it falls into, on whether the runs of a tile are computed by one CTA or by a cluster of CTAs, or on
// what other rows are in the batch: the same token gives the same bits alone and in any batch.  This is the
// matrix product of the 32-bit path (the reference's float32 path uses BLAS SGEMM, alpacca/tensor.py:91-97).
//
// What bounds it: the FMA pipes (128 multiply-adds per clock and SM, 74 TFLOP/s) for many rows, HBM (the
// weights) for few.  Two k of an output side by side in a register pair are one fma.rn.f32x2, whose operands
// come out of 16-byte shared loads without packing, so half the issue slots are free for the loads.  Rows
// stay [row][k] in shared memory (cp.async, no transposition), BK + 4 floats apart: eight neighbouring
// threads read eight rows without a bank conflict.  It reaches 46 TFLOP/s (2,048 rows of
// 16384x2048: 5.4 -> 3.0 ms); two fma.rn.f32 in place of the pair measured the same, so the shared loads bind, not
// the FMA pipes.  333 rows of q|k|v, o, gate|up and down of the 1B shape: 216 -> 123, 215 -> 87, 1055 -> 573,
// 866 -> 312 us; one row: 116 -> 11, 116 -> 11, 212 -> 38, 461 -> 33 us (3.6 TB/s on gate|up).
#include "common.cuh"
#include "launch.cuh"

#define BK 32
#define KP (BK + 4)      // floats from row to row in shared memory
#define GROUPS 8         // runs of k; also the CTAs of a cluster that share a tile
#define SHORTEST 128     // a run's k at least: adding up runs of 32 was a fifth of a product over 128 k
#define STAGES 2         // two of four CTAs per SM hide the copies: a third stage, three CTAs per SM, was 0 to 10 % slower

__device__ __forceinline__ void cp_async16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes));
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float pair_sum(unsigned long long v) {
  return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32));
}

// R rows from row r0 (n_rows exist; the others become zeros) of k0 .. k0 + BK - 1 (zeros from kend on).  A thread keeps its k
// and steps from row to row: an addition per copy where rows are not 16-byte aligned and a copy is four bytes (a
// division and a product of 64 bits per copy: 2,000 rows of 3000x1021 524 us, 454 with plain loads before, 359 now).
template <int R, int T, bool VEC>
__device__ __forceinline__ void stage_rows(float* dst, const float* src, int ld, int r0, int n_rows, int k0, int kend) {
  constexpr int W = VEC ? 4 : 1, RS = T / (BK / W);      // floats per copy, rows between a thread's copies
  static_assert(T % (BK / W) == 0 && (R % RS == 0 || R < RS), "whole rounds of copies");
  const int r = threadIdx.x / (BK / W), k = threadIdx.x % (BK / W) * W;
  if (R < RS && r >= R) return;
  const bool k_in = k0 + k < kend;                       // VEC: kend is a multiple of 4
  const float* p = src + (size_t)(r0 + r) * ld + k0 + k;
  float* d = dst + r * KP + k;
#pragma unroll 4
  for (int i = 0; i < (R + RS - 1) / RS; ++i, p += (size_t)RS * ld, d += RS * KP) {
    const bool in = k_in && r0 + r + i * RS < n_rows;
    if (VEC) cp_async16(d, in ? p : src, in ? 16 : 0);
    else cp_async4(d, in ? p : src, in ? 4 : 0);
  }
}

// the product's last step: z (bias included), or with inv_tau > 0 a decay, sigmoid(z)^inv_tau
__device__ __forceinline__ float finish(float z, float inv_tau) {
  if (inv_tau <= 0.f) return z;
  const float sp = -z > 20.f ? -z : log1pf(expf(-z));      // -log sigmoid(z)
  return expf(-sp * inv_tau);
}

// A tile of BM x BN outputs; a thread owns rows ty + NY i and columns tx + NX j.  SPLIT: the CTA of rank r in its
// cluster of GROUPS computes run r, then every CTA adds up an eighth of the tile through distributed shared memory.
template <int BM, int BN, int TM, int TN, bool VEC, bool SPLIT>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 4)
gemm_f32_nt_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                   const float* __restrict__ bias, float* __restrict__ C, int ldc, int M, int N, int K, int run,
                   float inv_tau) {
  constexpr int NX = BN / TN, NY = BM / TM, T = NX * NY;
  constexpr int STAGE = (BM + BN) * KP;
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  pdl_trigger();
  const int tx = threadIdx.x % NX, ty = threadIdx.x / NX;
  const int rank = SPLIT ? (int)(blockIdx.x % GROUPS) : 0;      // the cluster lies along x
  const int m0 = blockIdx.y * BM, n0 = (SPLIT ? blockIdx.x / GROUPS : blockIdx.x) * BN;
  const int kbegin = SPLIT ? min(K, rank * run) : 0, kend = SPLIT ? min(K, kbegin + run) : K;
  const int tiles = (kend - kbegin + BK - 1) / BK, per_run = run / BK;

  unsigned long long acc[TM][TN];
  float tot[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) { acc[i][j] = 0ull; tot[i][j] = 0.f; }

  // A thread copies the same four k of rows CR apart.  Inside the matrices that is an addition per copy: rows of A
  // below the last one read the last one (their outputs are not stored), W's rows lie a fixed step apart.
  constexpr int CR = T / (BK / 4), AR = BM > CR ? BM / CR : 1, WR = BN / CR;
  static_assert(BN % CR == 0 && (BM % CR == 0 || BM < CR), "whole rounds of copies");
  const int cr = threadIdx.x / (BK / 4), ck = threadIdx.x % (BK / 4) * 4;
  const float* ap[AR];
#pragma unroll
  for (int i = 0; i < AR; ++i) ap[i] = A + (size_t)min(m0 + cr + CR * i, M - 1) * lda + kbegin + ck;
  const float* wp = W + (size_t)min(n0 + cr, N - 1) * ldw + kbegin + ck;
  const size_t wstep = (size_t)CR * ldw;
  const bool inside = n0 + BN <= N;
  auto stage = [&](int t) {
    if (t < tiles) {
      float* s = smem + (t % STAGES) * STAGE;
      const int k0 = kbegin + t * BK;
      if (VEC && inside && k0 + BK <= kend) {
        float* d = s + cr * KP + ck;
        if (BM >= CR || cr < BM) {
#pragma unroll
          for (int i = 0; i < AR; ++i) cp_async16(d + CR * i * KP, ap[i] + t * BK, 16);
        }
        const float* w = wp + t * BK;
#pragma unroll
        for (int i = 0; i < WR; ++i) cp_async16(d + (BM + CR * i) * KP, w + i * wstep, 16);
      } else {
        stage_rows<BM, T, VEC>(s, A, lda, m0, M, k0, kend);
        stage_rows<BN, T, VEC>(s + BM * KP, W, ldw, n0, N, k0, kend);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");       // an empty group past the end keeps the count
  };
#pragma unroll
  for (int t = 0; t < STAGES - 1; ++t) stage(t);
  int in_run = 0;
  bool first = true;
#pragma unroll 1
  for (int t = 0; t < tiles; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                       // tile t is there for everybody; the buffer of tile t - 1 is free
    stage(t + STAGES - 1);
    const float* a_s = smem + (t % STAGES) * STAGE + ty * KP;
    const float* w_s = smem + (t % STAGES) * STAGE + (BM + tx) * KP;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {

      ulonglong2 a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(a_s + i * NY * KP + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(w_s + j * NX * KP + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a[i].x, w[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a[i].y, w[j].y, acc[i][j]);
    }
    if (++in_run == per_run || t == tiles - 1) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          tot[i][j] = first ? pair_sum(acc[i][j]) : tot[i][j] + pair_sum(acc[i][j]);
          acc[i][j] = 0ull;
        }
      in_run = 0;
      first = false;
    }
  }
  if (!SPLIT) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + ty + NY * i;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int n = n0 + tx + NX * j;
        if (n < N) C[(size_t)m * ldc + n] = finish(tot[i][j] + (bias ? bias[n] : 0.f), inv_tau);
      }
    }
    return;
  }
  __syncthreads();                         // the last tile has been read; no copy is in flight (only empty groups)
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) smem[(ty + NY * i) * BN + tx + NX * j] = tot[i][j];
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int runs = (K + run - 1) / run;
  const unsigned mine = (unsigned)__cvta_generic_to_shared(smem);
  for (int e = rank * (BM * BN / GROUPS) + threadIdx.x; e < (rank + 1) * (BM * BN / GROUPS); e += T) {
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (m >= M || n >= N) continue;
    float v[GROUPS];
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      unsigned there;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(mine + 4u * e), "r"(g));
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[g]) : "r"(there));
    }
    float sum = v[0];
#pragma unroll
    for (int g = 1; g < GROUPS; ++g)
      if (g < runs) sum += v[g];
    C[(size_t)m * ldc + n] = finish(sum + (bias ? bias[n] : 0.f), inv_tau);
  }
  // nobody leaves while its partial sums may still be read
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct F32Problem {
  const float *A, *W, *bias;
  float* C;
  int lda, ldw, ldc, M, N, K, run;
  float inv_tau;
  cudaStream_t stream;
};

template <int BM, int BN, int TM, int TN, bool VEC, bool SPLIT>
static int launch_f32(const F32Problem& p) {
  constexpr int smem = STAGES * (BM + BN) * KP * 4;
  static_assert(smem >= BM * BN * 4 && (BM * BN) % GROUPS == 0, "the partial sums take the tiles' place");
  auto kernel = gemm_f32_nt_kernel<BM, BN, TM, TN, VEC, SPLIT>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return AB_CUDA_ERR + (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + BN - 1) / BN * (SPLIT ? GROUPS : 1), (p.M + BM - 1) / BM);
  cfg.blockDim = dim3((BM / TM) * (BN / TN));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = p.stream;
  cudaLaunchAttribute attr[2];
  if (SPLIT) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = GROUPS;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (ab_pdl_enabled() && !ab_pdl_held) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  cfg.attrs = attr;
  e = cudaLaunchKernelEx(&cfg, kernel, p.A, p.lda, p.W, p.ldw, p.bias, p.C, p.ldc, p.M, p.N, p.K, p.run, p.inv_tau);
  return e == cudaSuccess ? AB_OK : AB_CUDA_ERR + (int)e;
}

template <int BM, int BN, int TM, int TN>
static int launch_f32(const F32Problem& p, bool vec, bool split) {
  if (vec) return split ? launch_f32<BM, BN, TM, TN, true, true>(p) : launch_f32<BM, BN, TM, TN, true, false>(p);
  return split ? launch_f32<BM, BN, TM, TN, false, true>(p) : launch_f32<BM, BN, TM, TN, false, false>(p);
}

static int gemm_f32(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc, int M, int N,
                    int K, float inv_tau, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return AB_OK;
  if (K < 0) return AB_BAD_ARG;
  if ((M + 63) / 64 > 65535) return AB_BAD_ARG;
  F32Problem p{A, W, bias, C, lda, ldw, ldc, M, N, K, 0, inv_tau, stream};
  p.run = ((K + GROUPS - 1) / GROUPS + BK - 1) / BK * BK;
  if (p.run < SHORTEST) p.run = SHORTEST;
  // 16-byte copies where every row of both operands starts on a 16-byte boundary and ends on one
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
  int sms = 148, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Split a tile's runs over a cluster where there are few tiles per SM: an SM needs three or four CTAs to fill its
  // pipes, and the last round is as long as a run.  us whole / split: 333 rows of 2048x2048 (1.2 tiles per SM) 122 / 87,
  // 777 of 3072x2048 (4.1) 280 / 259, 2,048 of 2048x2048 (6.9) 391 / 425, 333 of 16384x2048 (9.5) 573 / 590.
  auto split = [&](int bm, int bn) {
    const long long tiles = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
    return K >= 512 && tiles < 6LL * sms;
  };
  // Few rows are bound by the weights' bytes and the chain of a run: as low a tile as holds them.
  if (M <= 8) return launch_f32<8, 128, 8, 1>(p, vec, split(8, 128));
  if (M <= 16 || (M <= 32 && N <= 8192)) return launch_f32<16, 128, 8, 2>(p, vec, split(16, 128));
  // The tile that pads fewer rows; of equals the square one (2,048 rows: 4 % faster).
  const long long low = (M + 31) / 32 * 32LL, square = (M + 63) / 64 * 64LL;
  if (low < square * 0.97 && low / 32 <= 65535) return launch_f32<32, 128, 8, 4>(p, vec, split(32, 128));
  return launch_f32<64, 64, 8, 4>(p, vec, split(64, 64));
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
