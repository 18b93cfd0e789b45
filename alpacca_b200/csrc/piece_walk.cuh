// The walk of a recurrence S_t = decay_t S_{t-1} + k_t v_t^T, o_t = S_t^T q_t over prompts, in pieces of a sequence that
// are walked side by side: 32-bit multiply-adds, S [D, V] per (sequence, head).
//
//   CHANNEL   a decay per key row: S <- diag(a_t) S + k_t v_t^T          (a_t: D numbers per head and token)
//   SCALAR    a decay and a factor per head: S <- keep_t S + add_t k_t v_t^T     (coef [T, H, 3]: keep, add, -)
//
//   piece_local   what a piece alone leaves, S = sum over its tokens of (decays after the token) k v^T, walked backwards so
//                 that the decays after a token are one running product per row; and the product over the whole piece
//   piece_scan    per number of S: the state before every piece, from the sequence's state on
//   piece_walk    every piece from the state before it, with the read-outs; the last one leaves the sequence's state
//
// A thread holds 4 J rows x 4 columns of S (rows 32 j + 4 (lane % 8) .. + 3, j < J = D / 32): a token's 12 J numbers of q, k
// and decays that it loads from shared memory serve 16 J numbers of S, two rows side by side in one f32x2 operation, and
// eight lanes add their shares of four columns in four exchanges.  A thread with one column and 8 to 16 rows loads three
// numbers per number of S: that walk was bound by its shared loads (4.5 TFLOP/s).  Bound now by the FMA pipes: three
// operations per number of S and token with a decay per row, and half as much again for the local pass.
// One sequence of 2,048 tokens, 8 heads of 128 x 256 with one decay each, the whole mixer 522 -> 258 us (the walk token by
// token with one column per thread 448 us); 2,500 tokens of two sequences, 16 heads of 128 x 128 with a decay per row, the
// whole mixer with its decays out of the 32-bit product 898 -> 331 us (the walk 640).
// Pieces of one length for all sequences, as many as run at once (or in two rounds), and lanes that never leave the exchanges: 274
// -> 258, 371 -> 331 us against pieces counted per sequence.  A long prompt beside rows of one token is cut like a prompt alone:
// matrix memory, 8 heads, 2,048 + 17 x 1 tokens 1,300 -> 278 us, 8,192 + 11 x 1 3,073 -> 976, against a room shared by number of
// sequences; eight of 2,000 to 3,750 tokens in two rounds 3,109 -> 2,569.
#pragma once
#include "common.cuh"
#include "launch.cuh"

#define PW_TOKENS 8        // tokens staged per round
#define PW_STAGES 3        // rounds in flight or in use
#define PW_COLS 128        // most columns of [S | n] per CTA, four per eight lanes; tiles are of equal width

struct PieceArgs {
  const float *q, *k, *v;      // a token's rows at q + t * ldq + h * D, v + t * ldv + h * V; 16-byte aligned
  int ldq, ldk, ldv;
  const float* decay;          // CHANNEL: decay + t * ldd + h * D
  int ldd;
  const float* coef;           // SCALAR
  float* state;                // [slots, H, state_row]: S [D][V], then (WITH_N) n [D]
  int state_row;
  float* out;                  // out + (t * H + h) * out_row + column
  int out_row;
  const int *cu_q, *slots;
  int n_seqs, H, V, length;    // tokens per piece
  int items, kept;             // pieces of all sequences, and of those that have more than one (the host's sums)
  int cols;                    // columns per CTA, a multiple of 4 (set by the launch)
  float qscale;
  int write_state;
  float* local;                // [kept, H][D][V + (WITH_N ? 4 : 0)]
  float* prod;                 // [kept, H][CHANNEL ? D : 1]
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pw_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 pw_mul(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 pw_pair(float lo, float hi) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void pw_split(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void pw_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void pw_copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

// A piece: `length` of its sequence's tokens (a multiple of PW_TOKENS), the last one what is left.  Items count the pieces of
// all sequences one after another; every warp finds its own by itself, 32 sequences at a time, from the lengths on the device.
struct Piece {
  int b = -1;          // sequence; -1: no such item
  int n = 0, p = 0;    // its pieces, and which of them
  int at = 0;          // the sequence's first place in `local` (n > 1)
  int begin, end;
  // by_sequence: `item` is a sequence (begin and end are all of its tokens)
  __device__ __forceinline__ Piece(const int* __restrict__ cu_q, int n_seqs, int length, int item, bool by_sequence) {
    const int lane = threadIdx.x & 31;
    int items = 0, kept = 0;
    for (int base = 0; base < n_seqs; base += 32) {
      const int i = base + lane;
      const int t0 = cu_q[min(i, n_seqs)], t1 = cu_q[min(i + 1, n_seqs)];
      const unsigned pieces = (unsigned)(t1 - t0 + length - 1) / (unsigned)length;
      const unsigned word = pieces | (pieces > 1 ? pieces << 16 : 0u);      // both sums in one: 65,535 items at most
      unsigned up = word;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, up, o);
        if (lane >= o) up += v;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, by_sequence ? i == item : items + (int)(up & 0xffffu) > item);
      if (hit) {
        const int l = __ffs(hit) - 1;
        const unsigned before = __shfl_sync(0xffffffffu, up - word, l);
        b = base + l;
        n = (int)__shfl_sync(0xffffffffu, pieces, l);
        at = kept + (int)(before >> 16);
        begin = __shfl_sync(0xffffffffu, t0, l);
        end = __shfl_sync(0xffffffffu, t1, l);
        if (!by_sequence) {
          p = item - items - (int)(before & 0xffffu);
          begin += p * length;
          end = min(end, begin + length);
        }
        return;
      }
      const unsigned all = __shfl_sync(0xffffffffu, up, 31);
      items += (int)(all & 0xffffu);
      kept += (int)(all >> 16);
    }
  }
};

// the numbers of S that a thread holds, as pairs of rows
template <int J> struct PieceTile { f32x2 s[J][4][2]; };

template <int J>
__device__ __forceinline__ void tile_load(PieceTile<J>& m, const float* src, int ld, int dg) {      // src: row 0 of the thread's columns
#pragma unroll
  for (int j = 0; j < J; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float4 a = *reinterpret_cast<const float4*>(src + (size_t)(32 * j + 4 * dg + 2 * e) * ld);
      const float4 b = *reinterpret_cast<const float4*>(src + (size_t)(32 * j + 4 * dg + 2 * e + 1) * ld);
      m.s[j][0][e] = pw_pair(a.x, b.x);
      m.s[j][1][e] = pw_pair(a.y, b.y);
      m.s[j][2][e] = pw_pair(a.z, b.z);
      m.s[j][3][e] = pw_pair(a.w, b.w);
    }
}
template <int J>
__device__ __forceinline__ void tile_store(const PieceTile<J>& m, float* dst, int ld, int dg) {
#pragma unroll
  for (int j = 0; j < J; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float4 a, b;
      pw_split(m.s[j][0][e], a.x, b.x);
      pw_split(m.s[j][1][e], a.y, b.y);
      pw_split(m.s[j][2][e], a.z, b.z);
      pw_split(m.s[j][3][e], a.w, b.w);
      *reinterpret_cast<float4*>(dst + (size_t)(32 * j + 4 * dg + 2 * e) * ld) = a;
      *reinterpret_cast<float4*>(dst + (size_t)(32 * j + 4 * dg + 2 * e + 1) * ld) = b;
    }
}

// What a thread works on: four columns of [S | n] (c0 == V: n, whose value is 1, and three that stay zero)
struct PieceLane {
  int dg, c0;        // rows' share; first of the four columns
  int at;            // where the values lie in a staged row
  bool live;
  __device__ __forceinline__ PieceLane(int width, int cols) {
    dg = threadIdx.x & 7;
    const int c = (int)(threadIdx.x >> 3) * 4;
    c0 = blockIdx.x * cols + c;
    live = c < cols && c0 < width;
    at = c;          // (below PW_COLS: a block has 8 lanes for every four of its columns)
  }
};

template <int J, bool CHANNEL, bool READS_Q>
struct PieceRound {      // where a round's rows lie in shared memory, in floats
  static constexpr int D = 32 * J;
  static constexpr int K = 0, Q = K + PW_TOKENS * D, A = Q + (READS_Q ? PW_TOKENS * D : 0),
                       V = A + (CHANNEL ? PW_TOKENS * D : 0), C = V + PW_TOKENS * PW_COLS, SIZE = C + 2 * PW_TOKENS;
};

template <int J, bool CHANNEL, bool READS_Q>
__device__ __forceinline__ void stage_round(float* base, const PieceArgs& a, int h, int t, int n) {
  using R = PieceRound<J, CHANNEL, READS_Q>;
  constexpr int D = 32 * J;
  for (int i = threadIdx.x; i < n * (D / 4); i += blockDim.x) {
    const int tt = i / (D / 4), c = i % (D / 4) * 4;
    pw_copy16(base + R::K + tt * D + c, a.k + (size_t)(t + tt) * a.ldk + h * D + c);
    if (READS_Q) pw_copy16(base + R::Q + tt * D + c, a.q + (size_t)(t + tt) * a.ldq + h * D + c);
    if (CHANNEL) pw_copy16(base + R::A + tt * D + c, a.decay + (size_t)(t + tt) * a.ldd + h * D + c);
  }
  const int col0 = blockIdx.x * a.cols, left = min(a.cols, a.V - col0);      // (0 or less: n alone)
  for (int i = threadIdx.x; i < n * (PW_COLS / 4); i += blockDim.x) {
    const int tt = i / (PW_COLS / 4), c = i % (PW_COLS / 4) * 4;
    if (c < left) pw_copy16(base + R::V + tt * PW_COLS + c, a.v + (size_t)(t + tt) * a.ldv + h * a.V + col0 + c);
  }
  if (!CHANNEL && (int)threadIdx.x < 2 * n) {
    const int tt = threadIdx.x >> 1, c = threadIdx.x & 1;
    pw_copy4(base + R::C + 2 * tt + c, a.coef + ((size_t)(t + tt) * a.H + h) * 3 + c);
  }
}
__device__ __forceinline__ void pw_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void pw_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PW_STAGES - 2) : "memory"); }

// grid (tiles of columns, H, items)
template <int J, bool CHANNEL, bool WITH_N>
__global__ void __launch_bounds__(8 * PW_COLS / 4, J <= 4 ? 2 : 1) piece_local_kernel(PieceArgs a) {
  using R = PieceRound<J, CHANNEL, false>;
  constexpr int D = 32 * J;
  extern __shared__ __align__(16) float pw_sm[];
  pdl_wait();
  pdl_trigger();
  const int h = blockIdx.y;
  const Piece piece(a.cu_q, a.n_seqs, a.length, blockIdx.z, false);
  if (piece.b < 0 || piece.p + 1 >= piece.n || a.slots[piece.b] < 0) return;      // nothing follows the last piece
  __shared__ int kept_place;                     // SCALAR: needed after the walk, whose registers are all taken
  if (!CHANNEL && threadIdx.x == 0) kept_place = piece.at + piece.p;
  const PieceLane me(a.V + (WITH_N ? 4 : 0), a.cols);
  const bool is_n = WITH_N && me.c0 >= a.V;
  const int rounds = (piece.end - piece.begin) / PW_TOKENS;                  // whole ones: the piece is not the last
  PieceTile<J> m;
#pragma unroll
  for (int j = 0; j < J; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) m.s[j][c][0] = m.s[j][c][1] = 0ull;
  f32x2 w[CHANNEL ? J : 1][2];                   // the decays after the token, of the thread's rows
  float ws = 1.f;
#pragma unroll
  for (int j = 0; j < (CHANNEL ? J : 1); ++j) w[j][0] = w[j][1] = pw_pair(1.f, 1.f);
  auto stage = [&](int r) {
    if (r < rounds)
      stage_round<J, CHANNEL, false>(pw_sm + r % PW_STAGES * R::SIZE, a, h, piece.end - (r + 1) * PW_TOKENS, PW_TOKENS);
    pw_commit();
  };
  for (int r = 0; r < PW_STAGES - 1; ++r) stage(r);
  for (int r = 0; r < rounds; ++r) {
    pw_wait();
    __syncthreads();
    stage(r + PW_STAGES - 1);
    const float* base = pw_sm + r % PW_STAGES * R::SIZE;
    {
#pragma unroll 2
      for (int tt = PW_TOKENS - 1; tt >= 0; --tt) {
        float4 v = *reinterpret_cast<const float4*>(base + R::V + tt * PW_COLS + me.at);
        if (WITH_N && is_n) v = make_float4(1.f, 0.f, 0.f, 0.f);
        if (!CHANNEL) {
          const float f = base[R::C + 2 * tt + 1] * ws;
          v.x *= f; v.y *= f; v.z *= f; v.w *= f;
          ws *= base[R::C + 2 * tt];
        }
        const f32x2 vv[4] = {pw_pair(v.x, v.x), pw_pair(v.y, v.y), pw_pair(v.z, v.z), pw_pair(v.w, v.w)};
#pragma unroll
        for (int j = 0; j < J; ++j) {
          ulonglong2 k = *reinterpret_cast<const ulonglong2*>(base + R::K + tt * D + 32 * j + 4 * me.dg);
          if (CHANNEL) {
            const ulonglong2 dc = *reinterpret_cast<const ulonglong2*>(base + R::A + tt * D + 32 * j + 4 * me.dg);
            k.x = pw_mul(k.x, w[j][0]);
            k.y = pw_mul(k.y, w[j][1]);
            w[j][0] = pw_mul(w[j][0], dc.x);
            w[j][1] = pw_mul(w[j][1], dc.y);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            m.s[j][c][0] = pw_fma(k.x, vv[c], m.s[j][c][0]);
            m.s[j][c][1] = pw_fma(k.y, vv[c], m.s[j][c][1]);
          }
        }
      }
    }
  }
  if (!me.live) return;
  const int VW = a.V + (WITH_N ? 4 : 0);
  const size_t at = (size_t)(CHANNEL ? piece.at + piece.p : kept_place) * a.H + h;      // (written before the first round's barrier)
  tile_store<J>(m, a.local + at * D * VW + me.c0, VW, me.dg);
  if (blockIdx.x == 0 && me.c0 == 0) {
    if (CHANNEL) {
#pragma unroll
      for (int j = 0; j < J; ++j) {
        ulonglong2 x;
        x.x = w[j][0];
        x.y = w[j][1];
        *reinterpret_cast<ulonglong2*>(a.prod + at * D + 32 * j + 4 * me.dg) = x;
      }
    } else if (me.dg == 0) {
      a.prod[at] = ws;
    }
  }
}

// grid (ceil(D * VW / 4 / 256), H, n_seqs): four neighbouring columns of a row per thread
template <bool CHANNEL, bool WITH_N>
__global__ void __launch_bounds__(256) piece_scan_kernel(PieceArgs a, int D) {
  pdl_wait();
  pdl_trigger();
  const int h = blockIdx.y, VW = a.V + (WITH_N ? 4 : 0);
  const int i = blockIdx.x * 256 + threadIdx.x;
  const Piece seq(a.cu_q, a.n_seqs, a.length, blockIdx.z, true);
  if (seq.n < 2) return;                         // walked from the sequence's state as it stands
  const int slot = a.slots[seq.b], n = seq.n;
  if (slot < 0 || i >= D * (VW / 4)) return;
  const int d = i / (VW / 4), c = i % (VW / 4) * 4;
  const float* st = a.state + ((size_t)slot * a.H + h) * a.state_row;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < a.V) s = *reinterpret_cast<const float4*>(st + (size_t)d * a.V + c);
  else s.x = st[(size_t)D * a.V + d];            // n
  const size_t first = (size_t)seq.at * a.H + h;
  float* l = a.local + first * D * VW + (size_t)d * VW + c;
  const float* f = a.prod + first * (CHANNEL ? D : 1) + (CHANNEL ? d : 0);
  const size_t step = (size_t)a.H * D * VW, f_step = (size_t)a.H * (CHANNEL ? D : 1);
  float4 next = make_float4(0.f, 0.f, 0.f, 0.f);
  float keep = 0.f;
  next = *reinterpret_cast<const float4*>(l);
  keep = f[0];
  for (int p = 0; p < n; ++p) {
    const float4 own = next;
    const float g = keep;
    if (p + 2 < n) {                             // asked for before the store that might hold it up
      next = *reinterpret_cast<const float4*>(l + (p + 1) * step);
      keep = f[(p + 1) * f_step];
    }
    *reinterpret_cast<float4*>(l + p * step) = s;
    s.x = fmaf(g, s.x, own.x);
    s.y = fmaf(g, s.y, own.y);
    s.z = fmaf(g, s.z, own.z);
    s.w = fmaf(g, s.w, own.w);
  }
}

// grid (tiles of columns, H, items)
template <int J, bool CHANNEL, bool WITH_N>
__global__ void __launch_bounds__(8 * PW_COLS / 4, J <= 4 ? 2 : 1) piece_walk_kernel(PieceArgs a) {
  using R = PieceRound<J, CHANNEL, true>;
  constexpr int D = 32 * J;
  extern __shared__ __align__(16) float pw_sm[];
  pdl_wait();
  pdl_trigger();
  const int h = blockIdx.y;
  const Piece piece(a.cu_q, a.n_seqs, a.length, blockIdx.z, false);
  const int slot = piece.b < 0 ? -1 : a.slots[piece.b];
  if (slot < 0) return;
  __shared__ int last_of;                        // SCALAR: needed after the walk, whose registers are all taken
  if (!CHANNEL && threadIdx.x == 0) last_of = piece.p + 1 < piece.n ? -1 : slot;
  const PieceLane me(a.V + (WITH_N ? 4 : 0), a.cols);
  const bool is_n = WITH_N && me.c0 >= a.V;
  auto stage = [&](int r) {
    const int t = piece.begin + r * PW_TOKENS;
    if (t < piece.end) stage_round<J, CHANNEL, true>(pw_sm + r % PW_STAGES * R::SIZE, a, h, t, min(PW_TOKENS, piece.end - t));
    pw_commit();
  };
  for (int r = 0; r < PW_STAGES - 1; ++r) stage(r);
  PieceTile<J> m = {};
  float* st = a.state + ((size_t)slot * a.H + h) * a.state_row;
  if (me.live) {
    const int VW = a.V + (WITH_N ? 4 : 0);
    if (piece.n > 1) {
      tile_load<J>(m, a.local + ((size_t)(piece.at + piece.p) * a.H + h) * D * VW + me.c0, VW, me.dg);
    } else if (!is_n) {
      tile_load<J>(m, st + me.c0, a.V, me.dg);
    } else {
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(st + (size_t)D * a.V + 32 * j + 4 * me.dg);
        m.s[j][0][0] = x.x;
        m.s[j][0][1] = x.y;
#pragma unroll
        for (int c = 1; c < 4; ++c) m.s[j][c][0] = m.s[j][c][1] = 0ull;
      }
    }
  }
  const int rounds = (piece.end - piece.begin + PW_TOKENS - 1) / PW_TOKENS;
  // after the exchanges a lane holds column c0 + (dg >> 2) * 2 + (dg >> 1 & 1), its neighbour the same one
  const bool writes = me.live && !(me.dg & 1) && (!is_n || me.dg == 0), up4 = me.dg & 4, up2 = me.dg & 2;
  const size_t out_step = (size_t)a.H * a.out_row;
  float* out = a.out + ((size_t)piece.begin * a.H + h) * a.out_row + me.c0 + (up4 ? 2 : 0) + (up2 ? 1 : 0);
  for (int r = 0; r < rounds; ++r) {
    pw_wait();
    __syncthreads();
    stage(r + PW_STAGES - 1);
    const float* base = pw_sm + r % PW_STAGES * R::SIZE;
    const int n = min(PW_TOKENS, piece.end - piece.begin - r * PW_TOKENS);
    {
#pragma unroll 2
      for (int tt = 0; tt < n; ++tt, out += out_step) {
        float4 v = *reinterpret_cast<const float4*>(base + R::V + tt * PW_COLS + me.at);
        if (WITH_N && is_n) v = make_float4(1.f, 0.f, 0.f, 0.f);
        f32x2 keep = 0ull;
        if (!CHANNEL) {
          const float f = base[R::C + 2 * tt + 1];
          v.x *= f; v.y *= f; v.z *= f; v.w *= f;
          keep = pw_pair(base[R::C + 2 * tt], base[R::C + 2 * tt]);
        }
        const f32x2 vv[4] = {pw_pair(v.x, v.x), pw_pair(v.y, v.y), pw_pair(v.z, v.z), pw_pair(v.w, v.w)};
        f32x2 o[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(base + R::K + tt * D + 32 * j + 4 * me.dg);
          const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(base + R::Q + tt * D + 32 * j + 4 * me.dg);
          ulonglong2 dc;
          if (CHANNEL) dc = *reinterpret_cast<const ulonglong2*>(base + R::A + tt * D + 32 * j + 4 * me.dg);
          else dc.x = dc.y = keep;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            m.s[j][c][0] = pw_fma(k.x, vv[c], pw_mul(dc.x, m.s[j][c][0]));
            m.s[j][c][1] = pw_fma(k.y, vv[c], pw_mul(dc.y, m.s[j][c][1]));
            o[c] = pw_fma(m.s[j][c][0], q.x, o[c]);
            o[c] = pw_fma(m.s[j][c][1], q.y, o[c]);
          }
        }
        float x[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float lo, hi;
          pw_split(o[c], lo, hi);
          x[c] = lo + hi;
        }
        // eight lanes' shares of four columns: each exchange halves the columns that a lane looks after
        const float y0 = (up4 ? x[2] : x[0]) + __shfl_xor_sync(0xffffffffu, up4 ? x[0] : x[2], 4);
        const float y1 = (up4 ? x[3] : x[1]) + __shfl_xor_sync(0xffffffffu, up4 ? x[1] : x[3], 4);
        float z = (up2 ? y1 : y0) + __shfl_xor_sync(0xffffffffu, up2 ? y0 : y1, 2);
        z += __shfl_xor_sync(0xffffffffu, z, 1);
        if (writes) *out = z * a.qscale;
      }
    }
  }
  if (!a.write_state || !me.live || (CHANNEL ? piece.p + 1 < piece.n : last_of < 0)) return;
  if (!CHANNEL) st = a.state + ((size_t)last_of * a.H + h) * a.state_row;
  if (!is_n) {
    tile_store<J>(m, st + me.c0, a.V, me.dg);
  } else {
#pragma unroll
    for (int j = 0; j < J; ++j) {
      ulonglong2 x;
      x.x = m.s[j][0][0];
      x.y = m.s[j][0][1];
      *reinterpret_cast<ulonglong2*>(st + (size_t)D * a.V + 32 * j + 4 * me.dg) = x;
    }
  }
}

// Sizes the walk takes: D in steps of 32 up to 256 (J of the list below), V in steps of 4; the caller checks alignments.
static inline bool piece_walk_takes(int D, int V) {
  return V > 0 && V % 4 == 0 && (D == 32 || D == 64 || D == 96 || D == 128 || D == 192 || D == 256);
}

template <int J, bool CHANNEL, bool WITH_N>
static int piece_walk_go(PieceArgs a, cudaStream_t stream) {
  const int D = 32 * J, width = a.V + (WITH_N ? 4 : 0), tiles = (width + PW_COLS - 1) / PW_COLS;
  a.cols = ((width + tiles - 1) / tiles + 3) / 4 * 4;
  const dim3 block((a.cols + 15) / 16 * 32);
  const int local_smem = PW_STAGES * PieceRound<J, CHANNEL, false>::SIZE * 4, walk_smem = PW_STAGES * PieceRound<J, CHANNEL, true>::SIZE * 4;
  cudaError_t e = cudaFuncSetAttribute(piece_local_kernel<J, CHANNEL, WITH_N>, cudaFuncAttributeMaxDynamicSharedMemorySize, local_smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(piece_walk_kernel<J, CHANNEL, WITH_N>, cudaFuncAttributeMaxDynamicSharedMemorySize, walk_smem);
  if (e != cudaSuccess) return AB_CUDA_ERR + (int)e;
  if (a.kept > 0) {
    ab_launch(piece_local_kernel<J, CHANNEL, WITH_N>, dim3(tiles, a.H, a.items), block, local_smem, stream, a);
    int rc = ab_launch_status();
    if (rc) return rc;
    const int quads = D * (width / 4);
    ab_launch(piece_scan_kernel<CHANNEL, WITH_N>, dim3((quads + 255) / 256, a.H, a.n_seqs), dim3(256), 0, stream, a, D);
    rc = ab_launch_status();
    if (rc) return rc;
  }
  ab_launch(piece_walk_kernel<J, CHANNEL, WITH_N>, dim3(tiles, a.H, a.items), block, walk_smem, stream, a);
  return ab_launch_status();
}

template <bool CHANNEL, bool WITH_N>
static int piece_walk(const PieceArgs& a, int D, cudaStream_t stream) {
  if (!piece_walk_takes(D, a.V) || a.length < 1 || a.length % PW_TOKENS || a.H > 65535 || a.n_seqs > 65535 || a.items < 1 ||
      a.items > 65535 || a.kept < 0 || (a.kept > 0 && (!a.local || !a.prod)))
    return AB_BAD_ARG;
  switch (D / 32) {
    case 1: return piece_walk_go<1, CHANNEL, WITH_N>(a, stream);
    case 2: return piece_walk_go<2, CHANNEL, WITH_N>(a, stream);
    case 3: return piece_walk_go<3, CHANNEL, WITH_N>(a, stream);
    case 4: return piece_walk_go<4, CHANNEL, WITH_N>(a, stream);
    case 6: return piece_walk_go<6, CHANNEL, WITH_N>(a, stream);
    default: return piece_walk_go<8, CHANNEL, WITH_N>(a, stream);
  }
}
