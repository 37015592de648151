// The recurrences of delta_rule.cu over prompt portions, sixteen tokens at a time.
//
// Walked token by token, a sequence is one chain of dependent steps (480 clocks a token for the delta rule at heads of 128). Over a
// chunk of C tokens with the state S before it, G_t the product of the chunk's decays up to token t (per key channel or per head):
//
//     o_t = S^T (G_t q_t) + sum_{j <= t} B_tj u_j,      B_tj = (G_t / G_j k_j) . q_t
//     S  <- diag(G_C) S + sum_j (G_C / G_j k_j) u_j^T
//     u_j = beta_j v_j,  or with the delta rule  u = U - W S,  U = T V,  W = T (G k),  T = (I + diag(beta) A)^-1 diag(beta),
//           A_tj = (G_t / G_j k_j) . k_t for j < t, else 0;  then  o_t = S^T (G_t q_t - (B W)_t) + (B U)_t
//
// Everything but the three products with S is the same whatever S is and goes ahead, every chunk and head on its own (the prep
// kernels, which leave sum_j B_tj u_j, or B U, in the output). The quotients G_t / G_j are running products of decays, so nothing is
// divided by a number that may have gone to zero. The walk then has one dependent step a chunk. All of it is float32 on the
// FFMA pipe, as before.
#include <math.h>

#include "common.cuh"
#include "delta_state.cuh"

namespace tie {

constexpr int kChunk = 16;
constexpr int kChunkCols = 16;       // columns of S a block of the walk holds, four a warp

// Chunks of all sequences are numbered without knowing the sequences' lengths on the host: sequence s starts at
// query_start[s] / 16 + s, which leaves room for a part-filled chunk a sequence.
__device__ __forceinline__ int chunk_base(const int* query_start, int s) { return query_start[s] / kChunk + s; }

struct ChunkPlace {
  int t0, cn;      // first row of the chunk in the step, tokens in it (0: nobody's)
};

__device__ __forceinline__ ChunkPlace find_chunk(const int* __restrict__ query_start, int seqs, int number) {
  int lo = 0, hi = seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (chunk_base(query_start, mid) <= number) lo = mid;
    else hi = mid - 1;
  }
  const int first = query_start[lo] + (number - chunk_base(query_start, lo)) * kChunk;
  return ChunkPlace{first, max(0, min(kChunk, query_start[lo + 1] - first))};
}

template <int CH>
__device__ __forceinline__ void load_channels(const float* p, float (&v)[CH]) {
  if constexpr (CH == 4) {
    load4(p, v);
  } else {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x, v[1] = t.y;
  }
}
template <int CH>
__device__ __forceinline__ void store_channels(float* p, const float (&v)[CH]) {
  if constexpr (CH == 4) store4(p, v);
  else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

// What a block of the prep kernels does with its chunk's u [16][vdim] and weights [16][16]: out row `row` = sum over j <= row.
__device__ __forceinline__ void weighted_rows(const float* __restrict__ weights, const float* __restrict__ u, int vdim, int row, int lane,
                                              float* __restrict__ out) {
  for (int c = lane * 4; c < vdim; c += 128) {
    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
    for (int j = 0; j <= row; ++j) {
      const float f = weights[row * kChunk + j];
      float x[4];
      load4(u + j * vdim + c, x);
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = fmaf(f, x[e], o[e]);
    }
    store4(out + c, o);
  }
}

// Sums over the warp of 4 * KINDS values a lane; lane 4 i (+ 16 of the second kind) ends up with value i.
template <int KINDS>
__device__ __forceinline__ float sums_by_fours(float (&v)[4 * KINDS], int lane) {
  if constexpr (KINDS == 2) {
    const bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float give = up ? v[i] : v[4 + i], keep = up ? v[4 + i] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
  }
#pragma unroll
  for (int half = 2; half > 0; half >>= 1) {
    const bool up = lane & (4 * half);
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float give = up ? v[i] : v[half + i], keep = up ? v[half + i] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * half);
    }
  }
  float s = v[0];
  if constexpr (KINDS == 1) s += __shfl_xor_sync(0xffffffffu, s, 16);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

// Decays per key channel. One block per (chunk, head), a warp for tokens w and 15 - w (so that all have as many pairs to work on), CH =
// dim / 32 channels a lane. Writes the rows that the walk multiplies with the state: q_out (G_t q_t, less (B W)_t with the delta rule; may
// be q itself where every head has its own), k_out (G_C / G_j k_j; over the decays with the delta rule, over k without), w_out (W, delta
// rule), v (in place: U, delta rule), out, and per chunk and head G_C. Bound by issue slots.
template <int CH, bool DELTA>
__global__ void __launch_bounds__(256) chunk_prep_channel_kernel(const float* q, const float* k, float* v, const float* __restrict__ beta,
                                                                const float* decay, long long decay_stride,
                                                                const int* __restrict__ query_start, int seqs, DeltaShape sh, float* q_out,
                                                                float* k_out, long long k_out_stride, float* __restrict__ w_out,
                                                                float* __restrict__ gc_out, float* __restrict__ out) {
  pdl_sync();
  constexpr int DIM = 32 * CH, KINDS = DELTA ? 2 : 1;
  extern __shared__ __align__(16) float smem[];
  const int vdim = sh.vdim, nv = sh.heads * vdim;
  float* const qs = smem;                            // [16][DIM]
  float* const gs = qs + kChunk * DIM;               // decays
  float* const gp = gs + kChunk * DIM;               // their products G
  float* const bs = gp + kChunk * DIM;               // [16][16] B
  float* const vs = bs + kChunk * kChunk;            // [16][vdim] u, or V
  float* const ks = vs + kChunk * vdim;              // delta rule only, like what follows: [16][DIM], then W
  float* const as = ks + kChunk * DIM;               // [16][16] A
  float* const ts = as + kChunk * kChunk;            // [16][16] T
  float* const us = ts + kChunk * kChunk;            // [16][vdim] U
  const ChunkPlace at = find_chunk(query_start, seqs, blockIdx.x);
  if (at.cn == 0) return;
  const int h = blockIdx.y, g = h / (sh.heads / sh.kv_heads), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long qk_stride = static_cast<long long>(sh.kv_heads) * DIM;
  float keys[2][CH];
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int me = n ? kChunk - 1 - warp : warp;
    const long long t = at.t0 + me;
    float x[CH] = {}, gg[CH];
#pragma unroll
    for (int e = 0; e < CH; ++e) gg[e] = 1.0f, keys[n][e] = 0.0f;
    if (me < at.cn) {
      load_channels<CH>(k + t * qk_stride + g * DIM + lane * CH, keys[n]);
      load_channels<CH>(q + t * qk_stride + g * DIM + lane * CH, x);
      load_channels<CH>(decay + t * decay_stride + h * DIM + lane * CH, gg);
      const float f = !DELTA && beta ? beta[t * sh.heads + h] : 1.0f;
      for (int c = lane * 4; c < vdim; c += 128) {
        float u[4];
        load4(v + t * nv + h * vdim + c, u);
#pragma unroll
        for (int e = 0; e < 4; ++e) u[e] *= f;
        store4(vs + me * vdim + c, u);
      }
    }
    if (DELTA) store_channels<CH>(ks + me * DIM + lane * CH, keys[n]);
    store_channels<CH>(qs + me * DIM + lane * CH, x);
    store_channels<CH>(gs + me * DIM + lane * CH, gg);
  }
  __syncthreads();
  if (threadIdx.x < DIM) {
    float run = 1.0f;
#pragma unroll
    for (int i = 0; i < kChunk; ++i) {
      run *= gs[i * DIM + threadIdx.x];
      gp[i * DIM + threadIdx.x] = run;
    }
    gc_out[(static_cast<long long>(blockIdx.x) * sh.heads + h) * DIM + threadIdx.x] = run;
  }
  // a token's key, decayed on to every later token: its column of A and of B, and at the end its row of the update
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int me = n ? kChunk - 1 - warp : warp;
    float (&r)[CH] = keys[n];
    for (int block = me >> 2; block < 4; ++block) {
      float pair[4 * KINDS];
#pragma unroll
      for (int e4 = 0; e4 < 4; ++e4) {
        const int i = block * 4 + e4;
        float x[CH];
        if (i > me) {
          load_channels<CH>(gs + i * DIM + lane * CH, x);
#pragma unroll
          for (int e = 0; e < CH; ++e) r[e] *= x[e];
        }
        load_channels<CH>(qs + i * DIM + lane * CH, x);
        float d = 0.0f;
#pragma unroll
        for (int e = 0; e < CH; ++e) d = fmaf(x[e], r[e], d);
        pair[e4] = d;
        if (DELTA) {
          load_channels<CH>(ks + i * DIM + lane * CH, x);
          d = 0.0f;
#pragma unroll
          for (int e = 0; e < CH; ++e) d = fmaf(x[e], r[e], d);
          pair[4 * KINDS - 4 + e4] = d;
        }
      }
      const float s = sums_by_fours<KINDS>(pair, lane);        // (of tokens ahead of `me` too, which nobody reads)
      const int i = block * 4 + ((lane >> 2) & 3);
      if ((lane & 3) == 0 && (DELTA || lane < 16)) (DELTA && lane >= 16 ? as : bs)[i * kChunk + me] = s;
    }
    if (me < at.cn) store_channels<CH>(k_out + (at.t0 + me) * k_out_stride + h * DIM + lane * CH, r);
  }
  __syncthreads();
  if (DELTA) {
    // T, a column a lane: beta_j down from the diagonal, each row from the ones above it
    if (warp == 0 && lane < kChunk) {
      float x[kChunk];
#pragma unroll
      for (int i = 0; i < kChunk; ++i) {
        const float bt = i < at.cn ? beta[(at.t0 + i) * static_cast<long long>(sh.heads) + h] : 0.0f;
        float s[2] = {0.0f, 0.0f};
#pragma unroll
        for (int j4 = 0; j4 < i; j4 += 4) {
          float row[4];
          load4(as + i * kChunk + j4, row);
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (j4 + e < i) s[e & 1] = fmaf(row[e], x[j4 + e], s[e & 1]);
        }
        x[i] = i < lane ? 0.0f : (i == lane ? bt : -bt * (s[0] + s[1]));
        ts[i * kChunk + lane] = x[i];
      }
    }
    __syncthreads();
    float w[2][CH];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int me = n ? kChunk - 1 - warp : warp;
#pragma unroll
      for (int e = 0; e < CH; ++e) w[n][e] = 0.0f;
      if (me >= at.cn) continue;
      for (int j = 0; j <= me; ++j) {
        const float f = ts[me * kChunk + j];
        float x[CH], y[CH];
        load_channels<CH>(ks + j * DIM + lane * CH, x);
        load_channels<CH>(gp + j * DIM + lane * CH, y);
#pragma unroll
        for (int e = 0; e < CH; ++e) w[n][e] = fmaf(f, x[e] * y[e], w[n][e]);
      }
      store_channels<CH>(w_out + (at.t0 + me) * sh.heads * DIM + h * DIM + lane * CH, w[n]);
      weighted_rows(ts, vs, vdim, me, lane, us + me * vdim);
    }
    __syncthreads();                                 // everyone has read the keys
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int me = n ? kChunk - 1 - warp : warp;
      store_channels<CH>(ks + me * DIM + lane * CH, w[n]);
      if (me < at.cn)
        for (int c = lane * 4; c < vdim; c += 128) {
          float u[4];
          load4(us + me * vdim + c, u);
          store4(v + (at.t0 + me) * nv + h * vdim + c, u);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int me = n ? kChunk - 1 - warp : warp;
    if (me >= at.cn) continue;
    const long long t = at.t0 + me;
    float x[CH], y[CH];
    load_channels<CH>(qs + me * DIM + lane * CH, x);
    load_channels<CH>(gp + me * DIM + lane * CH, y);
#pragma unroll
    for (int e = 0; e < CH; ++e) x[e] *= y[e];
    if (DELTA)
      for (int j = 0; j <= me; ++j) {
        const float f = bs[me * kChunk + j];
        load_channels<CH>(ks + j * DIM + lane * CH, y);
#pragma unroll
        for (int e = 0; e < CH; ++e) x[e] = fmaf(-f, y[e], x[e]);
      }
    store_channels<CH>(q_out + t * sh.heads * DIM + h * DIM + lane * CH, x);
    weighted_rows(bs, DELTA ? us : vs, vdim, me, lane, out + t * nv + h * vdim);
  }
}

// One decay a token and head, the rows q and k shared by the heads of a group: k . q of all pairs, the products of decays before and
// behind every token (gc_out: [16] G_t, [16] G_C / G_t), and the outputs as above. One block per (chunk, head), a warp two tokens.
template <int CH>
__global__ void __launch_bounds__(256) chunk_prep_scalar_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                               const float* __restrict__ v, const float* __restrict__ beta,
                                                               const float* __restrict__ decay, long long decay_stride,
                                                               const int* __restrict__ query_start, int seqs, DeltaShape sh,
                                                               float* __restrict__ gc_out, float* __restrict__ out) {
  pdl_sync();
  constexpr int DIM = 32 * CH;
  extern __shared__ __align__(16) float smem[];
  float* const qs = smem;                            // [16][DIM]
  float* const bs = qs + kChunk * DIM;               // [16][16]
  float* const gs = bs + kChunk * kChunk;            // [16]
  float* const vs = gs + kChunk;                     // [16][vdim] u
  const ChunkPlace at = find_chunk(query_start, seqs, blockIdx.x);
  if (at.cn == 0) return;
  const int h = blockIdx.y, g = h / (sh.heads / sh.kv_heads), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vdim = sh.vdim, nv = sh.heads * vdim;
  const long long stride = static_cast<long long>(sh.kv_heads) * DIM;
  float keys[2][CH];
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int me = n ? kChunk - 1 - warp : warp;
    const long long t = at.t0 + me;
    const bool live = me < at.cn;
    float x[CH] = {};
#pragma unroll
    for (int e = 0; e < CH; ++e) keys[n][e] = 0.0f;
    if (live) {
      load_channels<CH>(k + t * stride + g * DIM + lane * CH, keys[n]);
      load_channels<CH>(q + t * stride + g * DIM + lane * CH, x);
      const float f = beta ? beta[t * sh.heads + h] : 1.0f;
      for (int c = lane * 4; c < vdim; c += 128) {
        float u[4];
        load4(v + t * nv + h * vdim + c, u);
#pragma unroll
        for (int e = 0; e < 4; ++e) u[e] *= f;
        store4(vs + me * vdim + c, u);
      }
    }
    store_channels<CH>(qs + me * DIM + lane * CH, x);
    if (lane == 0) gs[me] = live ? decay[t * decay_stride + h] : 1.0f;
  }
  __syncthreads();
  const long long place = static_cast<long long>(blockIdx.x) * sh.heads + h;
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int me = n ? kChunk - 1 - warp : warp;
    // lane 4 i' holds the decay from this token on to token block * 4 + i'
    float between = 1.0f;
    for (int block = me >> 2; block < 4; ++block) {
      float pair[4];
#pragma unroll
      for (int e4 = 0; e4 < 4; ++e4) {
        float x[CH], d = 0.0f;
        load_channels<CH>(qs + (block * 4 + e4) * DIM + lane * CH, x);
#pragma unroll
        for (int e = 0; e < CH; ++e) d = fmaf(x[e], keys[n][e], d);
        pair[e4] = d;
      }
      const float s = sums_by_fours<1>(pair, lane);
      float here = between;
#pragma unroll
      for (int e4 = 0; e4 < 4; ++e4) {
        const int i = block * 4 + e4;
        if (i > me) between *= gs[i];
        if (e4 == ((lane >> 2) & 3)) here = between;
      }
      if ((lane & 3) == 0 && lane < 16) bs[(block * 4 + (lane >> 2)) * kChunk + me] = s * here;
    }
    if (lane == 0) {
      float before = 1.0f;
      for (int i = 0; i <= me; ++i) before *= gs[i];
      gc_out[place * 2 * kChunk + me] = before;
      gc_out[place * 2 * kChunk + kChunk + me] = between;
    }
  }
  __syncthreads();
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int me = n ? kChunk - 1 - warp : warp;
    if (me < at.cn) weighted_rows(bs, vs, vdim, me, lane, out + (at.t0 + me) * static_cast<long long>(nv) + h * vdim);
  }
}

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  return static_cast<unsigned long long>(__float_as_uint(lo)) | static_cast<unsigned long long>(__float_as_uint(hi)) << 32;
}
__device__ __forceinline__ float low(unsigned long long v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float high(unsigned long long v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
__device__ __forceinline__ unsigned long long mul2(unsigned long long x, unsigned long long y) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long x, unsigned long long y, unsigned long long z) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
  return r;
}

struct ChunkWalk {
  const float* w;               // [T, heads * dim] (delta rule)
  const float* q;               // row strides, and whether a head's rows are its key head's (one decay a head) or its own
  const float* k;
  const float* v;               // [T, heads * vdim]: U, or the values
  const float* beta;            // [T, heads] or null (without the delta rule)
  const float* gc;              // [chunks, heads, dim] or [chunks, heads, 32]
  float* state;
  float* out;                   // holds what the chunk's own tokens add to the outputs
  const int* query_start;
  const int* state_slots;
  long long q_stride, k_stride, state_stride, conv_state_off;
  int by_key_head;
};

// One block per (sequence, head, 16 columns of S), a warp per four columns, with the delta rule two: one multiplies W with the state, the
// other q, each with a state of its own that both keep up. A lane holds CH = dim / 32 key channels of the warp's columns; a
// chunk's rows come through two buffers in shared memory (cp.async), the next chunk's while this one is worked on. The products
// with S leave 32 partial sums a lane for eight tokens, which the lanes sum up in 31 exchanges, each halving what a lane still holds.
// So that a lane need not choose what it gives away, it numbers the tokens by exclusive or with bits of its own number: what it
// keeps is the first half (the columns, which all lanes must number alike for the update, are chosen in the last two rounds).
// What bounds it is latency: one or two warps a scheduler, loads and exchanges in a row. (Two columns and twice the warps: the same
// time for one sequence, a tenth more for several.)
template <typename T, int CH, bool DELTA, bool SCALAR>
__global__ void __launch_bounds__(DELTA ? 256 : 128) chunk_walk_kernel(ChunkWalk a, const T* __restrict__ proj, long long proj_stride, int q_off,
                                                                      int k_off, int v_off, DeltaShape sh) {
  pdl_wait();      // started when the kernels ahead have drained: few blocks, long-running (see delta_rule.cu)
  constexpr int DIM = 32 * CH, PAIRS = CH / 2, LD = kChunkCols + 4, THREADS = DELTA ? 256 : 128;
  constexpr int GC = SCALAR ? 2 * kChunk : DIM;
  constexpr int W_AT = 0, Q_AT = W_AT + (DELTA ? kChunk * DIM : 0), K_AT = Q_AT + kChunk * DIM, V_AT = K_AT + kChunk * DIM,
                O_AT = V_AT + kChunk * LD, GC_AT = O_AT + kChunk * LD, BETA_AT = GC_AT + GC, STAGE = BETA_AT + kChunk;
  extern __shared__ __align__(16) float smem[];
  const int s = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * kChunkCols;
  const int slot = a.state_slots[s];
  if (slot < 0) return;
  const int q0 = a.query_start[s], n = a.query_start[s + 1] - q0, base = chunk_base(a.query_start, s);
  const int t0 = n > 0 ? q0 : 0;             // (a sequence without tokens: some row of the step, of which nothing is read)
  const int vdim = sh.vdim, nv = sh.heads * vdim;
  const int tid = threadIdx.x, warp = (tid >> 5) & 3, lane = tid & 31;
  const bool corrects = DELTA && tid < 128;      // the warps that multiply with W
  const int hq = a.by_key_head ? h / (sh.heads / sh.kv_heads) : h;
  float* const us = smem + 2 * STAGE + warp * 128;      // [16][4] pairs (u, u)
  float* const S = a.state + slot * a.state_stride + static_cast<long long>(h) * DIM * vdim;

  auto fetch = [&](int c, float* stage) {
    const int cn = min(kChunk, n - c * kChunk);
    const long long t = t0 + c * kChunk, place = static_cast<long long>(base + c) * sh.heads + h;
    auto copy16 = [](float* dst, const float* src, bool there) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(there ? 16 : 0) : "memory");
    };
    constexpr int PIECES = DIM / 4;
#pragma unroll 4
    for (int i = tid; i < kChunk * PIECES; i += THREADS) {
      const int r = i / PIECES, d = (i % PIECES) * 4;
      const long long row = r < cn ? t + r : t;
      if (DELTA) copy16(stage + W_AT + i * 4, a.w + row * sh.heads * DIM + h * DIM + d, r < cn);
      copy16(stage + Q_AT + i * 4, a.q + row * a.q_stride + hq * DIM + d, r < cn);
      copy16(stage + K_AT + i * 4, a.k + row * a.k_stride + hq * DIM + d, r < cn);
    }
    if (tid < 128) {
      const int r = (tid & 63) / 4, piece = tid & 3, col = col0 + piece * 4;
      const bool there = r < cn && col < vdim;
      copy16(stage + (tid < 64 ? V_AT : O_AT) + r * LD + piece * 4, (tid < 64 ? a.v : a.out) + (there ? (t + r) * nv + h * vdim + col : 0), there);
    }
    if (tid < GC / 4) copy16(stage + GC_AT + tid * 4, a.gc + place * GC + tid * 4, true);
    if (!DELTA && tid >= 64 && tid < 64 + kChunk) {
      const int r = tid - 64;
      stage[BETA_AT + r] = r < cn && a.beta ? a.beta[(t + r) * sh.heads + h] : 1.0f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // The block's columns of S come in through shared memory, in row pieces of 64 bytes.
  constexpr int PAD = kChunkCols + 1;
  float* const tile = smem + STAGE;      // the second buffer, not in use yet
  for (int i = tid; i < DIM * (kChunkCols / 4); i += THREADS) {
    const int r = i / (kChunkCols / 4), c = (i % (kChunkCols / 4)) * 4;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (col0 + c < vdim) load4(S + static_cast<long long>(r) * vdim + col0 + c, v);
#pragma unroll
    for (int e = 0; e < 4; ++e) tile[r * PAD + c + e] = v[e];
  }
  fetch(0, smem);
  __syncthreads();
  const int mine_tok = lane >> 2, mine_col = lane & 3;
  unsigned long long st[4][PAIRS];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int p = 0; p < PAIRS; ++p) {
      const float* x = tile + (lane * CH + 2 * p) * PAD + warp * 4 + c;
      st[c][p] = pack2(x[0], x[PAD]);
    }
  auto channels = [](const float* row, unsigned long long (&x)[PAIRS]) {
    if constexpr (CH == 4) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(row);
      x[0] = v.x, x[1] = v.y;
    } else {
      x[0] = *reinterpret_cast<const unsigned long long*>(row);
    }
  };

  const int chunks = (n + kChunk - 1) / kChunk;
  for (int c = 0; c < chunks; ++c) {
    const float* const stage = smem + (c & 1) * STAGE;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                          // this chunk is there, and everyone is through with the other buffer
    if (c + 1 < chunks) fetch(c + 1, smem + ((c + 1) & 1) * STAGE);
    // All the sums before anything is written: the two groups' loads and exchanges can then overlap.
    float sums[2];
    const float* const rows = stage + (corrects ? W_AT : Q_AT) + lane * CH;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      float part[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        unsigned long long x[PAIRS];
        channels(rows + (g * 8 + (i ^ mine_tok)) * DIM, x);
#pragma unroll
        for (int col = 0; col < 4; ++col) {
          unsigned long long d = mul2(x[0], st[col][0]);
#pragma unroll
          for (int p = 1; p < PAIRS; ++p) d = fma2(x[p], st[col][p], d);
          part[i * 4 + col] = low(d) + high(d);
        }
      }
#pragma unroll
      for (int half = 16; half > 2; half >>= 1)
#pragma unroll
        for (int i = 0; i < half; ++i) part[i] += __shfl_xor_sync(0xffffffffu, part[i + half], half);
#pragma unroll
      for (int half = 2; half > 0; half >>= 1) {
        const bool up = lane & half;
#pragma unroll
        for (int i = 0; i < half; ++i) {
          const float give = up ? part[i] : part[i + half], keep = up ? part[i + half] : part[i];
          part[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
      }
      sums[g] = part[0];
    }
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const int t = g * 8 + mine_tok, row = c * kChunk + t, at = t * LD + warp * 4 + mine_col;
      if (!DELTA || corrects) {
        const float u = DELTA ? stage[V_AT + at] - sums[g] : stage[V_AT + at] * stage[BETA_AT + t] * (SCALAR ? stage[GC_AT + kChunk + t] : 1.0f);
        *reinterpret_cast<float2*>(us + (t * 4 + mine_col) * 2) = make_float2(u, u);
      }
      if (!corrects && row < n && col0 + warp * 4 + mine_col < vdim)
        a.out[(t0 + row) * static_cast<long long>(nv) + h * vdim + col0 + warp * 4 + mine_col] =
            SCALAR ? fmaf(sums[g], stage[GC_AT + t], stage[O_AT + at]) : sums[g] + stage[O_AT + at];
    }
    if (DELTA) asm volatile("bar.sync %0, 64;" ::"r"(warp + 1) : "memory");      // the two warps of these columns
    else __syncwarp();
    // the state past this chunk
#pragma unroll
    for (int p = 0; p < PAIRS; ++p) {
      const float* d = stage + GC_AT + (SCALAR ? kChunk - 1 : lane * CH + 2 * p);
      const unsigned long long keep = pack2(d[0], SCALAR ? d[0] : d[1]);
#pragma unroll
      for (int col = 0; col < 4; ++col) st[col][p] = mul2(st[col][p], keep);
    }
#pragma unroll
    for (int t = 0; t < kChunk; ++t) {
      unsigned long long x[PAIRS];
      channels(stage + K_AT + t * DIM + lane * CH, x);
      const ulonglong2 u01 = *reinterpret_cast<const ulonglong2*>(us + t * 8), u23 = *reinterpret_cast<const ulonglong2*>(us + t * 8 + 4);
#pragma unroll
      for (int p = 0; p < PAIRS; ++p) {
        st[0][p] = fma2(x[p], u01.x, st[0][p]);
        st[1][p] = fma2(x[p], u01.y, st[1][p]);
        st[2][p] = fma2(x[p], u23.x, st[2][p]);
        st[3][p] = fma2(x[p], u23.y, st[3][p]);
      }
    }
    __syncwarp();                             // the warp's u is written again by the next chunk
  }
  pdl_launch_dependents();
  // A sequence without tokens has not waited for its first buffer, which the state goes out through. (Leaving at once for such sequences
  // made the walk over the others' chunks slower: 2,048 tokens with one decay a head 241.6 us against 229.2.)
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (!corrects) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int p = 0; p < PAIRS; ++p) {
        float* x = smem + (lane * CH + 2 * p) * PAD + warp * 4 + c;
        x[0] = low(st[c][p]), x[PAD] = high(st[c][p]);
      }
  }
  __syncthreads();
  for (int i = tid; i < DIM * (kChunkCols / 4); i += THREADS) {
    const int r = i / (kChunkCols / 4), c = (i % (kChunkCols / 4)) * 4;
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = smem[r * PAD + c + e];
    if (col0 + c < vdim) store4(S + static_cast<long long>(r) * vdim + col0 + c, v);
  }
  move_conv_tail(sh, a.state + slot * a.state_stride + a.conv_state_off, proj, proj_stride, q_off, k_off, v_off, t0, n,
                 blockIdx.y * gridDim.z + blockIdx.z, gridDim.y * gridDim.z);
}

// What the chunked kernels take. dim: 64 or 128 key channels a head.
inline bool chunked_takes(int heads, int kv_heads, int dim, int vdim, int plain, int decay_per_head, long long decay_stride,
                          long long state_stride, const void* const* ptrs, int n) {
  if (dim != 64 && dim != 128) return false;
  if (vdim % 4 != 0 || vdim > 256 || state_stride % 4 != 0 || heads > 65535) return false;
  if (decay_per_head ? !plain : (decay_stride % 4 != 0 || (plain && heads != kv_heads))) return false;
  for (int i = 0; i < n; ++i)
    if (reinterpret_cast<uintptr_t>(ptrs[i]) % 16 != 0) return false;
  return true;
}

template <int CH>
int launch_chunk_prep(const float* q, const float* k, float* v, const float* beta, float* decay, long long decay_stride,
                      const int* query_start, int seqs, int tokens, const DeltaShape& sh, int plain, int decay_per_head, float* q_out,
                      float* w_out, float* gc_out, float* out, cudaStream_t s) {
  const dim3 grid(tokens / kChunk + seqs, sh.heads);
  constexpr int DIM = 32 * CH;
  const size_t rows = kChunk * DIM * sizeof(float), pairs = kChunk * kChunk * sizeof(float), values = kChunk * sh.vdim * sizeof(float);
  const size_t smem = decay_per_head ? rows + pairs + kChunk * sizeof(float) + values : plain ? 3 * rows + pairs + values : 4 * rows + 3 * pairs + 2 * values;
  const long long own = static_cast<long long>(sh.heads) * DIM;
  auto ready = [&](auto kernel) {
    return smem <= 48 * 1024 || cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) == cudaSuccess;
  };
  bool ok = true;
  if (decay_per_head) {
    if ((ok = ready(chunk_prep_scalar_kernel<CH>)))
      TIE_LAUNCH((chunk_prep_scalar_kernel<CH>), grid, 256, smem, s, q, k, v, beta, decay, decay_stride, query_start, seqs, sh, gc_out, out);
  } else if (plain) {
    if ((ok = ready(chunk_prep_channel_kernel<CH, false>)))
      TIE_LAUNCH((chunk_prep_channel_kernel<CH, false>), grid, 256, smem, s, q, k, v, beta, decay, decay_stride, query_start, seqs, sh,
                 const_cast<float*>(q), const_cast<float*>(k), own, nullptr, gc_out, out);
  } else {
    if ((ok = ready(chunk_prep_channel_kernel<CH, true>)))
      TIE_LAUNCH((chunk_prep_channel_kernel<CH, true>), grid, 256, smem, s, q, k, v, beta, decay, decay_stride, query_start, seqs, sh, q_out,
                 decay, decay_stride, w_out, gc_out, out);
  }
  if (!ok) {
    set_error("delta_chunk: cannot reserve %zu bytes of shared memory", smem);
    return kCudaError;
  }
  TIE_RETURN_LAUNCH("delta_chunk_prep");
}

template <typename T, int CH, bool DELTA, bool SCALAR>
int launch_chunk_walk(const ChunkWalk& a, const void* proj, long long proj_stride, int q_off, int k_off, int v_off, int seqs, const DeltaShape& sh,
                      cudaStream_t s) {
  constexpr int DIM = 32 * CH, stage = (DELTA ? 3 : 2) * kChunk * DIM + 2 * kChunk * (kChunkCols + 4) + (SCALAR ? 2 * kChunk : DIM) + kChunk;
  constexpr int smem = (2 * stage + 4 * 128) * static_cast<int>(sizeof(float));
  auto kernel = chunk_walk_kernel<T, CH, DELTA, SCALAR>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    set_error("delta_chunk: cannot reserve %d bytes of shared memory", smem);
    return kCudaError;
  }
  launch_kernel_alone(kernel, dim3(seqs, sh.heads, ceil_div(sh.vdim, kChunkCols)), dim3(DELTA ? 256 : 128), smem, s, a, static_cast<const T*>(proj), proj_stride,
                      q_off, k_off, v_off, sh);
  TIE_RETURN_LAUNCH("delta_chunk_walk");
}

}  // namespace tie

using namespace tie;

TIE_API int tie_delta_chunk_takes(int heads, int kv_heads, int dim, int vdim, int plain, int decay_per_head, long long decay_stride,
                                  long long state_stride, const void* q, const void* k, const void* v, const void* decay, const void* state,
                                  const void* out, const void* scratch) {
  const void* ptrs[] = {q, k, v, state, out, scratch, decay_per_head ? nullptr : decay};
  return chunked_takes(heads, kv_heads, dim, vdim, plain, decay_per_head, decay_stride, state_stride, ptrs, 7) ? 1 : 0;
}

// Floats of scratch for `tokens` tokens of `seqs` sequences: the decays over every chunk of a head, and for the delta rule W and what the
// queries become.
TIE_API long long tie_delta_chunk_scratch(int tokens, int seqs, int heads, int dim, int plain) {
  const long long numbers = tokens / kChunk + seqs;
  return numbers * heads * (dim > 2 * kChunk ? dim : 2 * kChunk) + (plain ? 0 : 2ll * tokens * heads * dim);
}

// tie_delta_rule for steps with portions, in chunks. Overwritten are v and decay (delta rule), q and k (plain, a decay a channel), nothing with a
// decay a head: callers rely on it.
TIE_API int tie_delta_rule_chunked(int dtype, float* qn, float* kn, float* vn, const float* beta, float* decay, long long decay_stride,
                                   float* state, long long state_stride, long long conv_state_off, const void* proj, long long proj_stride,
                                   int q_off, int k_off, int v_off, const int* query_start, const int* state_slots, int seqs, int tokens,
                                   int heads, int kv_heads, int dim, int vdim, int taps, float* out, int plain, int decay_per_head,
                                   float* scratch, cudaStream_t s) {
  const DeltaShape sh{heads, kv_heads, dim, vdim, taps};
  TIE_REQUIRE(heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && taps >= 1 && taps <= 16, "delta rule: bad shape heads=%d/%d taps=%d", heads,
              kv_heads, taps);
  TIE_REQUIRE(tie_delta_chunk_takes(heads, kv_heads, dim, vdim, plain, decay_per_head, decay_stride, state_stride, qn, kn, vn, decay, state, out,
                                    scratch),
              "delta rule in chunks: sizes or addresses it does not take (dim=%d vdim=%d)", dim, vdim);
  TIE_REQUIRE(beta != nullptr || plain, "delta_rule: the delta rule needs beta");
  TIE_REQUIRE(dtype == TIE_F32 || dtype == TIE_BF16, "unknown dtype code %d", dtype);
  if (seqs <= 0 || tokens <= 0) return kOk;
  const long long numbers = tokens / kChunk + seqs;
  float* const gc = scratch;
  float* const w = gc + numbers * heads * (dim > 2 * kChunk ? dim : 2 * kChunk);
  float* const decayed_q = w + static_cast<long long>(tokens) * heads * dim;
  const int st = dim == 128 ? launch_chunk_prep<4>(qn, kn, vn, beta, decay, decay_stride, query_start, seqs, tokens, sh, plain, decay_per_head,
                                                   decayed_q, w, gc, out, s)
                            : launch_chunk_prep<2>(qn, kn, vn, beta, decay, decay_stride, query_start, seqs, tokens, sh, plain, decay_per_head,
                                                   decayed_q, w, gc, out, s);
  if (st != kOk) return st;
  const long long own = static_cast<long long>(heads) * dim, shared = static_cast<long long>(kv_heads) * dim;
  ChunkWalk a{w, decay_per_head || plain ? qn : decayed_q, decay_per_head || plain ? kn : decay, vn, plain ? beta : nullptr, gc, state, out,
              query_start, state_slots, decay_per_head ? shared : own, decay_per_head ? shared : (plain ? own : decay_stride), state_stride,
              conv_state_off, decay_per_head};
#define TIE_WALK(T, CH)                                                                                                    \
  (decay_per_head ? launch_chunk_walk<T, CH, false, true>(a, proj, proj_stride, q_off, k_off, v_off, seqs, sh, s)          \
   : plain        ? launch_chunk_walk<T, CH, false, false>(a, proj, proj_stride, q_off, k_off, v_off, seqs, sh, s)         \
                  : launch_chunk_walk<T, CH, true, false>(a, proj, proj_stride, q_off, k_off, v_off, seqs, sh, s))
  if (dtype == TIE_F32) return dim == 128 ? TIE_WALK(float, 4) : TIE_WALK(float, 2);
  return dim == 128 ? TIE_WALK(__nv_bfloat16, 4) : TIE_WALK(__nv_bfloat16, 2);
#undef TIE_WALK
}
