// Attention of prompt portions on the 5th-generation tensor cores for models whose softmax weights are to keep 16 bits of mantissa: the
// float weights enter the value product as two bfloat16 terms, p = hi + lo, each with an MMA of its own, as in the exact mode of
// attention_prompt.cu. Two kinds of keys and values:
//   pages     heads of 64 or 128, read through the block table like everywhere else;
//   expanded  latent attention (attention_latent.cu) with the cached latents multiplied out: keys of 128 + 64 dimensions, the first
//             part and the value of 128 per head from one product over the gathered latents, the rotated part shared by the heads.
//             Over 2,048 tokens a pair of positions then costs 192 + 2 x 128 multiplications a head instead of 576 + 2 x 512.
//
// The arrangement is that of attention_prompt_umma.cu (two row tiles of 128 a CTA, thread = row softmax, TMA producer, one issuer) with
// two differences. The weights stay in tensor memory: a row's hi and lo terms take exactly the columns of its scores, and the value
// product reads them there as its A operand, so that shared memory feeds K and V only once a tile and Q. And the scores have two
// buffers a row tile, so that Q K^T of the next tile runs before the softmax of this one is through. Tensor memory: 2 x 2 x 64
// columns of scores, 2 x 128 of accumulators.
// What bounds it is the issue of MMAs 64 columns wide (49 clocks each).
#include "attention_mma.cuh"
#include "umma.cuh"

namespace tie {

constexpr int kExactThreads = 320;

struct ExactPromptArgs {
  const __nv_bfloat16* q;
  __nv_bfloat16* out;
  const int* query_start;
  const int* context_lens;
  const int* block_tables;
  int* status;
  const float* sink;      // [q_heads] or null
  long long q_stride;
  int max_blocks, q_heads, kv_heads, page_size, page_shift, window, v_col, rot_col;
  float scale_log2;
  int cta_rows;
};

// Expanded keys lie sequence by sequence, each from its first key that anyone sees, rounded down to a whole tile, to its last, rounded
// up with zeros: no tile holds keys of two sequences.
__device__ __forceinline__ int expanded_first(int context, int queries, int window) {
  return window > 0 ? max(0, context - queries - window + 1) & ~(kKeysPerTile - 1) : 0;
}
__device__ __forceinline__ int expanded_rows(int context, int queries, int window) {
  return (context - expanded_first(context, queries, window) + kKeysPerTile - 1) & ~(kKeysPerTile - 1);
}

template <int KH, int VH, bool PAGED, int STAGES>
__global__ void __launch_bounds__(kExactThreads, 1)
attn_prompt_exact_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                         const __grid_constant__ CUtensorMap r_map, ExactPromptArgs a) {
  pdl_sync();
  constexpr int KD = KH * 64, VD = VH * 64;
  constexpr int HALF = 64 * 128;                  // 64 keys x 64 elements
  constexpr int STAGE_BYTES = (KH + VH) * HALF;
  constexpr int Q_HALF = 128 * 128;               // 128 rows x 64 elements
  constexpr int O_COL = 256;
  constexpr float kRescaleStep = 8.0f;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* q_smem = smem;                         // [row tile][half]
  uint8_t* ring = q_smem + 2 * KH * Q_HALF;
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(ring + STAGES * STAGE_BYTES);
  uint64_t* kv_empty = kv_full + STAGES;
  uint64_t* s_full = kv_empty + STAGES;           // [row tile][buffer]: scores written
  uint64_t* p_full = s_full + 4;                  // weights written, O rescaled
  uint64_t* o_done = p_full + 4;                  // P V retired
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(o_done + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seq = blockIdx.z, kvh = blockIdx.x;
  const int G = a.q_heads / a.kv_heads;
  const int t0 = a.query_start[seq];
  const int nq = a.query_start[seq + 1] - t0;
  const int rows = nq * G;
  const int row0 = (static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y)) * a.cta_rows;   // last rows (most keys) first
  if (row0 >= rows) return;
  const int pos0 = a.context_lens[seq] - nq;

  bool has[2];
  int first[2], last[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int r0 = row0 + 128 * q;
    has[q] = r0 < rows && 128 * q < a.cta_rows;
    const int lo_pos = pos0 + r0 / G, hi_pos = pos0 + min(rows - 1, r0 + 127) / G;
    first[q] = a.window > 0 ? max(0, lo_pos - a.window + 1) / kKeysPerTile : 0;
    last[q] = hi_pos / kKeysPerTile;
  }
  const int kt_first = first[0], kt_last = has[1] ? last[1] : last[0];
  const int n_tiles = kt_last - kt_first + 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(kv_full + s, 1);
      mbar_init(kv_empty + s, 1);
    }
    for (int b = 0; b < 4; ++b) {
      mbar_init(s_full + b, 1);
      mbar_init(p_full + b, 4);
      mbar_init(o_done + b, 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp < 8) {
    // Q: every softmax thread brings its own row (rows beyond the sequence: zeros)
    const int q = warp >> 2, rr = (warp & 3) * 32 + lane;
    const int row = row0 + 128 * q + rr;
    const uint4* src = row < rows ? reinterpret_cast<const uint4*>(a.q + static_cast<long long>(t0 + row / G) * a.q_stride +
                                                                  static_cast<long long>(kvh * G + row % G) * KD)
                                  : nullptr;
#pragma unroll
    for (int c = 0; c < KD / 8; ++c) {
      const uint4 v = src ? src[c] : make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(q_smem + (q * KH + (c >> 3)) * Q_HALF + rr * 128 + (((c & 7) ^ (rr & 7)) << 4)) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 8) {
    // ---- producer
    const int box_rows = PAGED ? min(a.page_size, kKeysPerTile) : kKeysPerTile;
    const int boxes_per_tile = kKeysPerTile / box_rows;
    const int* table = a.block_tables + static_cast<long long>(seq) * a.max_blocks;
    long long base = 0;                           // expanded: row of the sequence's key 0
    if (!PAGED) {
      for (int i = 0; i < seq; ++i) base += expanded_rows(a.context_lens[i], a.query_start[i + 1] - a.query_start[i], a.window);
      base -= expanded_first(a.context_lens[seq], nq, a.window);
    }
    for (int i = 0; i < n_tiles; ++i) {
      const int s = i % STAGES;
      int ok = 1;
      if (lane == 0) {
        ok = mbar_wait(kv_empty + s, ((i / STAGES) & 1) ^ 1, abort_flag, a.status, 11) ? 1 : 0;
        if (ok) mbar_expect_tx(kv_full + s, STAGE_BYTES);
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      if (lane < boxes_per_tile) {
        const int key = (kt_first + i) * kKeysPerTile + lane * box_rows;
        uint8_t* dst = ring + s * STAGE_BYTES + lane * box_rows * 128;
        if (PAGED) {
          const int idx = key >> a.page_shift;
          const int page = idx < a.max_blocks ? table[idx] : 0;   // beyond the table: any real page; those keys are masked
          const int row = (page * a.kv_heads + kvh) * a.page_size + (key & (a.page_size - 1));
#pragma unroll
          for (int h = 0; h < KH; ++h) tma_load_2d(dst + h * HALF, &k_map, h * 64, row, kv_full + s);
#pragma unroll
          for (int h = 0; h < VH; ++h) tma_load_2d(dst + (KH + h) * HALF, &v_map, h * 64, row, kv_full + s);
        } else {
          const int row = static_cast<int>(base + key);
#pragma unroll
          for (int h = 0; h < KH - 1; ++h) tma_load_2d(dst + h * HALF, &k_map, kvh * (KD - 64) + h * 64, row, kv_full + s);
          tma_load_2d(dst + (KH - 1) * HALF, &r_map, a.rot_col, row, kv_full + s);
#pragma unroll
          for (int h = 0; h < VH; ++h) tma_load_2d(dst + (KH + h) * HALF, &v_map, a.v_col + kvh * VD + h * 64, row, kv_full + s);
        }
      }
    }
  } else if (warp == 9) {
    // ---- MMA issuer: the whole warp walks the loop (uniform), one elected lane issues
    constexpr uint32_t idesc_qk = instr_desc(kKeysPerTile);          // 128 x 64, both operands k-major
    constexpr uint32_t idesc_pv = instr_desc(VD) | (1u << 16);       // 128 x VD, B (= V) with its N extent contiguous
    const uint32_t q_lo0 = desc_lo_sw128(smem_u32(q_smem));
    const uint32_t k_lo0 = desc_lo_sw128(smem_u32(ring));
    const uint32_t v_lo0 = desc_lo_sw128(smem_u32(ring + KH * HALF), HALF);   // blocks of 64 value columns lie 64 rows apart
    int n_qk[2] = {0, 0}, n_pv[2] = {0, 0};
    int s_qk = 0, s_pv = 0;
    uint32_t parity_qk = 0;
    bool ok = true;
    // Q K^T of key tile i for both row tiles. A buffer of scores is written again when P V of the tile two before, which reads its
    // weights there, has retired.
    auto scores = [&](int i) {
      ok = ok && __all_sync(0xffffffffu, mbar_wait(kv_full + s_qk, parity_qk, abort_flag, a.status, 12) ? 1 : 0);
      const uint32_t k_lo = k_lo0 + s_qk * (STAGE_BYTES >> 4);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int t = kt_first + i, b = n_qk[q] & 1;
        if (!ok || !(has[q] && t >= first[q] && t <= last[q])) continue;
        if (n_qk[q] >= 2) ok = __all_sync(0xffffffffu, mbar_wait(o_done + q * 2 + b, ((n_qk[q] - 2) >> 1) & 1, abort_flag, a.status, 12) ? 1 : 0);
        if (!ok) continue;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < KD / 16; ++ks)
            umma_bf16(tmem_base + (q * 2 + b) * kKeysPerTile,
                      desc_from_words(q_lo0 + (((q * KH + (ks >> 2)) * Q_HALF + (ks & 3) * 32) >> 4), kDescHiSw128),
                      desc_from_words(k_lo + (((ks >> 2) * HALF + (ks & 3) * 32) >> 4), kDescHiSw128), idesc_qk, ks > 0 ? 1u : 0u);
          umma_commit(s_full + q * 2 + b);
        }
        __syncwarp();
        ++n_qk[q];
      }
      if (++s_qk == STAGES) {
        s_qk = 0;
        parity_qk ^= 1;
      }
    };
    // Per tile: P V of both row tiles, then the scores of the tile after the next. What either waits for is then ready or behind
    // work of the other row tile that the tensor cores still have queued.
    scores(0);
    if (n_tiles > 1) scores(1);
    for (int i = 0; i < n_tiles && ok; ++i) {
      const uint32_t v_lo = v_lo0 + s_pv * (STAGE_BYTES >> 4);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int t = kt_first + i, pb = q * 2 + (n_pv[q] & 1);
        if (!ok || !(has[q] && t >= first[q] && t <= last[q])) continue;
        ok = __all_sync(0xffffffffu, mbar_wait(p_full + pb, (n_pv[q] >> 1) & 1, abort_flag, a.status, 12) ? 1 : 0);
        if (!ok) continue;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          const uint32_t p_tmem = tmem_base + pb * kKeysPerTile;
          const uint32_t keep = n_pv[q] > 0 ? 1u : 0u;
#pragma unroll
          for (int kk = 0; kk < kKeysPerTile / 16; ++kk) {
            const uint64_t vd = desc_from_words(v_lo + ((kk * 16 * 128) >> 4), kDescHiSw128);
            umma_bf16_a_tmem(tmem_base + O_COL + q * VD, p_tmem + kk * 8, vd, idesc_pv, kk > 0 ? 1u : keep);
            umma_bf16_a_tmem(tmem_base + O_COL + q * VD, p_tmem + 32 + kk * 8, vd, idesc_pv, 1u);
          }
          umma_commit(o_done + pb);
        }
        __syncwarp();
        ++n_pv[q];
      }
      if (!ok) break;
      if (elect_one()) umma_commit(kv_empty + s_pv);   // everything that reads the stage has been issued: free when it retires
      __syncwarp();
      if (++s_pv == STAGES) s_pv = 0;
      if (i + 2 < n_tiles) scores(i + 2);
    }
  } else {
    // ---- softmax: warps 0-3 own tile 0, warps 4-7 tile 1; thread = row
    const int q = warp >> 2, wq = warp & 3;
    const int rr = wq * 32 + lane;                           // row inside the tile = lane of tensor memory
    const int row = row0 + 128 * q + rr;
    const int pos = row < rows ? pos0 + row / G : -1;       // rows beyond the sequence see no key
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t o_tmem = tmem_base + lane_base + O_COL + q * VD;
    float m_run = -INFINITY, m_used = -INFINITY, l = 0.0f;
    bool ok = has[q];
    const int my_tiles = has[q] ? last[q] - first[q] + 1 : 0;
    for (int n = 0; n < my_tiles && ok; ++n) {
      const int key0 = (first[q] + n) * kKeysPerTile, b = q * 2 + (n & 1);
      const uint32_t s_tmem = tmem_base + lane_base + b * kKeysPerTile;
      ok = __all_sync(0xffffffffu, mbar_wait(s_full + b, (n >> 1) & 1, abort_flag, a.status, 12) ? 1 : 0) != 0;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t sr[4][16];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld16(s_tmem + 16 * c, sr[c]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");

      const bool full_tile = key0 + 63 <= pos && (a.window <= 0 || key0 > pos - a.window);
      if (!full_tile) {
#pragma unroll
        for (int c = 0; c < 64; ++c) {
          const int key = key0 + c;
          const bool seen = key <= pos && (a.window <= 0 || key > pos - a.window);
          sr[c >> 4][c & 15] = seen ? sr[c >> 4][c & 15] : 0xff800000u;   // -inf
        }
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 64; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], __uint_as_float(sr[c >> 4][c & 15]));
      m_run = fmaxf(m_run, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * a.scale_log2);
      const bool need = m_run > m_used + kRescaleStep;       // also: the first finite maximum of the row
      if (__any_sync(0xffffffffu, need)) {
        float f = 1.0f;
        if (need) {
          f = m_used == -INFINITY ? 1.0f : ex2(m_used - m_run);
          m_used = m_run;
          l *= f;
        }
        if (n > 0) {
          // O may be touched once P V of the tile before has retired
          ok = __all_sync(0xffffffffu, mbar_wait(o_done + 2 * q + ((n - 1) & 1), ((n - 1) >> 1) & 1, abort_flag, a.status, 12) ? 1 : 0) != 0;
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
          for (int c0 = 0; c0 < VD; c0 += 16) {
            uint32_t o[16];
            tmem_ld16(o_tmem + c0, o);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
            tmem_st16(o_tmem + c0, o);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
      }
      const float base = m_used == -INFINITY ? 0.0f : m_used;
      float sum4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      // two keys a column: the weights' first terms over the first 32 columns of the scores, what they leave over the others
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const int c = half * 32 + 2 * e;
          const float p0 = ex2(fmaf(__uint_as_float(sr[c >> 4][c & 15]), a.scale_log2, -base));
          const float p1 = ex2(fmaf(__uint_as_float(sr[c >> 4][(c & 15) + 1]), a.scale_log2, -base));
          sum4[e & 3] += p0 + p1;
          hi[e] = pack_bf16(p0, p1);
          lo[e] = pack_bf16_rest(p0, p1, hi[e]);
        }
        tmem_st16(s_tmem + half * 16, hi);
        tmem_st16(s_tmem + 32 + half * 16, lo);
      }
      l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(p_full + b)) : "memory");
    }
    if (ok && my_tiles > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(o_done + 2 * q + ((my_tiles - 1) & 1), ((my_tiles - 1) >> 1) & 1, abort_flag, a.status, 12) ? 1 : 0) != 0;
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float inv = l > 0.0f ? 1.0f / l : 0.0f;
        const int head = kvh * G + row % G;
        if (a.sink != nullptr && l > 0.0f && row < rows) {       // sums and sink brought to the larger of the two references
          const float sink = a.sink[head] * 1.4426950408889634f, top = fmaxf(m_used, sink), rescale = exp2f(m_used - top);
          inv = rescale / fmaf(l, rescale, exp2f(sink - top));
        }
        __nv_bfloat16* o_row = row < rows ? a.out + (static_cast<long long>(t0 + row / G) * a.q_heads + head) * VD : nullptr;
#pragma unroll 1
        for (int c0 = 0; c0 < VD; c0 += 16) {
          uint32_t o[16];
          tmem_ld16(o_tmem + c0, o);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (o_row) {
            uint32_t w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = pack_bf16(__uint_as_float(o[2 * e]) * inv, __uint_as_float(o[2 * e + 1]) * inv);
            *reinterpret_cast<uint4*>(o_row + c0) = make_uint4(w[0], w[1], w[2], w[3]);
            *reinterpret_cast<uint4*>(o_row + c0 + 8) = make_uint4(w[4], w[5], w[6], w[7]);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag != 0) {   // a wait ran out: let copies and MMAs that are still in flight finish before the CTA goes away
    const unsigned long long t_start = clock64();
    while (clock64() - t_start < 4000000ull) {
    }
    __syncthreads();
  }
  if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

template <int KH, int VH, bool PAGED>
static int launch_prompt_exact(const CUtensorMap& km, const CUtensorMap& vm, const CUtensorMap& rm, ExactPromptArgs a, int n_seqs, int max_queries,
                               cudaStream_t s) {
  constexpr int STAGES = KH + VH >= 5 ? 3 : 4;
  constexpr size_t smem = 2 * KH * 128 * 128 + static_cast<size_t>(STAGES) * (KH + VH) * 64 * 128 + (2 * STAGES + 12) * 8 + 16 + 1024;
  static_assert(smem <= 227 * 1024, "shared memory of one CTA");
  auto kernel = attn_prompt_exact_kernel<KH, VH, PAGED, STAGES>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess) {
    set_error("attention_prompt_exact: cannot reserve %zu bytes of shared memory", smem);
    return kCudaError;
  }
  // Few rows: with two row tiles a CTA, half of the SMs or more would have none
  const int max_rows = max_queries * (a.q_heads / a.kv_heads);
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
  a.cta_rows = static_cast<long long>(a.kv_heads) * ceil_div(max_rows, 256) * n_seqs * 2 <= sms ? 128 : 256;
  TIE_LAUNCH(kernel, dim3(a.kv_heads, ceil_div(max_rows, a.cta_rows), n_seqs), kExactThreads, smem, s, km, vm, rm, a);
  TIE_RETURN_LAUNCH("attention_prompt_exact");
}

// The latents and rotated key parts that the portions' rows see, from the pages into rows [.., kd] one after the other (what
// expanded_first and expanded_rows say), zeros behind a sequence's last key and ahead of the first key that the window leaves its first
// row: pages there have been given back, and what the table names in their place belongs to others. A warp a row.
__global__ void __launch_bounds__(256) latent_gather_kernel(const __nv_bfloat16* __restrict__ keys, const int* __restrict__ query_start,
                                                           const int* __restrict__ context_lens, const int* __restrict__ block_tables,
                                                           int max_blocks, int n_seqs, int window, int page_size, int kd, int rows,
                                                           __nv_bfloat16* __restrict__ out) {
  pdl_sync();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  int s = 0, at = row;
  for (; s < n_seqs; ++s) {
    const int n = expanded_rows(context_lens[s], query_start[s + 1] - query_start[s], window);
    if (at < n) break;
    at -= n;
  }
  int key = 0;
  bool there = false;
  if (s < n_seqs) {
    const int context = context_lens[s], queries = query_start[s + 1] - query_start[s];
    key = expanded_first(context, queries, window) + at;
    there = key < context && (window <= 0 || key > context - queries - window);
  }
  const __nv_bfloat16* src = keys;
  if (there) src += (static_cast<long long>(block_tables[static_cast<long long>(s) * max_blocks + key / page_size]) * page_size + key % page_size) * kd;
  for (int c = lane; c < kd / 8; c += 32)
    reinterpret_cast<uint4*>(out + static_cast<long long>(row) * kd)[c] = there ? reinterpret_cast<const uint4*>(src)[c] : make_uint4(0u, 0u, 0u, 0u);
}

}  // namespace tie

using namespace tie;

// Rows [0, rows) of the step belong to sequences 0..n_seqs-1, each bringing several tokens; max_queries is the largest number of tokens
// one of them brings; pages is the number of pages of the cache planes. sink: [q_heads] or null.
TIE_API int tie_attention_prompt_exact(const void* q, long long q_stride, const void* k_cache, const void* v_cache, void* out,
                                       const int* query_start, const int* context_lens, const int* block_tables, int max_blocks,
                                       int n_seqs, int max_queries, int q_heads, int kv_heads, int head_dim, int page_size, int pages,
                                       int window, float scale, const float* sink, cudaStream_t s) {
  TIE_REQUIRE(head_dim == 64 || head_dim == 128, "attention_prompt_exact: head_dim %d is not 64 or 128", head_dim);
  TIE_REQUIRE(q_heads > 0 && kv_heads > 0 && q_heads % kv_heads == 0, "attention_prompt_exact: %d query heads over %d kv heads", q_heads, kv_heads);
  TIE_REQUIRE(page_size >= 8 && (page_size & (page_size - 1)) == 0, "attention_prompt_exact: page size %d is not a power of two from 8 up", page_size);
  TIE_REQUIRE(q_stride % 8 == 0 && reinterpret_cast<uintptr_t>(q) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0,
              "attention_prompt_exact: q and out rows must be 16-byte aligned");
  TIE_REQUIRE(scale > 0.0f && window >= 0, "attention_prompt_exact: the scale must be positive, the window not negative");
  if (n_seqs == 0 || max_queries == 0) return kOk;
  TIE_REQUIRE(n_seqs <= 65535 && static_cast<long long>(max_queries) * (q_heads / kv_heads) <= 65535LL * 128,
              "attention_prompt_exact: %d queries in one portion are too many", max_queries);
  int shift = 0;
  while ((1 << shift) < page_size) ++shift;
  const int box_rows = page_size < kKeysPerTile ? page_size : kKeysPerTile;
  CUtensorMap km, vm;
  const long long rows = static_cast<long long>(pages) * kv_heads * page_size;
  TIE_REQUIRE(make_map_bf16(&km, k_cache, rows, head_dim, head_dim, 64, box_rows) && make_map_bf16(&vm, v_cache, rows, head_dim, head_dim, 64, box_rows),
              "attention_prompt_exact: cuTensorMapEncodeTiled failed");
  TIE_REQUIRE(status_word() != nullptr, "attention_prompt_exact: cannot allocate the status word");
  const ExactPromptArgs a{static_cast<const __nv_bfloat16*>(q), static_cast<__nv_bfloat16*>(out), query_start, context_lens, block_tables,
                          status_word(), sink, q_stride, max_blocks, q_heads, kv_heads, page_size, shift, window, 0, 0,
                          scale * 1.4426950408889634f, 256};
  return head_dim == 64 ? launch_prompt_exact<1, 1, true>(km, vm, km, a, n_seqs, max_queries, s)
                        : launch_prompt_exact<2, 2, true>(km, vm, km, a, n_seqs, max_queries, s);
}

// out [rows, kd] from the pages [pages, 1, page_size, kd] (kd a multiple of 8): what portions of `n_seqs` sequences see, padded to whole
// tiles of 64 rows a sequence.
TIE_API int tie_latent_gather(const void* keys, const int* query_start, const int* context_lens, const int* block_tables, int max_blocks,
                              int n_seqs, int window, int page_size, int kd, int rows, void* out, cudaStream_t s) {
  TIE_REQUIRE(kd > 0 && kd % 8 == 0 && page_size > 0 && window >= 0 && reinterpret_cast<uintptr_t>(keys) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0,
              "latent_gather: rows of %d must be whole 16-byte pieces", kd);
  if (rows <= 0) return kOk;
  TIE_LAUNCH(latent_gather_kernel, ceil_div(rows, 8), 256, 0, s, static_cast<const __nv_bfloat16*>(keys), query_start, context_lens, block_tables,
             max_blocks, n_seqs, window, page_size, kd, rows, static_cast<__nv_bfloat16*>(out));
  TIE_RETURN_LAUNCH("latent_gather");
}

// Latent attention over multiplied-out keys: q [T, heads * 192] (128 + 64 rotated), latents [kv_rows, kd] as tie_latent_gather leaves them
// (the rotated part the last 64 columns), kv [kv_rows, heads * 256]: every head's 128 key dimensions, then every head's value.
TIE_API int tie_attention_latent_expanded(const void* q, long long q_stride, const void* latents, int kd, const void* kv, int kv_rows, void* out,
                                          const int* query_start, const int* context_lens, int n_seqs, int max_queries, int heads, int window,
                                          float scale, const float* sink, cudaStream_t s) {
  TIE_REQUIRE(heads > 0 && kd >= 64 && kd % 8 == 0 && kv_rows >= 0 && scale > 0.0f && window >= 0, "latent attention: bad sizes heads=%d kd=%d", heads, kd);
  TIE_REQUIRE(q_stride % 8 == 0 && reinterpret_cast<uintptr_t>(q) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0,
              "latent attention: q and out rows must be 16-byte aligned");
  if (n_seqs <= 0 || max_queries <= 0) return kOk;
  TIE_REQUIRE(n_seqs <= 65535 && max_queries <= 65535 * 128, "latent attention: %d queries in one portion are too many", max_queries);
  CUtensorMap km, rm;
  const long long cols = static_cast<long long>(heads) * 256;
  TIE_REQUIRE(make_map_bf16(&km, kv, kv_rows, cols, cols, 64, kKeysPerTile) && make_map_bf16(&rm, latents, kv_rows, kd, kd, 64, kKeysPerTile),
              "latent attention: cuTensorMapEncodeTiled failed");
  TIE_REQUIRE(status_word() != nullptr, "latent attention: cannot allocate the status word");
  const ExactPromptArgs a{static_cast<const __nv_bfloat16*>(q), static_cast<__nv_bfloat16*>(out), query_start, context_lens, nullptr,
                          status_word(), sink, q_stride, 0, heads, heads, 0, 0, window, heads * 128, kd - 64,
                          scale * 1.4426950408889634f, 256};
  return launch_prompt_exact<3, 2, false>(km, km, rm, a, n_seqs, max_queries, s);
}
