// 32-bit matrix products on the tensor cores, out[M, N] = a[M, K] . w[N, K]^T with float operands and results.
//
// Every float is the sum of three bfloat16 numbers, x = hi + 2^-8 mid + 2^-16 lo, each the rounding of what the ones before it leave
// over: 8 bits of mantissa three times, 24 in all. The second and third are held 2^8 and 2^16 up, so that the three are x exactly for
// every float, subnormal ones too (unscaled, values below 2^-109 lost low bits: bfloat16 ends at 2^-133). Six of the nine products of
// terms are formed, the smallest first, and the accumulator comes down by 2^8 (scale-input-d) ahead of the next order of magnitude;
// what the other three (mid lo, lo mid, lo lo) leave out is below 2^-26 of a product, a quarter of a unit of the float product. This is
// Ozaki's error-free splitting with a fixed number of slices.
// The tensor core multiplies the terms exactly; its float accumulator is trusted with 64 k's only: a k-block's sum is then read out of
// tensor memory and added in registers, to the nearest. Its additions cut off: sums of one sign came out 0.7 to 1.4 units of 2^-24
// too small. Every second block's sum is therefore taken 2^-23 larger, in the addition, which leaves a mean of nearly nothing.
// Relative error against 64 bits, here and with the FFMAs of gemm_simt.cu, at k = 128, 1,024 and 4,096: normal operands 0.8, 1.0, 1.1e-7
// against 1.5, 2.1, 2.9e-7; operands of one sign 0.4, 0.5, 0.5e-7 against 0.9, 0.7, 0.8e-7 (before the correction 0.9, 1.0, 1.0e-7); operands
// spread over twelve decades, where a few products make the sum, 0.9, 1.1, 1.2e-7 against 0.7, 1.1, 1.4e-7. With one block of 64 k's nothing
// evens out (one sign: 0.9e-7 against 0.7e-7): such products stay with the FFMAs.
//
// One CTA computes a tile of 128 x BN. Warps 0-15 read both operands' k-block (float, straight from global memory, any size, stride
// and alignment; the next block's loads are in flight while this one is split), write the six term tiles in the tensor core's
// swizzled layout, and arrive on full[s]; warp 24 issues 24 MMAs a block (6 term pairs x 4 steps of 16); warps 16-23 add the
// block's sums from one of two accumulators while the other is filled. Where the tiles leave SMs idle, k is cut over the CTAs of a
// cluster, which exchange their sums through distributed shared memory, each adding a share of the columns in rank order.
//
// What bounds it: the splitting warps (a k-block of 128 x 64 takes them 1,750 cycles, of 128 x 96 2,100; the MMAs 1,250 and 1,580
// beside it), against 4,100 and 6,100 for the FFMAs of the same outputs. 800 threads of 72 registers keep a block of loads in
// flight; with half the splitting warps a block took 3,100 cycles. Two stages: a third left so little L1 that the loop's few
// spilled words came from L2 (2,400 cycles). 389 x 3,072 x 1,024: 112 -> 28.6 us, 389 x 1,024 x 1,024: 39.5 -> 15.6, 32 x 1,536 x
// 1,024: 17.9 -> 10.4, 1,000 x 2,048 x 2,048: 254 -> 74.
//
// Infinities and NaN: hi is one, and the terms behind it make NaN of every sum of its row or column (inf - inf). So does a float that
// rounds to an infinity in bfloat16, and partial sums beyond the largest float stay infinite: a thread that ends with a sum that is not
// finite computes its sums again with FFMAs.
#include "umma.cuh"

namespace tie {

constexpr int kFsSplitters = 16, kFsAdders = 8;     // warps
constexpr int kFsIssuer = kFsSplitters + kFsAdders, kFsThreads = 32 * (kFsIssuer + 1);
constexpr int kFsRowStep = kFsSplitters * 2;        // rows that the splitting warps take at once, half a warp a row
constexpr int kFsBM = 128, kFsBK = 64;

template <int BN> struct FsConfig {
  static constexpr int kA = kFsBM * kFsBK * 2, kB = BN * kFsBK * 2;      // one term's tile
  static constexpr int kStage = 3 * (kA + kB);
  static constexpr int kStages = 2;
  static_assert(kStages * kStage >= kFsBM * BN * 4, "the sums from the cluster's CTAs come into the stages' memory");
  static constexpr int kTmemCols = 2 * BN <= 64 ? 64 : 2 * BN <= 128 ? 128 : 256;
  static constexpr int kAccStride = kTmemCols / 2;
  static constexpr size_t kSmem = static_cast<size_t>(kStages) * kStage + 1024 + 128;
};

struct FsArgs {
  const float *a, *w;
  float* out;
  int M, N, K, tiles_m, splits, k_blocks, k_blocks_per_split;
  long long lda, ldw, ldo;
  int wide_a, wide_w, wide_out;      // rows are whole 16-byte pieces
  int* status;
};

__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// What is left of a and b beside the bfloat16 pair, 2^8 up (exact, as is the difference).
__device__ __forceinline__ void take_off(float& a, float& b, uint32_t pair) {
  asm("{\n\t.reg .b64 x, h;\n\t"
      "mov.b64 x, {%0, %1};\n\t"
      "mov.b64 h, {%2, %3};\n\t"
      "fma.rn.f32x2 x, h, %4, x;\n\t"
      "mul.rn.f32x2 x, x, %5;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(__uint_as_float(pair << 16)), "f"(__uint_as_float(pair & 0xffff0000u)), "l"(0xbf800000bf800000ull), "l"(0x4380000043800000ull));
}
// umma_bf16 onto 2^-8 times the accumulator.
__device__ __forceinline__ void umma_bf16_down8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, 1, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 8;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc)
      : "memory");
}

template <int BN>
__global__ void __launch_bounds__(kFsThreads, 1) gemm_f32_split_kernel(const __grid_constant__ FsArgs g) {
  using C = FsConfig<BN>;
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  float4* inbox = reinterpret_cast<float4*>(smem);       // once every CTA of the cluster is through with its stages
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStage);
  uint64_t* empty = full + C::kStages;
  uint64_t* acc_full = empty + C::kStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x % g.splits, tile = blockIdx.x / g.splits;
  const int m0 = (tile % g.tiles_m) * kFsBM, n0 = (tile / g.tiles_m) * BN;
  const int kb_begin = split * g.k_blocks_per_split, kb_end = min(g.k_blocks, kb_begin + g.k_blocks_per_split);

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(full + s, kFsSplitters);
      mbar_init(empty + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + b, 1);
      mbar_init(acc_empty + b, kFsAdders);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kFsIssuer) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(C::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;
  pdl_wait();

  if (warp < kFsSplitters) {
    constexpr int kRows = (kFsBM + BN) / kFsRowStep, kRowsA = kFsBM / kFsRowStep;      // a thread's rows, four k's of each
    const int r0 = threadIdx.x >> 4, chunk = threadIdx.x & 15;
    // Rows beyond the operand's end keep what the registers hold: they reach no output that is stored.
    const char* pa = reinterpret_cast<const char*>(g.a + static_cast<long long>(m0 + r0) * g.lda + chunk * 4);
    const char* pw = reinterpret_cast<const char*>(g.w + static_cast<long long>(n0 + r0) * g.ldw + chunk * 4);
    const int step_a = static_cast<int>(g.lda) * (kFsRowStep * 4), step_w = static_cast<int>(g.ldw) * (kFsRowStep * 4);     // (of wide rows)
    const int left_a = g.M - m0 - r0, left_w = g.N - n0 - r0;
    float4 next[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) next[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto load = [&](int i, int kb) {
      const bool of_a = i < kRowsA;
      const int j = of_a ? i : i - kRowsA;
      if (kFsRowStep * j < (of_a ? left_a : left_w))
        next[i] = __ldcg(reinterpret_cast<const float4*>((of_a ? pa + j * step_a : pw + j * step_w) + kb * (kFsBK * 4)));
    };
    auto load_any = [&](int kb) {         // a k-block that ends beyond K, or rows that are no whole 16-byte pieces
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const bool of_a = i < kRowsA;
        const int j = of_a ? i : i - kRowsA, left = g.K - kb * kFsBK - chunk * 4;
        if (kFsRowStep * j >= (of_a ? left_a : left_w)) continue;
        const float* p = reinterpret_cast<const float*>(of_a ? pa : pw) + static_cast<long long>(kFsRowStep * j) * (of_a ? g.lda : g.ldw) + kb * kFsBK;
        next[i] = make_float4(left > 0 ? p[0] : 0.0f, left > 1 ? p[1] : 0.0f, left > 2 ? p[2] : 0.0f, left > 3 ? p[3] : 0.0f);
      }
    };
    // k-blocks from here on are read that way
    const int kb_any = g.wide_a != 0 && g.wide_w != 0 ? g.K / kFsBK : 0;
    if (kb_begin < min(kb_end, kb_any)) {
#pragma unroll
      for (int i = 0; i < kRows; ++i) load(i, kb_begin);
    } else if (kb_begin < kb_end) {
      load_any(kb_begin);
    }
    uint8_t* const to_a = smem + r0 * 128 + (((chunk >> 1) ^ (r0 & 7)) << 4) + (chunk & 1) * 8;      // (rows of the next step: the same swizzle)
    for (int kb = kb_begin; kb < kb_end; ++kb) {
      const int it = kb - kb_begin, s = it % C::kStages;
      if (!__all_sync(0xffffffffu, mbar_wait(empty + s, ((it / C::kStages) & 1) ^ 1, abort_flag, g.status, 1) ? 1 : 0)) break;
      uint8_t* const stage = to_a + s * C::kStage;
      auto emit = [&](int i, float4 v) {
        const int term = i < kRowsA ? C::kA : C::kB;
        uint8_t* const to = stage + (i < kRowsA ? i : i - kRowsA) * (kFsRowStep * 128) + (i < kRowsA ? 0 : 3 * C::kA);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const uint32_t p = bf16_pair(v.x, v.y), q = bf16_pair(v.z, v.w);
          *reinterpret_cast<uint2*>(to + t * term) = make_uint2(p, q);
          if (t < 2) {
            take_off(v.x, v.y, p);
            take_off(v.z, v.w, q);
          }
        }
      };
      if (kb + 1 < min(kb_end, kb_any)) {
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const float4 v = next[i];
          load(i, kb + 1);
          emit(i, v);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kRows; ++i) emit(i, next[i]);
        if (kb + 1 < kb_end) load_any(kb + 1);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(full + s)) : "memory");
    }
    __syncthreads();
  } else if (warp == kFsIssuer) {
    constexpr uint32_t idesc = instr_desc(BN);
    // term pairs, the smallest products first: (a, w) with hi 0, mid 1, lo 2; three 2^16 up, two 2^8 up, then the products of hi
    constexpr int kTermA[6] = {2, 0, 1, 1, 0, 0}, kTermW[6] = {0, 2, 1, 0, 1, 0};
    const uint32_t ring_lo = desc_lo_sw128(smem_u32(smem));
    for (int kb = kb_begin; kb < kb_end; ++kb) {
      const int it = kb - kb_begin, s = it % C::kStages, buf = it & 1;
      const bool ok = mbar_wait(acc_empty + buf, ((it >> 1) & 1) ^ 1, abort_flag, g.status, 2) &&
                      mbar_wait(full + s, (it / C::kStages) & 1, abort_flag, g.status, 2);
      if (!__all_sync(0xffffffffu, ok ? 1 : 0)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a_lo = ring_lo + s * (C::kStage >> 4), w_lo = a_lo + (3 * C::kA >> 4);
      const uint32_t acc = tmem_base + buf * C::kAccStride;
      if (elect_one()) {
#pragma unroll
        for (int t = 0; t < 6; ++t) {
#pragma unroll
          for (int k = 0; k < kFsBK / 16; ++k) {
            const uint64_t da = desc_from_words(a_lo + kTermA[t] * (C::kA >> 4) + 2 * k, kDescHiSw128);
            const uint64_t dw = desc_from_words(w_lo + kTermW[t] * (C::kB >> 4) + 2 * k, kDescHiSw128);
            if (k == 0 && (t == 3 || t == 5)) umma_bf16_down8(acc, da, dw, idesc);
            else umma_bf16(acc, da, dw, idesc, t + k > 0 ? 1u : 0u);
          }
        }
        umma_commit(empty + s);
        umma_commit(acc_full + buf);
      }
      __syncwarp();
    }
    __syncthreads();      // the adding warps have read the accumulators
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::kTmemCols) : "memory");
  } else {
    constexpr int kCols = BN / 2;                    // four warps add one half of the columns each
    const int half = (warp - kFsSplitters) >> 2, col0 = half * kCols;
    float sum[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) sum[c] = 0.0f;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    for (int kb = kb_begin; kb < kb_end; ++kb) {
      const int it = kb - kb_begin, buf = it & 1;
      const float up = (kb & 1) != 0 ? 1.00000011920928955f : 1.0f;          // 1 + 2^-23
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full + buf, (it >> 1) & 1, abort_flag, g.status, 3) ? 1 : 0)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c0 = 0; c0 < kCols; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(tmem_base + buf * C::kAccStride + lanes + col0 + c0, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 16 == kCols) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(acc_empty + buf)) : "memory");
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) sum[c0 + e] = fmaf(__uint_as_float(r[e]), up, sum[c0 + e]);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    const int row = (warp & 3) * 32 + lane, n1 = n0 + col0;
    if (m0 + row < g.M) {
      bool finite = true;
#pragma unroll
      for (int c = 0; c < kCols; ++c) finite = finite && fabsf(sum[c]) <= 3.402823466e38f;
      if (!finite) {            // with FFMAs, in order of k
#pragma unroll
        for (int c = 0; c < kCols; ++c) sum[c] = 0.0f;
        const float* ar = g.a + static_cast<long long>(m0 + row) * g.lda;
        const int k_end = min(g.K, kb_end * kFsBK);
        for (int k = kb_begin * kFsBK; k < k_end; ++k) {
          const float x = ar[k];
#pragma unroll
          for (int c = 0; c < kCols; ++c)
            if (n1 + c < g.N) sum[c] = fmaf(x, g.w[static_cast<long long>(n1 + c) * g.ldw + k], sum[c]);
        }
      }
    }
    if (g.splits == 1) {
      float* const orow = g.out + static_cast<long long>(m0 + row) * g.ldo + n1;
      if (m0 + row < g.M) {
#pragma unroll
        for (int c = 0; c < kCols; c += 4) {
          if (g.wide_out != 0 && n1 + c + 4 <= g.N) {
            *reinterpret_cast<float4*>(orow + c) = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (n1 + c + e < g.N) orow[c + e] = sum[c + e];
          }
        }
      }
    } else {
      // Four columns at a time to the CTA that adds them: groups of four go round the cluster. No CTA uses its stages any more.
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      const int mine = BN / 4 / g.splits;                                        // (splits divide them)
#pragma unroll
      for (int q = 0; q < kCols / 4; ++q) {
        const int quad = col0 / 4 + q;
        const uint32_t to = smem_u32(inbox + (split * mine + quad / g.splits) * kFsBM + row);
        uint32_t addr;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(to), "r"(quad % g.splits));
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(sum[4 * q]), "f"(sum[4 * q + 1]), "f"(sum[4 * q + 2]),
                     "f"(sum[4 * q + 3]) : "memory");
      }
      __syncwarp();
    }
  }
  if (g.splits == 1) return;
  if (warp < kFsSplitters || warp >= kFsSplitters + kFsAdders)
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int mine = BN / 4 / g.splits;
  for (int id = threadIdx.x; id < mine * kFsBM; id += kFsThreads) {
    const int j = id / kFsBM, r = id % kFsBM, c = n0 + (j * g.splits + split) * 4;
    float4 v = inbox[j * kFsBM + r];
    for (int z = 1; z < g.splits; ++z) {
      const float4 u = inbox[(z * mine + j) * kFsBM + r];
      v.x += u.x, v.y += u.y, v.z += u.z, v.w += u.w;
    }
    if (m0 + r < g.M) {
      float* o = g.out + static_cast<long long>(m0 + r) * g.ldo + c;
      if (g.wide_out != 0 && c + 4 <= g.N) {
        *reinterpret_cast<float4*>(o) = v;
      } else {
        if (c < g.N) o[0] = v.x;
        if (c + 1 < g.N) o[1] = v.y;
        if (c + 2 < g.N) o[2] = v.z;
        if (c + 3 < g.N) o[3] = v.w;
      }
    }
  }
}

template <int BN>
static int launch_fs(const FsArgs& g, cudaStream_t s) {
  auto kernel = gemm_f32_split_kernel<BN>;
  constexpr int smem = static_cast<int>(FsConfig<BN>::kSmem);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    set_error("gemm_f32_split: cannot reserve %d bytes of shared memory", smem);
    return kCudaError;
  }
  const long long ctas = static_cast<long long>(g.tiles_m) * ceil_div(g.N, BN) * g.splits;
  if (g.splits == 1) {
    TIE_LAUNCH(kernel, dim3(static_cast<unsigned>(ctas)), kFsThreads, smem, s, g);
  } else {
    // clusters that hold tensor memory start when the kernel ahead has ended, like the pairs of gemm_tc2.cu
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(kFsThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = g.splits;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, g);
  }
  TIE_RETURN_LAUNCH("gemm_f32_split");
}

int launch_gemm_f32_split(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldw, long long ldo, int bn,
                          int splits, cudaStream_t s) {
  TIE_REQUIRE(status_word() != nullptr, "gemm_f32_split: cannot allocate the status word");
  FsArgs g = {};
  g.a = a, g.w = w, g.out = out, g.M = M, g.N = N, g.K = K, g.lda = lda, g.ldw = ldw, g.ldo = ldo;
  g.tiles_m = ceil_div(M, kFsBM);
  g.splits = splits;
  g.k_blocks = ceil_div(K, kFsBK);
  g.k_blocks_per_split = ceil_div(g.k_blocks, splits);
  g.wide_a = lda % 4 == 0 && lda < (1 << 22) && reinterpret_cast<uintptr_t>(a) % 16 == 0;
  g.wide_w = ldw % 4 == 0 && ldw < (1 << 22) && reinterpret_cast<uintptr_t>(w) % 16 == 0;
  g.wide_out = ldo % 4 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
  g.status = status_word();
  if (bn == 32) return launch_fs<32>(g, s);
  return bn == 64 ? launch_fs<64>(g, s) : launch_fs<96>(g, s);
}

// CTAs of the kernel that are resident at once in clusters of `splits` (1, 2, 4 or 8): which GPCs have how many SMs differs from GPU to
// GPU, so it is asked for, once (148, 132 and 120 for 2, 4 and 8 on one; taken for 128, sixteen clusters of eight ran in two waves: 32 x 512 x
// 1,024 14.7 us, now 9.2). Every width takes an SM for itself.
static int resident_ctas(int splits) {
  static int known[9] = {};
  if (known[splits] == 0) {
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(148 / splits * splits);
    cfg.blockDim = dim3(kFsThreads);
    cfg.dynamicSmemBytes = FsConfig<96>::kSmem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = splits;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (splits == 1 ||
        cudaFuncSetAttribute(gemm_f32_split_kernel<96>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(FsConfig<96>::kSmem)) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_f32_split_kernel<96>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = (splits < 4 ? 148 : splits == 4 ? 132 : 96) / splits;
    }
    known[splits] = n * splits;
  }
  return known[splits];
}

// The width and the splits with the least estimated time (us: a k-block of a tile, a wave of tiles, a cluster; fitted to a sweep of 18
// products of 32 to 389 rows, 64 to 6,144 columns, k 128 to 4,096, each launch's weight from memory: the choice costs 0.05 % more
// than the best one on average, 4 % at most). Clusters only where the tiles leave SMs idle: they never start early.
int launch_gemm_f32_split_chosen(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldw, long long ldo,
                                 cudaStream_t s) {
  const int k_blocks = ceil_div(K, kFsBK);
  int width = 0, splits = 1;
  float best = 0.0f;
  for (int bn = 32; bn <= 96; bn += 32) {
    const long long tiles = static_cast<long long>(ceil_div(M, kFsBM)) * ceil_div(N, bn);
    for (int c = 1; c <= 8; c *= 2) {
      if (c > 1 && (tiles > 148 || k_blocks < c)) break;
      const int at_once = resident_ctas(c);
      const float block = bn == 32 ? 0.85f : bn == 64 ? 1.0f : 1.35f;
      const float us = ceil_div(tiles * c, at_once) * (ceil_div(k_blocks, c) * block + 3.6f) + (c == 1 ? 0.0f : c == 2 ? 2.8f : c == 4 ? 3.0f : 4.0f);
      if (width == 0 || us < best) best = us, width = bn, splits = c;
    }
  }
  return launch_gemm_f32_split(a, w, out, M, N, K, lda, ldw, ldo, width, splits, s);
}

}  // namespace tie

using namespace tie;

// The float product by three bfloat16 terms with its tile width (32, 64 or 96 columns) and splits of k (1, 2, 4 or 8) given (tests).
TIE_API int tie_gemm_f32_split(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldw, long long ldo,
                               int bn, int splits, cudaStream_t s) {
  TIE_REQUIRE(M > 0 && N > 0 && K > 0 && lda >= K && ldw >= K && ldo >= N, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
  TIE_REQUIRE((bn == 32 || bn == 64 || bn == 96) && (splits == 1 || splits == 2 || splits == 4 || splits == 8), "gemm: tile %d, splits %d", bn, splits);
  return launch_gemm_f32_split(a, w, out, M, N, K, lda, ldw, ldo, bn, splits, s);
}
