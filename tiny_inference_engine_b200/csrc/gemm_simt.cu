// Matrix products on the CUDA cores: out[M, N] = a[M, K] . w[N, K]^T with float accumulation.
//
// These are the FFMA kernels of the true 32-bit path (float in, float out; no reduced-precision matrix mode): few rows,
// batches and short k. Its large products run on the tensor cores without giving precision up (gemm_f32_split.cu). They
// take every size; the bfloat16 instantiations serve sizes that the tensor-core kernels refuse. The reference's
// counterpart is its dot-product matmul (src/backend/cpu/cpu_backend.cpp:78-139): weights
// in the checkpoint's [out, in] layout, y = x . W^T, no bias.
#include <type_traits>

#include "common.cuh"
#include "launchers.h"

namespace tie {

int launch_gemm_f32_split_chosen(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldw, long long ldo,
                                 cudaStream_t s);      // gemm_f32_split.cu

// ---------------------------------------------------------------------------------------------
// Tiled kernel for any M, N, K (bfloat16 operands): 64 x 64 output tile, 16-deep k slices, 256 threads, 4 x 4
// outputs per thread. Both operands are k-contiguous, so a slice is read along k and stored
// transposed in shared memory.
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) gemm_tiled_kernel(const TI* __restrict__ a, const TI* __restrict__ w,
                                                         TO* __restrict__ out, int M, int N, int K, long long lda,
                                                         long long ldw, long long ldo, long long sa, long long sw,
                                                         long long so) {
  pdl_sync();
  a += blockIdx.z * sa, w += blockIdx.z * sw, out += blockIdx.z * so;      // one product of a batch (strides 0: the only one)
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ float as[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
  const int lr = tid / 4;        // row of the tile this thread loads (0..63)
  const int lk = (tid % 4) * 4;  // first of its 4 k's
  float acc[4][4] = {};

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + lk + j;
      const int m = m0 + lr, n = n0 + lr;
      as[lk + j][lr] = (m < M && k < K) ? ld(a + static_cast<long long>(m) * lda + k) : 0.0f;
      ws[lk + j][lr] = (n < N && k < K) ? ld(w + static_cast<long long>(n) * ldw + k) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float av[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = as[k][tm + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = ws[k][tn + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + tm + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tn + j;
      if (n < N) st(out + static_cast<long long>(m) * ldo + n, acc[i][j]);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Float operands, more than a few rows. A warp owns 32 x 32 outputs, 8 x 4 a lane; k slices of 32 come by cp.async through a ring
// of three buffers in shared memory, row by row as they lie in memory (no transposition), and a lane reads its rows 16 bytes (four
// k's) at a time: the rows of a quarter warp lie 36 words apart, so they hit different banks. The products are `fma.rn.f32x2` over
// neighbouring k's (an accumulator is the sums over even and over odd k's, added at the end): 64 instructions and 12 loads per
// four k's instead of 128 and 12. What bounds it is shared memory (128 bytes a clock and SM into registers, broadcast or not: 1.5
// clocks of loads a clock of FFMA), then the warps in flight; 8 x 8 and 8 x 16 outputs a lane need fewer bytes but 220 and 250
// registers, and were slower with the four warps an SM that leaves (a 389 x 1024 x 1024 product: 37.1, 40.2 and 40.2 us).
// Where the tiles of the output leave SMs idle, k is cut over the CTAs of a cluster, which add their sums in rank order through
// distributed shared memory.
constexpr int kSliceK = 32, kSliceLd = kSliceK + 4, kSliceStages = 3;

__device__ __forceinline__ void ffma2(unsigned long long& acc, unsigned long long x, unsigned long long y) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y));
}

// WIDE: K, the row strides and the bases are whole 16-byte pieces; else the copies are 4 bytes each.
template <int WM, int WN, bool WIDE>
__global__ void __launch_bounds__(32 * WM * WN, WM * WN == 8 ? 2 : 1) gemm_f32_kernel(const float* __restrict__ a, const float* __restrict__ w,
                                                          float* __restrict__ out, int M, int N, int K, long long lda, long long ldw,
                                                          long long ldo, long long sa, long long sw, long long so, int splits) {
  pdl_sync();
  constexpr int BM = 32 * WM, BN = 32 * WN, THREADS = 32 * WM * WN, STAGE = (BM + BN) * kSliceLd;
  extern __shared__ __align__(16) float ring[];
  const int product = blockIdx.z / splits, rank = blockIdx.z % splits;
  a += product * sa, w += product * sw, out += product * so;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;      // (the row tiles of one stretch of the weight run side by side)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slices = (K + kSliceK - 1) / kSliceK, per = (slices + splits - 1) / splits;
  const int first = min(rank * per, slices), count = min(per, slices - first);

  auto fetch = [&](int i) {
    if (i < count) {
      const int k0 = (first + i) * kSliceK;
      float* stage = ring + (i % kSliceStages) * STAGE;
      constexpr int PIECE = WIDE ? 4 : 1, PER_ROW = kSliceK / PIECE;
#pragma unroll 4
      for (int p = tid; p < (BM + BN) * PER_ROW; p += THREADS) {
        const int r = p / PER_ROW, k = k0 + (p % PER_ROW) * PIECE;
        const bool of_a = r < BM;
        const int row = of_a ? m0 + r : n0 + r - BM;
        const bool there = row < (of_a ? M : N) && k < K;
        const float* src = of_a ? a + (there ? row * lda + k : 0) : w + (there ? row * ldw + k : 0);
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(stage + r * kSliceLd + (k - k0)));
        if (WIDE) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(there ? 4 : 0) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int mrow = (warp / WN) * 32 + (lane >> 3), ncol = (warp % WN) * 32 + (lane & 7);      // + 4 i, + 8 j
  unsigned long long acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  for (int i = 0; i < kSliceStages - 1; ++i) fetch(i);
  for (int i = 0; i < count; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kSliceStages - 2) : "memory");
    __syncthreads();                          // slice i is there for everyone, and everyone is through with slice i - 1
    fetch(i + kSliceStages - 1);
    const float* as = ring + (i % kSliceStages) * STAGE + mrow * kSliceLd;
    const float* ws = ring + (i % kSliceStages) * STAGE + (BM + ncol) * kSliceLd;
#pragma unroll
    for (int k = 0; k < kSliceK; k += 4) {
      ulonglong2 av[8], wv[4];
#pragma unroll
      for (int x = 0; x < 8; ++x) av[x] = *reinterpret_cast<const ulonglong2*>(as + 4 * x * kSliceLd + k);
#pragma unroll
      for (int y = 0; y < 4; ++y) wv[y] = *reinterpret_cast<const ulonglong2*>(ws + 8 * y * kSliceLd + k);
#pragma unroll
      for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          ffma2(acc[x][y], av[x].x, wv[y].x);
          ffma2(acc[x][y], av[x].y, wv[y].y);
        }
    }
  }
  auto total = [](unsigned long long v) { return __uint_as_float(static_cast<uint32_t>(v)) + __uint_as_float(static_cast<uint32_t>(v >> 32)); };
  if (splits == 1) {
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const int m = m0 + mrow + 4 * x;
      if (m >= M) continue;
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int n = n0 + ncol + 8 * y;
        if (n < N) out[m * ldo + n] = total(acc[x][y]);
      }
    }
    return;
  }
  // The cluster's CTAs: each leaves its sums in its own shared memory and adds up a slice of the tile's rows.
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float* sums = ring;
#pragma unroll
  for (int x = 0; x < 8; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) sums[(mrow + 4 * x) * BN + ncol + 8 * y] = total(acc[x][y]);
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(sums));
  for (int p = tid; p < BM / splits * BN; p += THREADS) {
    const int r = (p / BN) * splits + rank, c = p % BN;
    if (m0 + r >= M || n0 + c >= N) continue;
    float v = 0.0f;
    for (int peer = 0; peer < splits; ++peer) {
      uint32_t at;
      float part;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine + (r * BN + c) * 4), "r"(peer));
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part) : "r"(at));
      v += part;
    }
    out[static_cast<long long>(m0 + r) * ldo + n0 + c] = v;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");      // nobody leaves while its sums are read
}

template <int WM, int WN>
int launch_f32_tile(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldw, long long ldo,
                    cudaStream_t s, int batch, long long sa, long long sw, long long so, int splits) {
  constexpr int BM = 32 * WM, BN = 32 * WN, ring = kSliceStages * (BM + BN) * kSliceLd, sums = BM * BN;
  constexpr int smem = (ring > sums ? ring : sums) * static_cast<int>(sizeof(float));
  const bool wide = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && sa % 4 == 0 && sw % 4 == 0 &&
                    reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0;
  auto kernel = wide ? gemm_f32_kernel<WM, WN, true> : gemm_f32_kernel<WM, WN, false>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    set_error("gemm_simt: cannot reserve %d bytes of shared memory", smem);
    return kCudaError;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ceil_div(M, BM), 0, batch * splits);
  cfg.blockDim = dim3(32 * WM * WN);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attrs[2];
  cfg.attrs = attrs;
  if (splits > 1) {
    attrs[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attrs[cfg.numAttrs].val.clusterDim.x = 1;
    attrs[cfg.numAttrs].val.clusterDim.y = 1;
    attrs[cfg.numAttrs].val.clusterDim.z = splits;
    ++cfg.numAttrs;
  }
  if (pdl_enabled()) {
    attrs[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  // A grid has 65,535 tiles of columns: a launch for as many columns each. (Tiles numbered in one direction cost the kernel two per cent.)
  constexpr int most = 65535 * BN;
  for (int n0 = 0; n0 < N; n0 = N - n0 > most ? n0 + most : N) {
    const int n = N - n0 < most ? N - n0 : most;
    cfg.gridDim.y = ceil_div(n, BN);
    cudaLaunchKernelEx(&cfg, kernel, a, w + n0 * ldw, out + n0, M, n, K, lda, ldw, ldo, sa, sw, so, splits);
  }
  TIE_RETURN_LAUNCH("gemm_f32");
}

// tile: 0 (128 x 64 outputs a CTA), 1 (64 x 64), 2 (32 x 64), -1: the tile and the splits with the least estimated time. Units are
// slices of 64 x 64 x 32: an SM does one in 1.0 us with eight warps of the large tile or more, 1.55 with the four of one middle
// tile (1.2 when it has several), 2.0 and 1.6 with the small one; a cluster costs 4 us and more (fitted to a sweep of 12 products,
// 20 to 2,048 rows, 1,024 to 32,000 columns: within 20 % of the best of the 12 choices everywhere).
int launch_gemm_f32(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldw, long long ldo,
                    cudaStream_t s, int batch, long long sa, long long sw, long long so, int tile, int splits) {
  if (tile < 0) {
    float best = 0.0f;
    const int slices = ceil_div(K, kSliceK);
    for (int t = 0; t < 3; ++t) {
      for (int c = 1; c <= 8; c *= 2) {
        if (c > 1 && (slices / c < 4 || static_cast<long long>(batch) * c > 65535)) break;
        const int per_sm = ceil_div(static_cast<long long>(ceil_div(M, 128 >> t)) * ceil_div(N, 64) * batch * c, 148);
        const float us = t == 0 ? 1.0f : t == 1 ? (per_sm == 1 ? 1.55f : 1.2f) : (per_sm <= 2 ? 2.0f : 1.6f);
        const float cost = per_sm * ceil_div(slices, c) * (2.0f / (1 << t)) * us + (c > 1 ? 4.0f + 0.5f * c : 0.0f);
        if (tile < 0 || cost < best) best = cost, tile = t, splits = c;
      }
    }
  }
  if (tile == 0) return launch_f32_tile<4, 2>(a, w, out, M, N, K, lda, ldw, ldo, s, batch, sa, sw, so, splits);
  if (tile == 1) return launch_f32_tile<2, 2>(a, w, out, M, N, K, lda, ldw, ldo, s, batch, sa, sw, so, splits);
  return launch_f32_tile<1, 2>(a, w, out, M, N, K, lda, ldw, ldo, s, batch, sa, sw, so, splits);
}

// ---------------------------------------------------------------------------------------------
// Few rows (decode): a warp per output column streams its weight row once with 16-byte
// loads and keeps MT accumulators; the MT activation rows come from L1/L2. Needs K to be a
// multiple of the 16-byte vector and 16-byte aligned rows. The loads' latency bounds it, so
// 1 << split warps of a block share a column's k where the columns are few, and the weight's
// lines are asked into L2 before the wait for the kernel in front (a hint: it reads nothing).
// The expert scores of 16 rows (32 columns, k 2,048): 7.2 us with one warp a column, 3.0 with eight.
template <typename TI, typename TO, int MT, int split>
__global__ void __launch_bounds__(256) gemm_small_m_kernel(const TI* __restrict__ a, const TI* __restrict__ w,
                                                           TO* __restrict__ out, int M, int N, int K, long long lda,
                                                           long long ldw, long long ldo, long long sa, long long sw,
                                                           long long so) {
  constexpr int V = Vec16<TI>::N;
  __shared__ float sums[8][MT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x * (8 >> split) + (warp >> split);
  const int m0 = blockIdx.y * MT;
  const TI* wr = w + blockIdx.z * sw + static_cast<long long>(n) * ldw;
  const int k0 = ((warp & ((1 << split) - 1)) * 32 + lane) * V;
  constexpr int step = (32 * V) << split;
  if (split != 0 && n < N && (lane & 7) == 0)
    for (int k = k0; k < K; k += step) asm volatile("prefetch.global.L2 [%0];" ::"l"(wr + k));
  pdl_sync();
  a += blockIdx.z * sa, out += blockIdx.z * so;
  if (split == 0 && n >= N) return;
  float acc[MT] = {};
  for (int k = split == 0 || n < N ? k0 : K; k < K; k += step) {
    Vec16<TI> wv;
    wv.load(wr + k);
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      if (m0 + i < M) {
        Vec16<TI> av;
        av.load(a + static_cast<long long>(m0 + i) * lda + k);
#pragma unroll
        for (int j = 0; j < V; ++j) acc[i] = fmaf(av.v[j], wv.v[j], acc[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const float v = warp_sum(acc[i]);
    if (lane == 0) {
      if (split != 0) sums[warp][i] = v;
      else if (m0 + i < M) st(out + static_cast<long long>(m0 + i) * ldo + n, v);
    }
  }
  if (split == 0) return;
  __syncthreads();
  const int col = threadIdx.x / MT, i = threadIdx.x % MT, nc = blockIdx.x * (8 >> split) + col;
  if (col < (8 >> split) && nc < N && m0 + i < M) {
    float v = 0.0f;
    for (int p = 0; p < (1 << split); ++p) v += sums[(col << split) + p][i];
    st(out + static_cast<long long>(m0 + i) * ldo + nc, v);
  }
}

template <typename TI, typename TO>
int launch_gemm(const void* a, const void* w, void* out, int M, int N, int K, long long lda, long long ldw,
                long long ldo, cudaStream_t s, int batch = 1, long long sa = 0, long long sw = 0, long long so = 0) {
  if (M == 0 || N == 0 || batch == 0) return kOk;
  const TI* ap = static_cast<const TI*>(a);
  const TI* wp = static_cast<const TI*>(w);
  TO* op = static_cast<TO*>(out);
  constexpr int V = Vec16<TI>::N;
  const bool vec_ok = K % V == 0 && lda % V == 0 && ldw % V == 0 && sa % V == 0 && sw % V == 0 &&
                      reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0;
  if (M <= 16 && vec_ok) {
    // warps share a column until the blocks fill the SMs, a whole vector a lane at least (16 rows, one warp a column before: 584
    // columns of k 2,048 7.5 -> 6.0 us, 256 of 4,096 12.7 -> 5.9; 600 of k 512 would go from 3.5 to 3.7); the rows have no say, so
    // that a row's sum is the same however many rows there are
    int split = 0;
    while (split < 3 && (static_cast<long long>(ceil_div(N, 8)) * batch << split) < 148 && K >= (64 * V) << split && K >= 128 * V) ++split;
    const dim3 grid(ceil_div(N, 8 >> split), ceil_div(M, M <= 4 ? 4 : 8), batch);
#define TIE_SMALL_M(MT, SPLIT) \
  TIE_LAUNCH((gemm_small_m_kernel<TI, TO, MT, SPLIT>), grid, 256, 0, s, ap, wp, op, M, N, K, lda, ldw, ldo, sa, sw, so)
#define TIE_SMALL_M_ROWS(SPLIT) \
  if (M <= 4) TIE_SMALL_M(4, SPLIT); \
  else TIE_SMALL_M(8, SPLIT)
    if (split == 0) { TIE_SMALL_M_ROWS(0); }
    else if (split == 1) { TIE_SMALL_M_ROWS(1); }
    else if (split == 2) { TIE_SMALL_M_ROWS(2); }
    else { TIE_SMALL_M_ROWS(3); }
#undef TIE_SMALL_M_ROWS
#undef TIE_SMALL_M
  } else if constexpr (std::is_same<TI, float>::value && std::is_same<TO, float>::value) {
    // One product of more than 16 rows by three bfloat16 terms on the tensor cores: nearer to 64 bits from two blocks of 64 k's on
    // (gemm_f32_split.cu), and, with the weights read from memory, 17 to 64 rows in 0.4 to 1.06 of the FFMAs' time, more in 0.25 to
    // 0.75 (64 to 65,536 columns, k 128 to 4,096). Not with up to 32 rows, short k and more than a wave of the widest
    // tiles: those wait for the weights, which the FFMA kernel's several CTAs an SM keep coming (17 x 16,384 x 256 15.3 us against 16.2, x
    // 128 8.4 against 11.3; from k 384 on even).
    const bool streams = M <= 32 && K < 384 && N > 148 * 96;
    if (batch == 1 && M > 16 && K >= 128 && !streams) return launch_gemm_f32_split_chosen(ap, wp, op, M, N, K, lda, ldw, ldo, s);
    return launch_gemm_f32(ap, wp, op, M, N, K, lda, ldw, ldo, s, batch, sa, sw, so, -1, 1);
  } else {
    TIE_LAUNCH((gemm_tiled_kernel<TI, TO>), dim3(ceil_div(N, 64), ceil_div(M, 64), batch), 256, 0, s, ap, wp, op, M, N, K, lda, ldw,
               ldo, sa, sw, so);
  }
  TIE_RETURN_LAUNCH("gemm_simt");
}

}  // namespace tie

using namespace tie;

// in_dtype / out_dtype: TIE_F32 or TIE_BF16. Supported: f32->f32, bf16->bf16, bf16->f32.
// lda, ldw, ldo are row strides in elements.
TIE_API int tie_gemm_simt(int in_dtype, int out_dtype, const void* a, const void* w, void* out, int M, int N, int K,
                          long long lda, long long ldw, long long ldo, cudaStream_t s) {
  TIE_REQUIRE(M >= 0 && N >= 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
  TIE_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm: a row stride is smaller than the row");
  if (in_dtype == TIE_F32 && out_dtype == TIE_F32) return launch_gemm<float, float>(a, w, out, M, N, K, lda, ldw, ldo, s);
  if (in_dtype == TIE_BF16 && out_dtype == TIE_BF16)
    return launch_gemm<__nv_bfloat16, __nv_bfloat16>(a, w, out, M, N, K, lda, ldw, ldo, s);
  if (in_dtype == TIE_BF16 && out_dtype == TIE_F32)
    return launch_gemm<__nv_bfloat16, float>(a, w, out, M, N, K, lda, ldw, ldo, s);
  set_error("gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
  return kBadArgument;
}

// `batch` products at once: product b reads a + b * sa and w + b * sw and writes out + b * so (strides in elements).
// With sa = K and so = N inside rows lda and ldo apart, the batch is the heads of a row: out[t, b, :] = w[b] a[t, b, :].
TIE_API int tie_gemm_simt_batched(int in_dtype, int out_dtype, const void* a, const void* w, void* out, int M, int N, int K,
                                  long long lda, long long ldw, long long ldo, int batch, long long sa, long long sw,
                                  long long so, cudaStream_t s) {
  TIE_REQUIRE(M >= 0 && N >= 0 && K > 0 && batch >= 0 && batch <= 65535, "gemm: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
  TIE_REQUIRE(ldw >= K, "gemm: a row stride is smaller than the row");
  if (in_dtype == TIE_F32 && out_dtype == TIE_F32)
    return launch_gemm<float, float>(a, w, out, M, N, K, lda, ldw, ldo, s, batch, sa, sw, so);
  if (in_dtype == TIE_BF16 && out_dtype == TIE_BF16)
    return launch_gemm<__nv_bfloat16, __nv_bfloat16>(a, w, out, M, N, K, lda, ldw, ldo, s, batch, sa, sw, so);
  if (in_dtype == TIE_BF16 && out_dtype == TIE_F32)
    return launch_gemm<__nv_bfloat16, float>(a, w, out, M, N, K, lda, ldw, ldo, s, batch, sa, sw, so);
  set_error("gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
  return kBadArgument;
}

// The float product with its tile and splits of k given (tests): tile 0, 1 or 2 (launch_gemm_f32), splits 1, 2, 4 or 8.
TIE_API int tie_gemm_f32_tiled(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldw,
                               long long ldo, int tile, int splits, cudaStream_t s) {
  TIE_REQUIRE(M > 0 && N > 0 && K > 0 && lda >= K && ldw >= K && ldo >= N, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
  TIE_REQUIRE(tile >= 0 && tile < 3 && (splits == 1 || splits == 2 || splits == 4 || splits == 8), "gemm: tile %d, splits %d", tile, splits);
  return launch_gemm_f32(a, w, out, M, N, K, lda, ldw, ldo, s, 1, 0, 0, 0, tile, splits);
}
