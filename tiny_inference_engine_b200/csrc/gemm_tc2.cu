// bfloat16 matrix products on pairs of SMs: tcgen05.mma with cta_group::2, out[M, N] = a[M, K] . w[N, K]^T. Two CTAs of a
// cluster compute one tile of 256 rows of the row operand by bn (a multiple of 32 up to 256) rows of the column operand: each
// stages its own 128 rows of the first and its half of the second (32 KB per 64-deep k-block at bn = 256 instead of the 48 KB
// a lone CTA needs for 128 x 256), one thread of the leader issues the MMAs for both, and each CTA's tensor memory receives
// its 128 x bn float accumulator. The tokens are the row operand, or, up to 256 of them, the column operand (`transposed`:
// the weights fill the 256 rows, so 100 tokens are not padded to 256). k may be split: the work items of a launch are
// tiles x splits, float sums per split.
//
// What bounds it, measured at about 2 GHz: a k-block of a tile takes 2 cycles a column on the tensor cores (522 cycles at bn =
// 256, 457 at 224, 428 at 192), or its operands' way from L2 where that is longer, 66 bytes a cycle and SM (360 cycles at bn =
// 128). Around it stand about 1.3 us between two launches, 0.8 of set-up, 0.9 until the first operands land and 2 to 3 for the
// last tile's epilogue, so that short products want every pair busy for few k-blocks: which side, width and split that is,
// ops/gemm_select.py estimates. 512 tokens x 2,560 x 9,728: 31.4 -> 23.2 us (k split three ways on pairs instead of one CTA a
// tile), 128 x 6,144 x 4,096: 15.8 -> 13.4, 2,048 x 19,456 x 2,560 with the SiLU: 163 -> 141 (its epilogue).
//
// Per CTA: warps 0-7 epilogue (tcgen05.ld, optional activation, rows through shared memory and TMA), warp 8 TMA producer,
// warp 9 (leader CTA only) MMA issuer. Barriers: full[s] lives in the leader and counts the
// bytes of BOTH CTAs' loads (the loads carry .cta_group::2 and name the leader's barrier);
// empty[s] and acc_full[b] exist in both CTAs and are signalled by tcgen05.commit with a
// cluster multicast mask; acc_empty[b] lives in the leader and collects the sixteen epilogue
// warps of the pair. A pair walks the work items pair, pair + pairs, ...; two accumulators let a
// tile's epilogue overlap the next tile's MMAs. No TMA multicast: every CTA fetches its own operands.
//
// Waits. Every mbarrier wait is bounded (status word as in gemm_tc.cu), and so is the handshake of the pair
// before it frees its tensor memory (`peer_done`: a remote arrive and a bounded wait, code 4). Three waits have
// no limit, because the instruction set gives them none: tcgen05.alloc (returns once 512 columns are free on both
// SMs; this kernel never shares an SM with another holder of tensor memory, since its 225 KB of shared memory
// exclude every kernel of this library that allocates some), the barrier.cluster right behind it (it waits for
// the partner CTA, which the hardware schedules together with this one and which has nothing ahead of it but the
// same allocation), and griddepcontrol.wait (never executed by this kernel as it is launched, see below).
//
// Programmatic dependent launch: the kernel behind this one may start while it runs (launch_dependents at the
// top), but this kernel itself is launched without the attribute and so starts only when the kernel ahead of it
// has finished. Started early, steps of 512 tokens that mixed two prompt portions with decoded tokens (Qwen3-8B
// shapes: 48 pairs of CTAs for the q/k/v product) hung about once in five runs with no bounded wait expired, so
// in one of the waits named above or in the cluster barrier that used to stand at the end; as it is, hundreds of
// runs of the same steps are clean. The prologue this gives up is two to three microseconds of a
// product. The pdl_wait() below stays (it returns at once for a kernel launched this way) so that the
// order of loads and stores against the kernel ahead does not rest on the launch mode.
#include "umma.cuh"
#include "launchers.h"

namespace tie {

constexpr int k2EpilogueWarps = 8;
constexpr int k2Threads = 32 * (k2EpilogueWarps + 2);
constexpr int k2BK = 64;
constexpr int k2MaxStages = 10;
constexpr int k2StageX = 128 * k2BK * 2;      // this CTA's 128 rows of the row operand; its half of the tile's bn rows of the column operand behind them
constexpr int k2Ring = 6 * 32 * 1024;         // six stages of 32 KB at bn = 256, up to ten of narrower tiles
constexpr int k2Staging = 32 * 1024;          // rows on their way out: 128 rows of 32 columns, 16 KB per group of four epilogue warps
constexpr int k2TmemCols = 512;               // two accumulators of up to 256 columns
constexpr size_t k2Smem = static_cast<size_t>(k2Ring) + k2Staging + 1024 + 256;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The address of `p` (in this CTA's shared memory) as seen in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_cta(const void* p, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_u32(p)), "r"(rank));
  return out;
}
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(leader_bar)
      : "memory");
}
__device__ __forceinline__ void umma2_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far retire.
__device__ __forceinline__ void umma2_commit_both(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}
__device__ __forceinline__ void remote_arrive(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// The same where nothing in memory is handed over: it does not wait for this CTA's stores.
__device__ __forceinline__ void remote_arrive_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// What a launch works on. The row operand x fills the 256-row side of a tile, the column operand y the side of bn.
struct PairArgs {
  void* out;
  float* partial;          // with splits: float sums [splits][tokens][ldp] instead of `out`
  long long part_stride, ldp, ldo;
  int rows_x, rows_y, bn, stages;
  int k_blocks, k_blocks_per_split, tiles_x, n_tiles, n_work;
  int transposed;          // x are the weights and the epilogue writes the tile's transpose
  int epilogue, by_tma;    // by_tma: a tensor map describes the output (or the sums), else rows are stored element by element
  int w_rows, w_row0;
  GatedUnit unit;
  // Grouped (tokens on the row side, k whole): x is group_meta[0] tiles of 256 rows, fewer than the grid was sized for, and row tile t
  // multiplies the rows_y weight rows of group group_of_tile[t], one group's behind the other's in y. Null: one product.
  const int *group_meta, *group_of_tile;
  int* status;
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Where piece p (16 bytes) of a row of 32 columns stands in a warp's part of the staging memory.
template <typename OutT>
__device__ __forceinline__ int piece_at(int row, int p) {
  return sizeof(OutT) == 2 ? (row * 4 + (p ^ ((row >> 1) & 3))) * 16 : (row * 8 + (p ^ (row & 7))) * 16;
}
template <typename OutT, int N>
__device__ __forceinline__ void put_pieces(uint8_t* mine, int row, int first, const float (&v)[N]) {
  constexpr int kPer = 16 / sizeof(OutT);
#pragma unroll
  for (int p = 0; p < N / kPer; ++p) {
    uint8_t* to = mine + piece_at<OutT>(row, first + p);
    if constexpr (sizeof(OutT) == 2)
      *reinterpret_cast<uint4*>(to) = make_uint4(pack_bf16(v[8 * p], v[8 * p + 1]), pack_bf16(v[8 * p + 2], v[8 * p + 3]),
                                                 pack_bf16(v[8 * p + 4], v[8 * p + 5]), pack_bf16(v[8 * p + 6], v[8 * p + 7]));
    else
      *reinterpret_cast<float4*>(to) = make_float4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
  }
}

template <typename OutT>
__global__ void __launch_bounds__(512, 1)      // (launched with 320 threads: 128 registers a thread leave the next kernel some)
gemm_tc2_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
                const __grid_constant__ CUtensorMap map_out, const __grid_constant__ PairArgs g) {
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* staging = smem + k2Ring;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + k2Staging);         // used in the leader
  uint64_t* empty = full + k2MaxStages;                                      // both CTAs
  uint64_t* acc_full = empty + k2MaxStages;                                  // [2], both CTAs
  uint64_t* acc_empty = acc_full + 2;                                        // [2], used in the leader
  uint64_t* peer_done = acc_empty + 2;                                       // both CTAs: the partner is through
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(peer_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int bn = g.bn, stages = g.stages;
  const uint32_t stage_bytes = k2StageX + (bn / 2) * k2BK * 2;
  int* const status = g.status;

  if (warp == 0) {      // a lane a barrier
    if (lane < stages) {
      mbar_init(full + lane, 1);
      mbar_init(empty + lane, 1);
    }
    if (lane < 2) {
      mbar_init(acc_full + lane, 1);
      mbar_init(acc_empty + lane, 2 * k2EpilogueWarps);     // the epilogue warps of both CTAs of the pair
    }
    if (lane == 0) {
      mbar_init(peer_done, 1);
      *abort_flag = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
  }
  if (warp == k2EpilogueWarps && elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_x)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_y)) : "memory");
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  if (warp == k2EpilogueWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(k2TmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // both CTAs' barriers exist before anyone signals across the pair
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;
  pdl_wait();
  int tiles_x = g.tiles_x, n_tiles = g.n_tiles, n_work = g.n_work;
  if (g.group_meta != nullptr) {
    const int tiles_y = n_tiles / tiles_x;
    tiles_x = g.group_meta[0];
    n_tiles = n_work = tiles_x * tiles_y;
  }

  if (warp == k2EpilogueWarps) {
    // ---- TMA producer (both CTAs): own 128 rows of x, own half of the tile's rows of y; bytes count on the leader's
    // barrier. The whole warp walks the loop (uniform) and one elected lane issues.
    int s = 0;
    uint32_t parity = 1;   // a fresh barrier passes a wait on parity 1
    bool ok = true;
    const uint32_t both = 2 * stage_bytes;
    const int x_blocks = g.transposed ? g.w_rows : 0, y_blocks = g.transposed ? 0 : g.w_rows;   // rows of an operand in k-blocks, else 0
    for (int work = pair; work < n_work && ok; work += pairs) {
      const int tile = work % n_tiles, z = work / n_tiles;
      const int row_x = (tile % tiles_x) * 256 + static_cast<int>(rank) * 128 + (x_blocks ? g.w_row0 : 0);
      const int row_y = (tile / tiles_x) * bn + static_cast<int>(rank) * (bn / 2) + (y_blocks ? g.w_row0 : 0) +
                        (g.group_of_tile != nullptr ? g.group_of_tile[tile % tiles_x] * g.rows_y : 0);
      const int kb_end = min(g.k_blocks, (z + 1) * g.k_blocks_per_split);
      for (int kb = z * g.k_blocks_per_split; kb < kb_end; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait(empty + s, parity, abort_flag, status, 1) ? 1 : 0)) {
          ok = false;
          break;
        }
        const uint32_t bar = map_to_cta(full + s, 0);
        uint8_t* sx = smem + s * stage_bytes;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(full + s, both);
          tma_load_2d_pair(sx, &map_x, x_blocks ? 0 : kb * k2BK, kb * x_blocks + row_x, bar);
          tma_load_2d_pair(sx + k2StageX, &map_y, y_blocks ? 0 : kb * k2BK, kb * y_blocks + row_y, bar);
        }
        __syncwarp();
        if (++s == stages) {
          s = 0;
          parity ^= 1;
        }
      }
    }
  } else if (warp == k2EpilogueWarps + 1) {
    // ---- MMA issuer: a warp of the leader CTA walks the loop (uniform), one elected lane drives both CTAs' tensor cores
    if (rank == 0) {
      const uint32_t idesc = instr_desc(bn, 256);
      const uint32_t ring_lo = desc_lo_sw128(smem_u32(smem));   // descriptors as (low word, constant high word)
      int s = 0, local = 0;
      uint32_t parity = 0;
      bool ok = true;
      for (int work = pair; work < n_work && ok; work += pairs, ++local) {
        const int buf = local & 1, z = work / n_tiles;
        const int kb_begin = z * g.k_blocks_per_split, kb_end = min(g.k_blocks, kb_begin + g.k_blocks_per_split);
        if (!__all_sync(0xffffffffu, mbar_wait(acc_empty + buf, ((local >> 1) & 1) ^ 1, abort_flag, status, 2) ? 1 : 0)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_acc = tmem_base + buf * 256;      // the second accumulator at column 256 whatever the width
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!__all_sync(0xffffffffu, mbar_wait(full + s, parity, abort_flag, status, 2) ? 1 : 0)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t x_lo = ring_lo + s * (stage_bytes >> 4), y_lo = x_lo + (k2StageX >> 4);
          const uint32_t keep = kb > kb_begin ? 1u : 0u;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < k2BK / 16; ++k) {
              umma2_bf16(tmem_acc, desc_from_words(x_lo + 2 * k, kDescHiSw128), desc_from_words(y_lo + 2 * k, kDescHiSw128), idesc,
                         k > 0 ? 1u : keep);
            }
            umma2_commit_both(empty + s);
          }
          __syncwarp();
          if (++s == stages) {
            s = 0;
            parity ^= 1;
          }
        }
        if (ok && elect_one()) umma2_commit_both(acc_full + buf);
        __syncwarp();
      }
    }
  } else {
    // ---- epilogue (both CTAs): rows i0 .. i0 + 127 of the pair's tile, all its columns
    const int group = warp >> 2, quarter = warp & 3;
    const bool gated = gated_epilogue(g.epilogue);
    const bool squared = g.epilogue == kEpilogueSquaredRelu && g.partial == nullptr;
    int local = 0;
    for (int work = pair; work < n_work; work += pairs, ++local) {
      const int buf = local & 1;
      const int tile = work % n_tiles, z = work / n_tiles;
      const int i0 = (tile % tiles_x) * 256 + static_cast<int>(rank) * 128, j0 = (tile / tiles_x) * bn;
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full + buf, (local >> 1) & 1, abort_flag, status, 3) ? 1 : 0)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem_base + buf * 256 + (static_cast<uint32_t>(quarter * 32) << 16);
      // This warp has read its last columns of the accumulator: the leader's MMA thread may reuse it once all have. Told
      // before the rows are stored: the arrive waits for stores ahead of it.
      // The last tile's need not be told.
      const bool last = work + pairs >= n_work;
      bool released = last;
      auto release = [&] {
        if (released) return;
        released = true;
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) remote_arrive(map_to_cta(acc_empty + buf, 0));
      };
      if (g.transposed) {
        const int i = i0 + quarter * 32 + lane;
        // out[j, i]: a warp's lanes hold 32 neighbouring i
#pragma unroll 1
        for (int c0 = group * 16; c0 < bn; c0 += 32) {
          if (j0 + c0 >= g.rows_y) break;
          uint32_t r[16];
          tmem_ld16(acc + c0, r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (gated && g.unit.ones > 0 && i0 < g.rows_x && i0 + 128 >= g.rows_x) store_ones(static_cast<OutT*>(g.out), g.ldo, g.rows_x >> 1, g.unit.ones, j0 + c0, min(16, g.rows_y - (j0 + c0)), quarter * 32 + lane);
          if (gated) {
            // lanes 0-15 hold 16 gate rows, lanes 16-31 the matching up rows: exchange, then the lower half finishes
            // columns 0-7 and the upper half columns 8-15
            const bool upper = lane >= 16;
            const int o = (i0 >> 1) + quarter * 16 + (lane & 15);
            const int c1 = j0 + c0 + (upper ? 8 : 0);
            uint32_t gv[8], uv[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? r[e] : r[e + 8], 16);
              gv[e] = upper ? got : r[e];
              uv[e] = upper ? r[e + 8] : got;
            }
            if (o < (g.rows_x >> 1)) {
              float v[8];
              gated_values<8, true, true>(gv, uv, v, g.epilogue, g.unit, g.unit.bias_gate + o, g.unit.bias_up + o);
              OutT* at = static_cast<OutT*>(g.out) + static_cast<long long>(c1) * g.ldo + o;
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (c1 + e < g.rows_y) st(at + e * g.ldo, v[e]);
            }
          } else if (i < g.rows_x) {
            const int n = min(16, g.rows_y - (j0 + c0));
            if (g.partial != nullptr) {
              float* at = g.partial + z * g.part_stride + static_cast<long long>(j0 + c0) * g.ldp + i;
#pragma unroll
              for (int e = 0; e < 16; ++e)
                if (e < n) at[e * g.ldp] = __uint_as_float(r[e]);
            } else {
              OutT* at = static_cast<OutT*>(g.out) + static_cast<long long>(j0 + c0) * g.ldo + i;
#pragma unroll
              for (int e = 0; e < 16; ++e)
                if (e < n) st(at + e * g.ldo, squared ? squared_relu(__uint_as_float(r[e])) : __uint_as_float(r[e]));
            }
          }
        }
      } else {
        // 32 columns of the accumulator at a time (of a gated product 64: 32 output columns), the next ones on their way while
        // these go into shared memory (16-byte pieces exchanged within groups of rows, so that no bank is met twice) and out
        // by TMA, a box of this warp's 32 rows. The last tile's boxes lie in the operand ring, which nothing uses any more, so
        // that none waits for another; and that one fence does for all of them; those of tiles before it take turns in 4 KB of the warp.
        constexpr int kPieces = 2 * sizeof(OutT), kPer = 16 / sizeof(OutT);       // 16-byte pieces of 32 columns, columns of one
        constexpr int kBox = 512 * kPieces, kTurns = 4096 / kBox;                 // bytes of a box, boxes in 4 KB
        const int per = gated ? 64 : 32;
        const int end = min(bn, g.rows_y - j0);       // this tile's columns that exist
        const int i1 = i0 + quarter * 32;
        uint8_t* const base = last ? smem + warp * (k2Ring / k2EpilogueWarps) : staging + warp * 4096;
        // `n` boxes that lie one after the other, of every second 32 output columns from o0 on: one fence, one lane
        auto store_boxes = [&](uint8_t* from, int o0, int n) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            for (int b = 0; b < n && i1 < g.rows_x; ++b) {
              asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];"
                           ::"l"(reinterpret_cast<uint64_t>(&map_out)), "r"(o0 + 64 * b), "r"(i1), "r"(z), "r"(smem_u32(from + b * kBox))
                           : "memory");
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        };
        uint32_t r[32];
        int turn = 0, waiting = 0;
        if (group * per < end) tmem_ld32(acc + group * per, r);
#pragma unroll 1
        for (int c0 = group * per; c0 < end; c0 += 2 * per) {
          const int halves = gated && c0 + 32 < end ? 2 : 1;
          uint8_t* const mine = base + (last ? turn : turn % kTurns) * kBox;
          if (!last && turn >= kTurns) {
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kTurns - 1) : "memory");
            __syncwarp();
          }
          ++turn;
#pragma unroll 1
          for (int h = 0; h < halves; ++h) {
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (gated) {
              float v[16];
              const int column = ((j0 + c0) >> 1) + h * 16;
              gated_values<16, false, true>(r, r + 16, v, g.epilogue, g.unit, g.unit.bias_gate + column, g.unit.bias_up + column);
              const int next = h + 1 < halves ? c0 + 32 : c0 + 2 * per;
              if (next < end) tmem_ld32(acc + next, r);
              else release();
              put_pieces<OutT, 16>(mine, lane, h * (kPieces / 2), v);
            } else {
              float v[32];
#pragma unroll
              for (int e = 0; e < 32; ++e) v[e] = squared ? squared_relu(__uint_as_float(r[e])) : __uint_as_float(r[e]);
              if (c0 + 2 * per < end) tmem_ld32(acc + c0 + 2 * per, r);
              else release();
              put_pieces<OutT, 32>(mine, lane, 0, v);
            }
          }
          const int o0 = gated ? (j0 + c0) >> 1 : j0 + c0;
          if (g.by_tma && (!gated || halves == 2)) {
            if (!last) store_boxes(mine, o0, 1);
            else ++waiting;
          } else {
            // rows that no tensor map describes, and the 16 outputs at the end of a gated tile of 32 (mod 64) columns
            __syncwarp();
            OutT* const out = (g.partial != nullptr ? reinterpret_cast<OutT*>(g.partial + z * g.part_stride) : static_cast<OutT*>(g.out)) + o0;
            const long long out_ld = g.partial != nullptr ? g.ldp : g.ldo;
            const int left = min(16 * halves * (gated ? 1 : 2), (gated ? g.rows_y >> 1 : g.rows_y) - o0);
            if (lane < left) {
              for (int row = 0; row < 32 && i1 + row < g.rows_x; ++row)
                out[(i1 + row) * out_ld + lane] = reinterpret_cast<const OutT*>(mine + piece_at<OutT>(row, lane / kPer))[lane % kPer];
            }
            __syncwarp();
          }
        }
        if (gated && g.unit.ones > 0 && j0 + bn >= g.rows_y && group == 0 && i1 < g.rows_x)
          store_ones(static_cast<OutT*>(g.out), g.ldo, g.rows_y >> 1, g.unit.ones, i1, min(32, g.rows_x - i1), lane);
        if (last) {
          if (waiting > 0) store_boxes(base, (j0 + group * per) >> (gated ? 1 : 0), waiting);
        } else {      // what the next tile writes into the 4 KB has left them by then
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
        }
      }
      release();
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag != 0) {
    const unsigned long long t0 = clock64();
    while (clock64() - t0 < 4000000ull) {
    }
  }
  // Neither CTA leaves, or frees tensor memory, while its partner may still touch its shared or tensor memory:
  // each tells the other that it is through and waits (with the limit of every other wait) to be told. The
  // partner's arrive is its last access to this CTA's memory, and it comes before this wait can return.
  // A CTA that gave up a wait still waits here for its partner, which may need a limit of its own to get
  // here, so this limit is twice the usual one and does not look at the abort flag.
  if (threadIdx.x == 0) {
    remote_arrive_relaxed(map_to_cta(peer_done, rank ^ 1u));
    const unsigned long long t0 = clock64();
    while (!mbar_try_wait(peer_done, 0)) {
      if (clock64() - t0 > 2 * kWaitCycles) {
        *reinterpret_cast<volatile int*>(status) = 4;
        break;
      }
    }
  }
  __syncthreads();
  if (warp == k2EpilogueWarps + 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(k2TmemCols) : "memory");
  }
}

// Pairs of SMs that can hold the kernel at once (SMs pair up inside a GPC, so it may be fewer than half the SMs);
// 0 if the query fails. The same for both instantiations: they differ in neither threads nor shared memory.
static int resident_pairs() {
  static int pairs = -1;
  if (pairs < 0) {
    pairs = 0;
    if (cudaFuncSetAttribute(gemm_tc2_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(k2Smem)) == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.blockDim = dim3(k2Threads);
      cfg.dynamicSmemBytes = k2Smem;
      cfg.gridDim = dim3(2 * 74);
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 2;
      attr.val.clusterDim.y = 1;
      attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, gemm_tc2_kernel<__nv_bfloat16>, &cfg) == cudaSuccess && n >= 1) pairs = n;
      else cudaGetLastError();
    }
  }
  return pairs;
}

template <typename OutT>
static int launch_tc2(const CUtensorMap& mx, const CUtensorMap& my, const CUtensorMap& mo, const PairArgs& g, cudaStream_t s) {
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_tc2_kernel<OutT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(k2Smem)) != cudaSuccess) {
      set_error("gemm_tc2: cannot reserve %zu bytes of shared memory", k2Smem);
      return kCudaError;
    }
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(k2Threads);
  cfg.dynamicSmemBytes = k2Smem;
  cfg.stream = s;
  cudaLaunchAttribute attrs[1];     // the cluster shape and nothing else: no early start (see the top of this file)
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = 2;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 1;
  const int resident = resident_pairs();
  if (resident < 1) {
    set_error("gemm_tc2: no pair of SMs can hold the kernel");
    return kCudaError;
  }
  cfg.gridDim = dim3(2 * (g.n_work < resident ? g.n_work : resident));
  cudaLaunchKernelEx(&cfg, gemm_tc2_kernel<OutT>, mx, my, mo, g);
  return kOk;
}

}  // namespace tie

using namespace tie;

// How many pairs of SMs hold the kernel at once: what the host counts waves of tiles with.
TIE_API int tie_gemm_tc2_pairs() { return resident_pairs(); }

// out[M, N] (or, with a gated unit, silu 1, 2, 4, 5, 6, out[M, N / 2] for w in blocks of 16 gate + 16 up rows: GatedUnit;
// with 3, out[M, N] = max(product, 0)^2)
// = a[M, K] . w[N, K]^T on pairs of SMs. a, w bfloat16 with K and row strides multiples of 8. w_rows > 0: w is
// stored in k-blocks, [ceil(K / 64)][w_rows][64], and the product uses its rows w_row0 .. w_row0 + N - 1 (gemm_tc.cu).
// transposed != 0: the weights fill the tiles' 256-row side. bn: the other side, a multiple of 32 up to 256 (0: 256).
// splits > 1: k is cut, and float sums [real splits][M][N] go to scratch (tie_gemm_tc_real_splits says how many there are): added
// into out by a second kernel, or with reduce == 0 left there for a consumer that adds them itself.
static int gemm_tc2_of(int out_dtype, const void* a, const void* w, void* out, int M, int N, int K, long long lda, long long ldw, long long ldo,
                       int silu, int w_rows, int w_row0, int bn, int transposed, int splits, float* scratch, int reduce, GatedUnit unit,
                       cudaStream_t s) {
  if (bn == 0) bn = 256;
  TIE_REQUIRE(bn >= 32 && bn <= 256 && bn % 32 == 0, "gemm_tc2: tile width %d", bn);
  TIE_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_tc2: bad sizes M=%d N=%d K=%d", M, N, K);
  TIE_REQUIRE(K % 8 == 0 && lda % 8 == 0 && (w_rows > 0 || ldw % 8 == 0), "gemm_tc2: K=%d and the row strides must be multiples of 8", K);
  TIE_REQUIRE(w_rows == 0 || (w_row0 >= 0 && w_row0 + N <= w_rows), "gemm_tc2: rows %d..%d of a weight of %d rows", w_row0, w_row0 + N, w_rows);
  TIE_REQUIRE(reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0,
              "gemm_tc2: operands must be 16-byte aligned");
  TIE_REQUIRE(out_dtype == TIE_BF16 || out_dtype == TIE_F32, "gemm_tc2: output dtype code %d", out_dtype);
  TIE_REQUIRE(silu >= 0 && silu <= kEpilogueBiasedGelu, "gemm_tc2: epilogue %d", silu);
  TIE_REQUIRE(!gated_epilogue(silu) || N % 32 == 0, "gemm_tc2: a gated unit needs weight rows in blocks of 16 gate + 16 up (N=%d)", N);
  TIE_REQUIRE(silu < kEpilogueBiasedSilu || (unit.bias_gate != nullptr && unit.bias_up != nullptr), "gemm_tc2: epilogue %d needs biases", silu);
  TIE_REQUIRE(splits >= 1 && (splits == 1 || scratch != nullptr), "gemm_tc2: splits=%d needs scratch memory", splits);
  TIE_REQUIRE(splits == 1 || silu == 0 || (silu == kEpilogueSquaredRelu && reduce),
              "gemm_tc2: epilogue %d of a split product (the squared ReLU needs the reduction here)", silu);
  if (splits == 1) scratch = nullptr;
  TIE_REQUIRE(status_word() != nullptr, "gemm_tc2: cannot allocate the status word");
  PairArgs g = {};
  g.transposed = transposed != 0;
  g.rows_x = transposed ? N : M;
  g.rows_y = transposed ? M : N;
  g.bn = bn;
  const int stage = k2StageX + (bn / 2) * k2BK * 2;
  g.stages = k2Ring / stage < k2MaxStages ? k2Ring / stage : k2MaxStages;
  g.k_blocks = ceil_div(K, k2BK);
  g.k_blocks_per_split = ceil_div(g.k_blocks, splits);
  const int real = ceil_div(g.k_blocks, g.k_blocks_per_split);
  g.tiles_x = ceil_div(g.rows_x, 256);
  g.n_tiles = g.tiles_x * ceil_div(g.rows_y, bn);
  g.n_work = g.n_tiles * real;
  g.out = out;
  g.partial = scratch;
  g.part_stride = static_cast<long long>(M) * N;
  g.ldp = N;
  g.ldo = ldo;
  g.epilogue = silu;
  g.unit = unit;
  if (!gated_epilogue(silu)) g.unit.ones = 0;
  g.w_rows = w_rows;
  g.w_row0 = w_row0;
  g.status = status_word();
  CUtensorMap mw, ma, mo;
  const int rows_of_w = transposed ? 128 : bn / 2, rows_of_a = transposed ? bn / 2 : 128;
  const bool w_ok = w_rows > 0 ? make_map_bf16(&mw, w, static_cast<long long>(g.k_blocks) * w_rows, k2BK, k2BK, k2BK, rows_of_w)
                               : make_map_bf16(&mw, w, N, K, ldw, k2BK, rows_of_w);
  TIE_REQUIRE(make_map_bf16(&ma, a, M, K, lda, k2BK, rows_of_a) && w_ok, "gemm_tc2: cuTensorMapEncodeTiled failed (M %d, N %d, K %d)", M, N, K);
  const bool as_float = scratch != nullptr || out_dtype == TIE_F32;
  g.by_tma = !transposed && make_map_rows(&mo, scratch != nullptr ? scratch : out, as_float, M, gated_epilogue(silu) ? N / 2 : N,
                                          scratch != nullptr ? N : ldo, scratch != nullptr ? real : 1, 32, 32);
  if (!g.by_tma) mo = ma;
  const CUtensorMap &mx = transposed ? mw : ma, &my = transposed ? ma : mw;
  const int st = as_float ? launch_tc2<float>(mx, my, mo, g, s) : launch_tc2<__nv_bfloat16>(mx, my, mo, g, s);
  if (st != kOk) return st;
  if (scratch != nullptr && reduce) launch_splitk_reduce(out_dtype, scratch, g.part_stride, real, out, ldo, N, g.part_stride, silu, s);
  TIE_RETURN_LAUNCH("gemm_tc2");
}

TIE_API int tie_gemm_tc2(int out_dtype, const void* a, const void* w, void* out, int M, int N, int K, long long lda, long long ldw, long long ldo,
                         int silu, int w_rows, int w_row0, int bn, int transposed, int splits, float* scratch, int reduce, cudaStream_t s) {
  return gemm_tc2_of(out_dtype, a, w, out, M, N, K, lda, ldw, ldo, silu, w_rows, w_row0, bn, transposed, splits, scratch, reduce, GatedUnit{}, s);
}

// The same with what a gated unit takes beside its code (GatedUnit).
TIE_API int tie_gemm_tc2_unit(int out_dtype, const void* a, const void* w, void* out, int M, int N, int K, long long lda, long long ldw,
                              long long ldo, int silu, int w_rows, int w_row0, int bn, int transposed, int splits, float* scratch, int reduce,
                              const float* bias_gate, const float* bias_up, float limit, float slope, float up_shift, int ones, cudaStream_t s) {
  return gemm_tc2_of(out_dtype, a, w, out, M, N, K, lda, ldw, ldo, silu, w_rows, w_row0, bn, transposed, splits, scratch, reduce,
                     GatedUnit{bias_gate, bias_up, limit, slope, up_shift, ones}, s);
}

// Grouped product: a [M_cap, K] holds `meta[0]` tiles of 256 rows (M_cap is what the buffers were sized for); tile t multiplies the N weight
// rows of group `group_of_tile[t]`, and out[M_cap, N] (or, with a gated unit's epilogue, out[M_cap, N / 2]) gets the rows in the same order. w
// is stored in k-blocks, [ceil(K / 64)][w_rows][64], group g's rows at g * N .. g * N + N - 1 (w_rows = groups * N). meta and group_of_tile
// live on the device and may be written by the kernel right ahead of this one. (On single SMs, tiles of 128 rows, 6,124 pairs over 32
// experts of 3,072 x 2,048 took 130 us.)
TIE_API int tie_gemm_tc2_grouped(int out_dtype, const void* a, const void* w, void* out, int M_cap, int N, int K, long long lda, long long ldo,
                                 int w_rows, int epilogue, float limit, float slope, float up_shift, const int* meta, const int* group_of_tile,
                                 cudaStream_t s) {
  TIE_REQUIRE(M_cap > 0 && M_cap % 256 == 0 && N > 0 && K > 0, "gemm_tc2_grouped: bad sizes M=%d (whole tiles of 256) N=%d K=%d", M_cap, N, K);
  TIE_REQUIRE(K % 8 == 0 && lda % 8 == 0 && w_rows >= N && w_rows % N == 0, "gemm_tc2_grouped: K=%d, lda and the weight's %d rows", K, w_rows);
  TIE_REQUIRE(reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0, "gemm_tc2_grouped: operands must be 16-byte aligned");
  TIE_REQUIRE(out_dtype == TIE_BF16 || out_dtype == TIE_F32, "gemm_tc2_grouped: output dtype code %d", out_dtype);
  TIE_REQUIRE((epilogue == 0 || epilogue == kEpilogueClamped) && (epilogue == 0 || N % 32 == 0), "gemm_tc2_grouped: epilogue %d (N=%d)", epilogue, N);
  TIE_REQUIRE(meta != nullptr && group_of_tile != nullptr && status_word() != nullptr, "gemm_tc2_grouped: no tile list");
  PairArgs g = {};
  g.rows_x = M_cap;
  g.rows_y = N;
  g.bn = N >= 256 ? 256 : ceil_div(N, 32) * 32;
  const int stage = k2StageX + (g.bn / 2) * k2BK * 2;
  g.stages = k2Ring / stage < k2MaxStages ? k2Ring / stage : k2MaxStages;
  g.k_blocks = g.k_blocks_per_split = ceil_div(K, k2BK);
  g.tiles_x = M_cap / 256;
  g.n_tiles = g.n_work = g.tiles_x * ceil_div(N, g.bn);
  g.out = out;
  g.ldo = ldo;
  g.epilogue = epilogue;
  g.w_rows = w_rows;
  g.unit = GatedUnit{nullptr, nullptr, limit, slope, up_shift, 0};
  g.group_meta = meta;
  g.group_of_tile = group_of_tile;
  g.status = status_word();
  CUtensorMap ma, mw, mo;
  TIE_REQUIRE(make_map_bf16(&ma, a, M_cap, K, lda, k2BK, 128) &&
                  make_map_bf16(&mw, w, static_cast<long long>(g.k_blocks) * w_rows, k2BK, k2BK, k2BK, g.bn / 2),
              "gemm_tc2_grouped: cuTensorMapEncodeTiled failed (rows %d, K %d)", M_cap, K);
  const bool as_float = out_dtype == TIE_F32;
  g.by_tma = make_map_rows(&mo, out, as_float, M_cap, epilogue ? N / 2 : N, ldo, 1, 32, 32);
  if (!g.by_tma) mo = ma;
  const int st = as_float ? launch_tc2<float>(ma, mw, mo, g, s) : launch_tc2<__nv_bfloat16>(ma, mw, mo, g, s);
  if (st != kOk) return st;
  TIE_RETURN_LAUNCH("gemm_tc2_grouped");
}
