// What the recurrence kernels share: the layer's sizes, and the convolution's inputs that a slot keeps behind its state.
#pragma once

#include "common.cuh"

namespace tie {

struct DeltaShape {
  int heads, kv_heads, dim, vdim, taps;
  int channels() const { return 2 * kv_heads * dim + heads * vdim; }
};

// The convolution's last taps - 1 inputs after a step of n tokens from row t0 on: from the step's rows where it brought enough, else
// what the slot held moves up. Block `mine` of the `blocks` of a sequence takes a slice of the channels.
template <typename T>
__device__ __forceinline__ void move_conv_tail(const DeltaShape& sh, float* tail, const T* __restrict__ proj, long long proj_stride, int q_off,
                                               int k_off, int v_off, int t0, int n, int mine, int blocks) {
  if (sh.taps <= 1) return;
  const int nqk = sh.kv_heads * sh.dim, C = 2 * nqk + sh.heads * sh.vdim, keep = sh.taps - 1;
  const int per = (C + blocks - 1) / blocks;
  const int c_end = min(C, (mine + 1) * per);
  for (int c = mine * per + threadIdx.x; c < c_end; c += blockDim.x) {
    const int pc = c < nqk ? q_off + c : (c < 2 * nqk ? k_off + (c - nqk) : v_off + (c - 2 * nqk));
    for (int i = 0; i < keep; ++i) {
      const int from = n - keep + i;        // offset in the step of the token that lands at place i
      tail[static_cast<long long>(i) * C + c] = from >= 0 ? ld(proj + (t0 + from) * proj_stride + pc)
                                                          : tail[static_cast<long long>(n + i) * C + c];
    }
  }
}

}  // namespace tie
