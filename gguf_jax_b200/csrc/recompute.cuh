// Outputs of the tensor-core kernels that are not finite, computed once more from the decoded weights.
#pragma once

#include "gemv.cuh"
#include "ggq_decode.cuh"

namespace ggq {

// The kernels on the tensor cores take a weight apart (into codes and multiples of sum(x), or into three bf16 terms of which the
// last are often zero), so an activation or a scale that is infinite, or a sum that leaves the float32 range on the way,
// makes their result NaN where the product of the decoded weights is not.  Such an output is computed once more the plain
// way, float32 weights of the block decoders times the activations, by all lanes of the warp that has it, after it was stored
// like the others; a batch row with a NaN in it needs no weights.  us with one lane per output, walking the whole row -> this way:
// IQ2_XS 8192 x 28672 at batch 1 (47 with finite activations) with one NaN 2417 -> 70, one infinity 2414 -> 818; Q8_0 14336 x 4096
// at 16 rows (47) 235 -> 51, 235 -> 94.
static __device__ __noinline__ bool has_nan(const __nv_bfloat16* xrow, int K) {
  bool nan = false;
#pragma unroll 4
  for (int e = 8 * (threadIdx.x & 31); e < K; e += 256) {
    const uint4 v = *reinterpret_cast<const uint4*>(xrow + e);
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) nan |= (u[i] & 0x7FFF0000u) > 0x7F800000u || (u[i] << 16 & 0x7FFF0000u) > 0x7F800000u;
  }
  return __any_sync(0xFFFFFFFFu, nan);
}
template <int QT>
__device__ __noinline__ float exact_dot(const uint8_t* wrow, const __nv_bfloat16* xrow, int K, const uint8_t* tab) {
  constexpr int BS = block_elems_of(QT), TS = block_bytes_of(QT);
  // the row into the L2 first, so that the rounds of loads below are short ones
  for (int64_t b = 128 * (threadIdx.x & 31); b < (int64_t)(K / BS) * TS; b += 128 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(wrow + b));
  float acc = 0.f;
#pragma unroll 4
  for (int e = 8 * (threadIdx.x & 31); e < K; e += 256) {
    float v[8];
    Dec<QT>::run(wrow + (int64_t)(e / BS) * TS, (e % BS) >> 3, tab, v);
#pragma unroll
    for (int i = 0; i < 8; i++) acc = fmaf(v[i], __bfloat162float(xrow[e + i]), acc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
  return acc;
}
// Called by all lanes of a warp: the outputs (row, m) of the lanes with `bad` set.
template <int QT>
__device__ __noinline__ void recompute(bool bad, int row, int m, const uint8_t* w, int64_t row_bytes, int N, const __nv_bfloat16* x, int K,
                                       const uint8_t* tab, void* y, int y_dtype) {
  uint32_t nan_rows = 0, seen = 0;
  for (uint32_t lanes = __ballot_sync(0xFFFFFFFFu, bad); lanes; lanes &= lanes - 1) {
    const int src = __ffs(lanes) - 1, r = __shfl_sync(0xFFFFFFFFu, row, src), mr = __shfl_sync(0xFFFFFFFFu, m, src);
    const __nv_bfloat16* xrow = x + (int64_t)mr * K;
    if (!((seen >> mr) & 1)) { seen |= 1u << mr; nan_rows |= (uint32_t)has_nan(xrow, K) << mr; }
    const float v = ((nan_rows >> mr) & 1) ? __uint_as_float(0x7FFFFFFFu) : exact_dot<QT>(w + r * row_bytes, xrow, K, tab);
    if ((threadIdx.x & 31) == src) store_out(y, y_dtype, (int64_t)mr * N + r, v);
  }
}
// An output as it was stored (by a lane of this warp).
__device__ __forceinline__ float load_out(const void* y, int y_dtype, int64_t idx) {
  if (y_dtype == GGQ_F32) return reinterpret_cast<const volatile float*>(y)[idx];
  const uint32_t u = reinterpret_cast<const volatile unsigned short*>(y)[idx];
  return y_dtype == GGQ_BF16 ? __uint_as_float(u << 16) : __half2float(__ushort_as_half((unsigned short)u));
}
__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) <= 3.402823466e38f); }

}  // namespace ggq
