// Any block format for the fused decode + GEMM (gemm_bf16w.cuh), out of the octet decoders of the decode kernel.
#pragma once

#define GGQ_DECODE_GENERIC_LOADS   // blocks are read from shared memory
#include "ggq_decode.cuh"

#include "gemm_bf16w.cuh"

namespace ggq {
namespace gemmb {

// A warp takes eight rows of a superblock, four lanes a row, every fourth octet each; rows are an odd number of 16-byte pieces apart, and the two rows of eight
// consecutive lanes differ in bit 2, so that their 16-byte stores to the swizzled tile fall on different banks.  The decoders take 6 to 13 instructions a weight (the
// K-quants' own above: 3), which the MMAs hide from 300 batch rows on; below, the decode is what bounds.
template <int QT>
struct FGen {
  static constexpr int kBlock = block_elems_of(QT), kBytes = block_bytes_of(QT), kTs = 256 / kBlock * kBytes;
  static constexpr int gcd16(int v) { return v % 16 == 0 ? 16 : v % 8 == 0 ? 8 : v % 4 == 0 ? 4 : v % 2 == 0 ? 2 : 1; }
  static constexpr int kPieces = (16 - gcd16(kTs) + kTs + 15) / 16, kBoxWords = 4 * (kPieces | 1);       // the 16-byte aligned window of a superblock
  static constexpr bool kWholeSuperblock = true, kDirect = true;
  struct Raw {};
  __device__ static int row_of(int warp, int lane) { const int rr = lane >> 2; return 8 * warp + (rr & 1) * 4 + (rr >> 1); }
  // half H of the superblock into the tiles at a0 (stage 2 H) and a1 (stage 2 H + 1)
  template <int H>
  __device__ static void decode(const uint8_t* bytes, uint32_t a0, uint32_t a1, int warp, int lane, const uint8_t* tab) {
    const uint32_t row = (uint32_t)row_of(warp, lane) & 7, j = lane & 3, dst = 1024 * warp + 128 * row;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t e = 128 * H + 32 * i + 8 * j;          // first of the octet's weights
      float v[8];
      Dec<QT>::run(bytes + e / kBlock * kBytes, (e % kBlock) >> 3, tab, v);
      const uint32_t chunk = (4 * i + j) & 7;
      sts_v4((i < 2 ? a0 : a1) + dst + ((chunk ^ row) << 4), pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    }
  }
};

template <int QT>
static cudaError_t launch_generic(const Call& c) {
  using F = FGen<QT>;
  switch (c.plan.mt * 10 + c.plan.cg) {
    case 641: return launch_one<F, 64, 1>(c.w, c.N, c.K, c.x, c.M, c.y, c.y_dtype, c.status, c.plan, c.partials, c.counters, c.tab, c.st);
    case 1281: return launch_one<F, 128, 1>(c.w, c.N, c.K, c.x, c.M, c.y, c.y_dtype, c.status, c.plan, c.partials, c.counters, c.tab, c.st);
    case 2562: return launch_one<F, 256, 2>(c.w, c.N, c.K, c.x, c.M, c.y, c.y_dtype, c.status, c.plan, c.partials, c.counters, c.tab, c.st);
    case 5122: return launch_one<F, 512, 2>(c.w, c.N, c.K, c.x, c.M, c.y, c.y_dtype, c.status, c.plan, c.partials, c.counters, c.tab, c.st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gemmb
}  // namespace ggq
