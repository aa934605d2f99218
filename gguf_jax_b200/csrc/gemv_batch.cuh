// Fused decode + multiply for up to 16 batch rows per launch on B200 (ggq_gemv calls it from 3 on): the formats of batch_formats.cuh (one float scale per block of 256).
//
// Arithmetic.  mma.sync.m16n8k16 with float16 operands: A = 16 weight rows x 16 weights as exact integers (group scale times code),
// B = 16 activations of eight batch rows (one or two column tiles share the decoded A).  The integers of a whole block add up in
// one accumulator per output; the block's float scale is applied once per block, and a block's offsets (dmin) are two or three more MMAs
// on bfloat16 pairs (the 4- or 6-bit mins times the group sums of x, split into three terms of 8 bits).
// Activations are bfloat16 and are staged as float16 times a power of two that puts the largest magnitude of a batch row and block just
// below 2^15.  Eight significant bits are exact down to 2^-17, so magnitudes within 2^32 of the block's largest are exact; smaller ones are
// left out of the staged copy and multiplied in further passes over the block (planes), straight from x: no activation is rounded.  (Their
// sums are in units of the block's largest: 2^120 below it they reach the end of the float32 range.)
//
// Work split.  A cluster of Q CTAs owns a contiguous range of 16-row tiles, and each of its CTAs a Q-th of K (in P passes, where the
// activations of one do not fit): the CTA stages its share of the activations once and deals its steps (16 rows x nb blocks, tile by tile)
// to its sixteen warps as equal contiguous ranges.  A warp copies its own steps through a private ring (a TMA box of 16 rows per step, or
// cp.async of the 16-byte windows around rows that are not 16-byte aligned), keeps the 16 x 8 NT sums of a tile in registers and leaves
// them in shared memory when the tile or its range ends; after a cluster barrier each CTA adds up a Q-th of the tiles, over the warps and
// the cluster's CTAs in a fixed order, and stores the outputs.  No scratch, no counters, no atomics: a launch is deterministic.
// (Partial sums through global memory, one arrival counter per row tile, took 2 us more on small weights for the fence, the atomic and the
// read back, and staged more activations per CTA.)
// What bounds it: 8192 x 8192 Q4_K at 8 rows takes 17 us (5.8 us of HBM): issue slots 47 % busy, the half-rate integer pipe (codes out of
// bytes) 41 %, the tensor pipe 10 %, four warps per scheduler at 128 registers and no stall above an eighth of the time.  The kernels before it
// kept groups apart (an MMA for two batch rows, or a pair of them per scale group and column tile, with a scale on every partial sum):
// us before / here at 8 and 16 rows, Q4_K 23.9 / 17.4, 27.0 / 21.5; IQ3_S 37.3 / 22.7, 82.4 / 30.1; Q6_K 29.9 / 24.6, 33.0 / 30.8; IQ3_S
// 8192 x 28672 93 / 68, 186 / 91; 5003 x 2816 Q6_K at 5 rows 18.0 / 10.9.
#pragma once

#include "gemv_tile.cuh"
#include "batch_formats.cuh"

namespace ggq {
namespace batch {

using tile::cp_async16;
using tile::cp_async_commit;
using tile::cp_async_wait_pending;

constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kMaxDepth = 6;
constexpr int kMaxBatch = 16;

struct Geo {
  int nb, spu, chunk_sb;            // blocks per step, steps per unit (a tile in one pass), blocks per pass
  int Q, P, J, RT, tile0;           // CTAs per cluster, passes, clusters, 16-row tiles of the launch and the first of them
  int depth, pitch, slot_bytes;     // ring of a warp
  int off_x, off_sum, off_tab, off_misc, off_bar, total;
  int tma;                          // steps come as TMA boxes
  int row_skew;                     // bytes by which consecutive rows differ modulo 16
};

template <class F> constexpr int mins_bytes() { return F::kMins == 0 ? 0 : F::kMins == 2 ? 512 : 768; }
// Staged activations of one block and eight batch rows: 8 octets x 32 lanes x 16 bytes, the sums' fragments, eight factors.
template <class F> constexpr int x_tile_bytes() { return 4096 + mins_bytes<F>() + 32; }

// Steps of a CTA and pass: T; first step of warp v (0 .. 16), and the warp that has step s.
__host__ __device__ __forceinline__ int warp_begin(int T, int v) { return T * v / kWarps; }
__host__ __device__ __forceinline__ int warp_of(int T, int s) { return ((s + 1) * kWarps - 1) / T; }
__host__ __device__ __forceinline__ int first_tile(const Geo& g, int j) { return g.tile0 + (int)((int64_t)g.RT * j / g.J); }

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_half(float lo, float hi) {
  const __half2 p = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}
// Packed pairs of floats.
__device__ __forceinline__ void mul2(float& a, float& b, float x0, float x1, float y0, float y1) {
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\tmul.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}"
      : "=f"(a), "=f"(b) : "f"(x0), "f"(x1), "f"(y0), "f"(y1));
}
__device__ __forceinline__ void fma2(float& a, float& b, float x0, float x1, float y0, float y1) {
  asm("{\n\t.reg .b64 p, q, r;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\tmov.b64 r, {%0, %1};\n\tfma.rn.f32x2 r, p, q, r;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "+f"(a), "+f"(b) : "f"(x0), "f"(x1), "f"(y0), "f"(y1));
}
__device__ __forceinline__ uint32_t exponent_of(float v) { return (__float_as_uint(v) >> 23) & 0xFF; }

// Eight activations (quads a and b of an octet) as floats.
struct Octet {
  float v[8];
  __device__ __forceinline__ Octet(uint2 a, uint2 b)
      : v{tile::bf16lo(a.x), tile::bf16hi(a.x), tile::bf16lo(a.y), tile::bf16hi(a.y), tile::bf16lo(b.x), tile::bf16hi(b.x), tile::bf16lo(b.y),
          tile::bf16hi(b.y)} {}
  template <int PAIR_ORDER>
  __device__ __forceinline__ uint4 fragment(float up) const {
    constexpr int kA[4] = {0, 1, PAIR_ORDER ? 2 : 4, PAIR_ORDER ? 3 : 5}, kB[4] = {PAIR_ORDER ? 4 : 2, PAIR_ORDER ? 5 : 3, 6, 7};
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      float a, b;
      mul2(a, b, v[kA[i]], v[kB[i]], up, up);
      r[i] = pack_half(a, b);
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
  }
};

// A block's product with the activations of eight batch rows (x, M of them) that the staged copy leaves out: plane p has those whose
// exponent is 32 p to 32 p + 31 below the largest of their batch row.  Adds the sums to acc.  Rare, so nothing of it is kept in registers.
template <class F>
__device__ __noinline__ void more_planes(uint32_t blk0, uint32_t blk1, tf::Tables tb, const __nv_bfloat16* x, int M, int K, int k0,
                                         uint32_t fac_addr, int planes, float* acc) {
  typedef typename F::Base B;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t eb = exponent_of(tile::lds_f32(fac_addr + 4 * g)) + 4;      // biased exponent of the batch row's largest
  for (int p = 1; p <= planes; p++) {
    float part[4] = {0.f, 0.f, 0.f, 0.f};
    typename F::Run run0, run1;
    bf::load_pair<F>(tf::BlockLd{blk0}, tf::BlockLd{blk1}, t, run0, run1);
#pragma unroll
    for (int q = 0; q < 8; q++) {
      uint32_t a0[4], b0[4], a1[4], b1[4];
      F::octet(run0, q, tb, a0, b0);
      F::octet(run1, q, tb, a1, b1);
      int qa, qb;
      F::src_quads(t, q, qa, qb);
      uint2 va = make_uint2(0, 0), vb = make_uint2(0, 0);
      if (g < M) {
        va = __ldcg(reinterpret_cast<const uint2*>(x + (int64_t)g * K + k0 + qa));
        vb = __ldcg(reinterpret_cast<const uint2*>(x + (int64_t)g * K + k0 + qb));
      }
      Octet o(va, vb);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if ((int)(eb - exponent_of(o.v[i])) >> 5 != p) o.v[i] = 0.f;
        for (int j = 0; j < p; j++) o.v[i] *= 4294967296.0f;
      }
      __syncwarp();
      const uint4 xv = o.template fragment<B::kPairOrder>(__uint_as_float((268 - eb) << 23));
      mma_f16(part, a0[0], a1[0], a0[1], a1[1], xv.x, xv.y);
      mma_f16(part, a0[2], a1[2], a0[3], a1[3], xv.z, xv.w);
      if constexpr (F::kPlanes == 2) {
        mma_f16(part, b0[0], b1[0], b0[1], b1[1], xv.x, xv.y);
        mma_f16(part, b0[2], b1[2], b0[3], b1[3], xv.z, xv.w);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      for (int j = 0; j < p; j++) part[i] *= 2.3283064365386963e-10f;
      acc[i] += part[i];
    }
  }
}

template <class F, int NT>
__global__ void __launch_bounds__(kThreads, 1)
gemv_batch_kernel(const uint8_t* __restrict__ w, int N, int K, const __nv_bfloat16* __restrict__ x, int M, void* __restrict__ y, int y_dtype,
                  const Geo geo, const uint8_t* __restrict__ tab, int* __restrict__ status, const __grid_constant__ CUtensorMap map) {
  typedef typename F::Base B;
  constexpr int XR = 8 * NT, kXTile = x_tile_bytes<F>(), kXBlock = NT * kXTile;
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);           // uniform, and known to be
  const int g = lane >> 2, t = lane & 3;
  const int SB = K / 256;
  const uint32_t row_bytes = (uint32_t)SB * B::kTs;                 // N rows take less than 2^31 bytes
  const int nb = geo.nb, spu = geo.spu, depth = geo.depth, pitch = geo.pitch;

  // ---- this CTA's tiles and part of K, this warp's steps of a pass: step s = (tile rt, position k)
  const int rank = blockIdx.x % geo.Q, tile_lo = first_tile(geo, blockIdx.x / geo.Q), tiles = first_tile(geo, blockIdx.x / geo.Q + 1) - tile_lo;
  const int T = tiles * spu, s_begin = warp_begin(T, warp), pass_steps = warp_begin(T, warp + 1) - s_begin;
  const int rt0 = s_begin / spu, k0 = s_begin - rt0 * spu;

  // ---- copy side
  const uint32_t smem_base = tile::smem_u32(smem);
  const uint32_t my_ring = smem_base + warp * (depth * geo.slot_bytes);
  const uint32_t my_bars = smem_base + geo.off_bar + warp * (8 * kMaxDepth);
  if (geo.tma) tma_bars_init(my_bars, depth, lane);
  const int hl = lane >> 4, kl = lane & 15;
  int to_issue = pass_steps * geo.P, left_i = pass_steps, slot_i = 0, sbc_i = rank * geo.P * geo.chunk_sb, rt_i = rt0, k_i = k0;
  auto issue_next = [&]() {
    if (to_issue > 0) {
      const int sb0 = sbc_i + k_i * nb;
      const uint32_t dst = my_ring + slot_i * geo.slot_bytes, boff = (uint32_t)sb0 * B::kTs;
      if (geo.tma) {
        // the window of the step's blocks that starts on a 16-byte boundary; rows and blocks past the end arrive as zeros
        if (lane == 0) tma_box_load(dst, &map, (int)((boff & ~15u) >> 2), (tile_lo + rt_i) * 16, my_bars + 8 * slot_i, geo.slot_bytes);
      } else {
        // a half-warp copies a row, lane kl the 16-byte pieces kl and kl + 16 of its window; rows past the end repeat row N - 1
        // (multiplied, never stored); a copied piece holds at least one byte of its row
        const int nbh = min(nb, SB - sb0);
        static_assert(14 + 2 * B::kTs + 15 <= 512, "two pieces per lane cover a window of two blocks");
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const uint32_t off = (uint32_t)min((tile_lo + rt_i) * 16 + 2 * i + hl, N - 1) * row_bytes + boff;
          const int pieces = nbh > 0 ? ((off & 15) + nbh * B::kTs + 15) >> 4 : 0;
          const uint8_t* src = w + (off & ~15u) + 16 * kl;
          const uint32_t to = dst + (2 * i + hl) * pitch + 16 * kl;
          if (kl < pieces) cp_async16(to, src);
          if (kl + 16 < pieces) cp_async16(to + 256, src + 256);
        }
      }
      --to_issue;
      if (++slot_i == depth) slot_i = 0;
      if (++k_i == spu) { k_i = 0; ++rt_i; }
      if (--left_i == 0) { left_i = pass_steps; rt_i = rt0; k_i = k0; sbc_i += geo.chunk_sb; }
    }
    if (!geo.tma) cp_async_commit();
  };

  // ---- look-up tables (immutable), as in the tiled kernel; the code book's byte pairs are signed here
  tf::Tables tb{};
  constexpr bool kGrid = B::kTableBytes > 0 && tf::KvOf<B>::value == 0;
  [[maybe_unused]] uint32_t grid_v[tile::GridFill<B>::kRounds][2];
  if constexpr (kGrid) {
    constexpr int kEW = B::kEntryBytes / 4;
    constexpr int kOff = B::kQt == QT_IQ1_S || B::kQt == QT_IQ1_M ? TAB_IQ1 : B::kQt == QT_IQ2_XXS ? TAB_IQ2_XXS :
                         B::kQt == QT_IQ2_XS ? TAB_IQ2_XS : B::kQt == QT_IQ2_S ? TAB_IQ2_S : B::kQt == QT_IQ3_XXS ? TAB_IQ3_XXS : TAB_IQ3_S;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(tab + kOff);
#pragma unroll
    for (int j = 0; j < tile::GridFill<B>::kRounds; j++) {
      const int e = (tid + j * kThreads) / tile::GridFill<B>::kPieces;
      if constexpr (kEW == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(src) + e);
        grid_v[j][0] = v.x; grid_v[j][1] = v.y;
      } else grid_v[j][0] = grid_v[j][1] = __ldg(src + e);
    }
  }
  for (int d = 0; d < depth - 1; d++) issue_next();
  if constexpr (kGrid) {
    tb.grid = smem_base + geo.off_tab + (lane % B::kCopies) * B::kEntryBytes;
    uint4* dst = reinterpret_cast<uint4*>(smem + geo.off_tab);
#pragma unroll
    for (int j = 0; j < tile::GridFill<B>::kRounds; j++) {
      uint32_t v[2] = {grid_v[j][0], grid_v[j][1]};
      if constexpr (B::kQt == QT_IQ1_S || B::kQt == QT_IQ1_M) {
#pragma unroll
        for (int h = 0; h < 2; h++) {            // int8 grid {-1, 0, 1} -> code bytes 8 * grid + 9
          const uint32_t neg = (v[h] >> 7) & 0x01010101u, pos = v[h] & ~(v[h] >> 7) & 0x01010101u;
          v[h] = 0x09090909u - 8u * neg + 8u * pos;
        }
      }
      dst[tid + j * kThreads] = make_uint4(v[0], v[1], v[0], v[1]);
    }
    if constexpr (B::kSignTable) {
      constexpr int kGridBytes = B::kEntries * B::kEntryBytes * B::kCopies;
      tb.sign = smem_base + geo.off_tab + kGridBytes + (lane % tf::kSignCopies) * 8;
      uint4* sd = reinterpret_cast<uint4*>(smem + geo.off_tab + kGridBytes);
      for (int i = tid; i < (1 << B::kSignBits) * (tf::kSignCopies / 2); i += kThreads) {
        const uint32_t bits = tf::sign_bits_of(B::kSignBits, (uint32_t)i / (tf::kSignCopies / 2));
        const uint32_t s0 = tf::spread_signs4(bits), s1 = tf::spread_signs4(bits >> 4);
        sd[i] = make_uint4(s0, s1, s0, s1);
      }
    }
  }
  if constexpr (tf::KvOf<B>::value == 1) {
    const int8_t* kv = reinterpret_cast<const int8_t*>(tab + TAB_KV_IQ4);
    tb.grid = smem_base + geo.off_tab + (lane % tf::kByteTableCopies) * 4;
    uint4* dst = reinterpret_cast<uint4*>(smem + geo.off_tab);
    for (int i = tid; i < 256 * (tf::kByteTableCopies / 4); i += kThreads) {
      const int e = i / (tf::kByteTableCopies / 4), lo = __ldg(kv + (e & 15)), hi = __ldg(kv + (e >> 4));
      const uint32_t v = (uint32_t)(lo < 0 ? 0x8000 - lo : lo) | (uint32_t)(hi < 0 ? 0x8000 - hi : hi) << 16;
      dst[i] = make_uint4(v, v, v, v);
    }
  }
  int* planes = reinterpret_cast<int*>(smem + geo.off_misc);        // further planes of every staged block, then: whether there are any
  float4* sums = reinterpret_cast<float4*>(smem + geo.off_sum);
  // A segment is what a warp does of a tile; segments are numbered by tile + warp, which grows from each to the next.
  auto sum_at = [&](int seg) { return (uint32_t)(seg * (32 * NT) + lane); };

  // ---- everything below reads or writes memory the previous kernel may still be using
  pdl_wait();
  int slot = 0;
  uint32_t phase = 0;
  for (int pass = 0; pass < geo.P; pass++) {
    const int sb_lo = (rank * geo.P + pass) * geo.chunk_sb, sb_n = max(0, min(SB - sb_lo, geo.chunk_sb));
    __syncthreads();         // tables written; the previous pass's activations are read
    for (int i = tid; i <= geo.chunk_sb; i += kThreads) planes[i] = 0;
    __syncthreads();
    // Staging: a warp takes one batch row of one block at a time, lane 8 t + q octet q of run t; four rounds' loads are in flight.
    {
      const int items = sb_n * XR, q = lane & 7, tt = lane >> 3;
      int qa, qb;
      F::src_quads(tt, q, qa, qb);
      constexpr int kAhead = 4;
      for (int base = warp; base < items; base += kWarps * kAhead) {
        uint4 v4[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
          const int it = base + j * kWarps, m = it % XR, sb = sb_lo + it / XR;
          v4[j] = make_uint4(0, 0, 0, 0);
          if (it < items && m < M) {
            const __nv_bfloat16* xr = x + (int64_t)m * K + (int64_t)sb * 256;
            if constexpr (B::kPairOrder == 0) v4[j] = __ldcg(reinterpret_cast<const uint4*>(xr + qa));      // quads side by side
            else {
              const uint2 va = __ldcg(reinterpret_cast<const uint2*>(xr + qa)), vb = __ldcg(reinterpret_cast<const uint2*>(xr + qb));
              v4[j] = make_uint4(va.x, va.y, vb.x, vb.y);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
          const int it = base + j * kWarps;
          if (it >= items) break;
          const int m = it % XR, blk = it / XR;
          // largest and smallest non-zero magnitude, as pairs of halves with the top bit set (less one for the smallest: a zero is then
          // the largest signed half)
          const uint32_t u0 = v4[j].x | 0x80008000u, u1 = v4[j].y | 0x80008000u, u2 = v4[j].z | 0x80008000u, u3 = v4[j].w | 0x80008000u;
          uint32_t top = __vmaxu2(__vmaxu2(u0, u1), __vmaxu2(u2, u3));
          uint32_t low = __vmins2(__vmins2(u0 - 0x00010001u, u1 - 0x00010001u), __vmins2(u2 - 0x00010001u, u3 - 0x00010001u));
          top = __reduce_max_sync(0xFFFFFFFFu, max(top >> 16, top & 0xFFFFu)) & 0x7FFFu;
          // (above 0x7F80, a NaN, the exponent is 255 all the same)
          const uint32_t eb = max(top >> 7, 17u);
          const int least = min((int)(short)(low & 0xFFFFu), (int)low >> 16) + 32769;      // magnitude bits, 65536 for zeros only
          uint8_t* xt = smem + geo.off_x + blk * kXBlock + (m >> 3) * kXTile;
          const float up = __uint_as_float((268 - eb) << 23);          // 2^(14 - E)
          Octet o(make_uint2(v4[j].x, v4[j].y), make_uint2(v4[j].z, v4[j].w));
          if constexpr (F::kMins > 0) {
            // sums of the run's groups in the staged scale, as three bfloat16 terms
            float sum = ((o.v[0] + o.v[1]) + (o.v[2] + o.v[3])) + ((o.v[4] + o.v[5]) + (o.v[6] + o.v[7]));
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
            if (F::kMins == 2) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
            sum *= up;
            // (terms by truncation: eight bits each, and what is left has no more)
            const uint32_t hi = __float_as_uint(sum) & 0xFFFF0000u;
            const float r1 = sum - __uint_as_float(hi);
            const uint32_t mid = __float_as_uint(r1) & 0xFFFF0000u;
            const uint32_t hm = __byte_perm(hi, mid, 0x7632), l = __float_as_uint(r1 - __uint_as_float(mid)) >> 16;
            uint8_t* st = xt + 4096 + ((m & 7) * 4 + tt) * 16;
            if constexpr (F::kMins == 2) {
              const uint32_t hm1 = __shfl_xor_sync(0xFFFFFFFFu, hm, 4), l1 = __shfl_xor_sync(0xFFFFFFFFu, l, 4);
              if (q == 0) *reinterpret_cast<uint4*>(st) = make_uint4(__byte_perm(hm, hm1, 0x5410), __byte_perm(hm, hm1, 0x7632), l | l1 << 16, 0u);
            } else {
              const uint32_t hm1 = __shfl_xor_sync(0xFFFFFFFFu, hm, 2), l1 = __shfl_xor_sync(0xFFFFFFFFu, l, 2);
              const uint32_t hp = __byte_perm(hm, hm1, 0x5410), mp = __byte_perm(hm, hm1, 0x7632), lp = l | l1 << 16;     // groups 0, 1 (lane q = 0)
              const uint32_t hp2 = __shfl_xor_sync(0xFFFFFFFFu, hp, 4), mp2 = __shfl_xor_sync(0xFFFFFFFFu, mp, 4), lp2 = __shfl_xor_sync(0xFFFFFFFFu, lp, 4);
              if (q == 0) {
                *reinterpret_cast<uint4*>(st) = make_uint4(hp, hp2, mp, mp2);
                *reinterpret_cast<uint2*>(xt + 4096 + 512 + ((m & 7) * 4 + tt) * 8) = make_uint2(lp, lp2);
              }
            }
          }
          // magnitudes more than 2^31 below the largest: left out here, see more_planes (next to an infinity or a NaN nothing counts: every
          // output is recomputed)
          if (eb < 255 && __any_sync(0xFFFFFFFFu, (uint32_t)(least >> 7) + 31 < eb)) {
            const uint32_t e = __reduce_min_sync(0xFFFFFFFFu, (uint32_t)(least >> 7));
            if (lane == 0) { atomicMax(&planes[blk], (int)((eb - e) >> 5)); planes[geo.chunk_sb] = 1; }
#pragma unroll
            for (int i = 0; i < 8; i++)
              if (exponent_of(o.v[i]) + 31 < eb) o.v[i] = 0.f;
          }
          *reinterpret_cast<uint4*>(xt + q * 512 + ((m & 7) * 4 + tt) * 16) = o.template fragment<B::kPairOrder>(up);
          // 2^(E - 14 + 10); the other 2^10 of kExp = 20 go with the block's scale, so that both stay in range
          if (lane == 0) reinterpret_cast<float*>(xt + 4096 + mins_bytes<F>())[m & 7] = __uint_as_float((eb - 4) << 23);
        }
      }
    }
    __syncthreads();

    // kExtra: some staged block has further planes.  A loop of its own: the call costs registers that the usual loop is short of.
    auto multiply = [&]<bool kExtra>() {
      int rt = rt0, k = k0;
      float out[NT][4];
#pragma unroll
      for (int n = 0; n < NT; n++) out[n][0] = out[n][1] = out[n][2] = out[n][3] = 0.f;
      for (int i = 0; i < pass_steps; i++) {
        issue_next();
        if (geo.tma) tma_box_wait(my_bars + 8 * slot, phase, status, lane);
        else cp_async_wait_pending(depth - 1);
        __syncwarp();
        const int sb0 = sb_lo + k * nb, nbh = min(nb, SB - sb0);
        const uint32_t ring = my_ring + slot * geo.slot_bytes + g * pitch;
        uint32_t skew0 = (sb0 * B::kTs) & 15, skew1 = skew0;
        if (geo.row_skew != 0) {
          skew0 = (sb0 * B::kTs + min((tile_lo + rt) * 16 + g, N - 1) * geo.row_skew) & 15;
          skew1 = (sb0 * B::kTs + min((tile_lo + rt) * 16 + g + 8, N - 1) * geo.row_skew) & 15;
        }
        for (int blk = 0; blk < nbh; blk++) {
          const uint32_t blk0 = ring + skew0 + blk * B::kTs, blk1 = ring + 8 * pitch + skew1 + blk * B::kTs;
          const uint32_t xb = smem_base + geo.off_x + (uint32_t)(k * nb + blk) * kXBlock;
          typename F::Run run0, run1;
          bf::load_pair<F>(tf::BlockLd{blk0}, tf::BlockLd{blk1}, t, run0, run1);
          float acc[NT][4], acc2[NT][4];             // acc2: a second chain where there is one column tile; the offsets' sums
#pragma unroll
          for (int n = 0; n < NT; n++) {
            acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
            acc2[n][0] = acc2[n][1] = acc2[n][2] = acc2[n][3] = 0.f;
          }
#pragma unroll
          for (int q = 0; q < 8; q++) {
            uint32_t a0[4], b0[4], a1[4], b1[4];
            F::octet(run0, q, tb, a0, b0);
            F::octet(run1, q, tb, a1, b1);
#pragma unroll
            for (int n = 0; n < NT; n++) {
              const uint4 xv = tf::lds_v4(xb + n * kXTile + q * 512 + lane * 16);
              float (&second)[4] = NT == 1 ? acc2[n] : acc[n];
              mma_f16(acc[n], a0[0], a1[0], a0[1], a1[1], xv.x, xv.y);
              mma_f16(second, a0[2], a1[2], a0[3], a1[3], xv.z, xv.w);
              if constexpr (F::kPlanes == 2) {
                mma_f16(acc[n], b0[0], b1[0], b0[1], b1[1], xv.x, xv.y);
                mma_f16(second, b0[2], b1[2], b0[3], b1[3], xv.z, xv.w);
              }
            }
          }
          if constexpr (NT == 1) {
#pragma unroll
            for (int j = 0; j < 4; j++) { acc[0][j] += acc2[0][j]; acc2[0][j] = 0.f; }
          }
          const uint32_t fac_addr = xb + 4096 + mins_bytes<F>();
          if constexpr (kExtra) {
            const int extra = planes[k * nb + blk];
            if (extra) {
#pragma unroll 1
              for (int n = 0; n < NT; n++) {
                float rest[4] = {0.f, 0.f, 0.f, 0.f};
                more_planes<F>(blk0, blk1, tb, x + (int64_t)n * 8 * K, M - 8 * n, K, (sb0 + blk) * 256, fac_addr + n * kXTile, extra, rest);
#pragma unroll
                for (int nn = 0; nn < NT; nn++)
#pragma unroll
                  for (int j = 0; j < 4; j++) acc[nn][j] += nn == n ? rest[j] : 0.f;
              }
            }
          }
          if constexpr (F::kMins == 2) {
#pragma unroll
            for (int n = 0; n < NT; n++) {
              const uint4 sv = tf::lds_v4(xb + n * kXTile + 4096 + lane * 16);
              tile::mma16816(acc2[n], run0.mn[0], run1.mn[0], run0.mn[0], run1.mn[0], sv.x, sv.y);
              tile::mma16816(acc2[n], run0.mn[0], run1.mn[0], 0u, 0u, sv.z, 0u);
            }
          } else if constexpr (F::kMins == 4) {
#pragma unroll
            for (int n = 0; n < NT; n++) {
              const uint4 sv = tf::lds_v4(xb + n * kXTile + 4096 + lane * 16);
              const uint2 lv = tf::lds_v2(xb + n * kXTile + 4096 + 512 + lane * 8);
              tile::mma16816(acc2[n], run0.mn[0], run1.mn[0], run0.mn[1], run1.mn[1], sv.x, sv.y);
              tile::mma16816(acc2[n], run0.mn[0], run1.mn[0], run0.mn[1], run1.mn[1], sv.z, sv.w);
              tile::mma16816(acc2[n], run0.mn[0], run1.mn[0], run0.mn[1], run1.mn[1], lv.x, lv.y);
            }
          }
          const float d0 = run0.d * 1024.0f, d1 = run1.d * 1024.0f;
          const float n0 = run0.nd * (1.0f / 1024.0f), n1 = run1.nd * (1.0f / 1024.0f);
#pragma unroll
          for (int n = 0; n < NT; n++) {
            const uint2 fu = tf::lds_v2(fac_addr + n * kXTile + 8 * t);
            const float f0 = __uint_as_float(fu.x), f1 = __uint_as_float(fu.y);
            float (&a)[4] = acc[n], (&a2)[4] = acc2[n], (&o)[4] = out[n];
            mul2(a[0], a[1], a[0], a[1], f0, f1);
            mul2(a[2], a[3], a[2], a[3], f0, f1);
            fma2(o[0], o[1], d0, d0, a[0], a[1]);
            fma2(o[2], o[3], d1, d1, a[2], a[3]);
            if constexpr (F::kMins > 0) {
              mul2(a2[0], a2[1], a2[0], a2[1], f0, f1);
              mul2(a2[2], a2[3], a2[2], a2[3], f0, f1);
              fma2(o[0], o[1], n0, n0, a2[0], a2[1]);
              fma2(o[2], o[3], n1, n1, a2[2], a2[3]);
            }
          }
        }
        __syncwarp();          // every lane is done with the slot before a later copy overwrites it
        if (++slot == depth) { slot = 0; phase ^= 1; }
        if (k == spu - 1 || i == pass_steps - 1) {      // end of the tile, or of this warp's range
#pragma unroll
          for (int n = 0; n < NT; n++) {
            float4* p = sums + sum_at(rt + warp) + 32 * n;
            float4 v = make_float4(out[n][0], out[n][1], out[n][2], out[n][3]);
            if (pass > 0) { const float4 o = *p; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
            *p = v;
            out[n][0] = out[n][1] = out[n][2] = out[n][3] = 0.f;
          }
        }
        if (++k == spu) { k = 0; ++rt; }
      }
    };
    if (planes[geo.chunk_sb]) multiply.template operator()<true>();
    else multiply.template operator()<false>();
  }
  if (!geo.tma) cp_async_wait_pending(0);

  // ---- the tiles' sums over the warps and the cluster's CTAs, and the outputs
  __syncthreads();
  if (geo.Q > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int tile = tiles * rank / geo.Q + warp; tile < tiles * (rank + 1) / geo.Q; tile += kWarps) {
    const int w0 = warp_of(T, tile * spu), w1 = warp_of(T, tile * spu + spu - 1);
    float v[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) v[n][0] = v[n][1] = v[n][2] = v[n][3] = 0.f;
    for (int q = 0; q < geo.Q; q++) {
      uint32_t peer = smem_base + geo.off_sum;
      if (geo.Q > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(smem_base + geo.off_sum), "r"(q));
      for (int ww = w0; ww <= w1; ww++) {
        if (warp_begin(T, ww) == warp_begin(T, ww + 1)) continue;       // no step, no segment
#pragma unroll
        for (int n = 0; n < NT; n++) {
          float4 s;
          asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(s.x), "=f"(s.y), "=f"(s.z), "=f"(s.w)
                       : "r"(peer + 16 * (sum_at(tile + ww) + 32 * n)) : "memory");
          v[n][0] += s.x; v[n][1] += s.y; v[n][2] += s.z; v[n][3] += s.w;
        }
      }
    }
    bool bad = false;
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int row = (tile_lo + tile) * 16 + g + 8 * (i >> 1), m = n * 8 + 2 * t + (i & 1);
        if (row < N && m < M) { store_out(y, y_dtype, (int64_t)m * N + row, v[n][i]); bad |= not_finite(v[n][i]); }
      }
    if (__any_sync(0xFFFFFFFFu, bad)) {          // outputs that are not finite
#pragma unroll 1
      for (int j = 0; j < 4 * NT; j++) {
        const int row = (tile_lo + tile) * 16 + g + 8 * ((j >> 1) & 1), m = (j >> 2) * 8 + 2 * t + (j & 1);
        const bool again = row < N && m < M && not_finite(load_out(y, y_dtype, (int64_t)m * N + row));
        recompute<B::kQt>(again, row, m, w, (int64_t)row_bytes, N, x, K, tab, y, y_dtype);
      }
    }
  }
  // a CTA's shared memory stays until its peers have read it
  if (geo.Q > 1) asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

struct Args {
  Geo* geo;
  int NT;
  cudaStream_t st;
  const uint8_t* w;
  int N, K;
  const void* x;
  int M;
  void* y;
  int y_dtype;
  const uint8_t* tab;
  int* status;
  const CUtensorMap* map;
};
template <class F, int NT>
static cudaError_t launch(const Args& a) {
  static std::atomic<bool> attr_done[64];   // setting the attribute twice is harmless, so a flag per device suffices
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev].load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(gemv_batch_kernel<F, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile::kSmemLimit);
    if (e != cudaSuccess) return e;
    attr_done[dev].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(a.geo->J * a.geo->Q));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)a.geo->total;
  cfg.stream = a.st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)a.geo->Q;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.geo->Q > 1 ? 2 : 1;
  cudaError_t err = cudaLaunchKernelEx(&cfg, gemv_batch_kernel<F, NT>, a.w, a.N, a.K, (const __nv_bfloat16*)a.x, a.M, a.y, a.y_dtype, (const Geo)*a.geo,
                                       a.tab, a.status, *a.map);
  return err != cudaSuccess ? err : cudaPeekAtLastError();
}
template <class F>
static cudaError_t launch_tiles(const Args& a) { return a.NT == 1 ? launch<F, 1>(a) : launch<F, 2>(a); }
int max_clusters(int Q);            // clusters of Q CTAs on the current device at once, 0 if it cannot be told
cudaError_t launch_k(int qtype, const Args& a);
cudaError_t launch_iq(int qtype, const Args& a);

}  // namespace batch
}  // namespace ggq
