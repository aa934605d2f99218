// Block formats of the tiled fused multiply (gemv_tile.cuh): how one lane turns raw block bytes
// into tensor-core operands.
//
// The multiply uses mma.sync.m16n8k16 with *exact integer codes* as the A operand.  A bf16 whose
// upper byte is 0x00 (or 0x80) is linear in its lower byte: bits 0x00vv are +v * 2^-133, bits
// 0x80vv are -v * 2^-133, for every v in 0..255.  So a 32-bit register (v0 | s0 << 15 | v1 << 16 |
// s1 << 31) is a pair of bf16 weights without any conversion, and a masked field that was not
// shifted down (v << n) is the same weight times 2^n, which the activation side absorbs with an
// exact power-of-two scale.  Scales are applied to the float32 accumulators, once per scale group.
//
// A superblock of 256 weights is split into four lane runs of 64 weights; lane (g, t) of a warp
// owns run t of rows g and g + 8 of the warp's 16-row tile.  A run is eight octets of eight
// weights; an octet feeds two MMAs (four weights per row and MMA sit in the k-slots 2t, 2t+1,
// 2t+8, 2t+9).  Which weights form run t / octet oo, and in which order they enter the k-slots,
// is the format's choice (src_quads + kPairOrder): the activations are permuted to match when
// they are staged in shared memory.  A format provides
//
//   kTs, kQt            block bytes, qtype code
//   kOct                octets per run: 8, or 16 for the two-plane formats (Q5_K, Q6_K), whose codes are
//                       split into a nibble plane and a high-bit plane that are multiplied separately
//                       (every weight then appears in two octets, with its activation staged twice)
//   kGroupOct           octets per scale group inside a run (1, 2 or 4 = groups of 8, 16, 32)
//   kSums, kSumOct      the fold needs the activations' sum per scale group, taken over the group's first
//                       kSumOct octets (all of them, or the first plane of a two-plane format)
//   kPairOrder          0: an octet is 8 consecutive weights e..e+7 entering as (e, e+2), (e+1, e+3),
//                          (e+4, e+6), (e+5, e+7)    [byte pairs (0,2), (1,3) of two words]
//                       1: an octet is two quads a..a+3, b..b+3 entering as (a, b), (a+1, b+1),
//                          (a+2, b+2), (a+3, b+3)     [the two nibbles of each byte of a word]
//   src_quads(t, oo)    first weight of the octet's two quads
//   x_exp(t, oo)        exponent e <= 0: the octet's activations are staged times 2^e
//   kAlign              alignment of every block when rows start 16-byte aligned: gcd(kTs, 16)
//   kUnrollGroups       true for the bit-plane formats, whose groups share the same words (the run is
//                       loaded once and the group loop is unrolled); false for the grid formats, whose
//                       groups are loaded one at a time inside a real loop (keeps the loop body small)
//   Run, load_run(ld, t)             what is read once per run and row
//   Group, load_group(ld, run, t, grp)   the raw fields and the scale of group grp of the run
//   kKv                 16-entry code book behind a table of its byte pairs: absent / 0 none, 1 IQ4 values + 128,
//                       2 MXFP4 values + 12
//   kScaleExp           the group scales carry 2^kScaleExp (taken back out of the row sums; 0 where the trait is absent)
//   kLean, load_group_lean(ld, t, grp)   the group straight from the block, nothing kept for the run (absent: load_run only).  At
//                       four passes the registers are what is short: there the
//                       groups are loaded one at a time inside a real loop (octet<false>; us at 8 rows, whole runs / group
//                       by group: Q4_1 14336 x 4096 30.1 / 27.8, Q5_1 37.5 / 31.2, NVFP4 37.3 / 33.6 and 16384 x 8192 69.6 / 58.0)
//   octet(group, q, tab, p)   the four A-operand registers of octet q of the group: p[0], p[1] = first
//                       MMA (k-slot pairs 2t.. and 2t+8..), p[2], p[3] = second MMA
//   fold(group, acc, xsum, out) -> float   out + the group's contribution given acc = sum(code * x)
//                       and xsum = sum(x) over the group (both in the same power-of-two scale)
//
// Everything here is plain integer and float32 arithmetic written for host and device, so the
// per-format logic is checked on the CPU against the block decoders (tests/test_tile_formats.py).
// Decode formulas: src/gguf_jax/quants.py:219-239 (Q2_K), :275-305 (Q4_K), :493-664 (IQ2/IQ3/IQ1),
// :686-712 (IQ4_XS) in the reference; gguf/quants.py for the same formats in gguf-py.
#pragma once

#include <stdint.h>
#include <string.h>

// Under nvcc everything here is device code (blocks and tables are addressed in shared memory);
// a plain C++ compiler gets the same functions over ordinary memory for the host-side check.
#if defined(__CUDACC__)
#define TF_HD __device__ __forceinline__
#define TF_DEVICE 1
#else
#define TF_HD inline
#define TF_DEVICE 0
#endif

namespace ggq {
namespace tf {

// ---- small portable helpers -----------------------------------------------------------------
TF_HD uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
#if TF_DEVICE
  return __byte_perm(a, b, sel);
#else
  const uint64_t v = (uint64_t)a | ((uint64_t)b << 32);
  uint32_t r = 0;
  for (int i = 0; i < 4; i++) r |= (uint32_t)((v >> (8 * ((sel >> (4 * i)) & 7))) & 0xFF) << (8 * i);
  return r;
#endif
}
TF_HD uint32_t popc(uint32_t v) {
#if TF_DEVICE
  return __popc(v);
#else
  return (uint32_t)__builtin_popcount(v);
#endif
}
TF_HD uint32_t funnel16(uint32_t lo, uint32_t hi) {   // bytes 2..5 of the eight bytes (lo, hi)
#if TF_DEVICE
  return __funnelshift_r(lo, hi, 16);
#else
  return (lo >> 16) | (hi << 16);
#endif
}
TF_HD float f16_bits_to_float(uint32_t h) {
#if TF_DEVICE
  return __half2float(__ushort_as_half((unsigned short)h));
#else
  const uint32_t s = (h >> 15) & 1, e = (h >> 10) & 31, m = h & 1023;
  uint32_t u;
  if (e == 0) {
    if (m == 0) u = s << 31;
    else { int k = 0; uint32_t mm = m; while (!(mm & 1024)) { mm <<= 1; k++; } u = (s << 31) | ((uint32_t)(113 - k) << 23) | ((mm & 1023) << 13); }
  } else if (e == 31) u = (s << 31) | 0x7F800000u | (m << 13);
  else u = (s << 31) | ((e + 112) << 23) | (m << 13);
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}
TF_HD float mulf(float a, float b) {
#if TF_DEVICE
  return __fmul_rn(a, b);
#else
  volatile float r = a * b;
  return r;
#endif
}
TF_HD float fmaf_(float a, float b, float c) {
#if TF_DEVICE
  return __fmaf_rn(a, b, c);
#else
  return __builtin_fmaf(a, b, c);
#endif
}
TF_HD float u2f(uint32_t v) { return (float)v; }

// Pair registers from a word of four code bytes: bytes (0, 2) and bytes (1, 3), each byte widened
// to a bf16 with a zero upper byte.
TF_HD uint32_t pair02(uint32_t w) { return prmt(w, 0u, 0x4240u); }
TF_HD uint32_t pair13(uint32_t w) { return prmt(w, 0u, 0x4341u); }
// The same with sign bits: `s` holds 0x80 or 0x00 in byte j for the sign of code byte j.
TF_HD uint32_t pair02s(uint32_t w, uint32_t s) { return prmt(w, s, 0x6240u); }
TF_HD uint32_t pair13s(uint32_t w, uint32_t s) { return prmt(w, s, 0x7351u); }
// Four sign bits (bit j of `nib`, j = 0..3) spread to 0x80 in byte j.
TF_HD uint32_t spread_signs4(uint32_t nib) { return ((nib & 15u) * 0x10204080u) & 0x80808080u; }
// ksigns[i] = i | parity(i) << 7 (gguf/quants.py IQ2_XXS.ksigns)
TF_HD uint32_t ksigns(uint32_t i7) { return i7 | ((popc(i7) & 1u) << 7); }

// Reads 32-bit words starting at byte offset `off` of a block.  A is the alignment the caller
// guarantees for that address (16, 8, 4: vector or word loads; 2: aligned words and a funnel shift by
// 0 or 16 bits, without a branch: lanes of a warp hold different rows, which may start at different
// offsets modulo 4).
// On the device a block lives in shared memory and is addressed by its 32-bit shared-window
// address, so that field offsets fold into the load instructions.
#if TF_DEVICE
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) { uint16_t v; asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint2 lds_v2(uint32_t a) { uint2 v; asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); return v; }
__device__ __forceinline__ uint4 lds_v4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
struct BlockLd {
  uint32_t p;        // shared-window address of the block's first byte
  __device__ __forceinline__ uint32_t u16(int off) const { return lds_u16(p + off); }
  // Sixteen bytes at an even address as two aligned 16-byte loads and a shift by their offset in the piece (selects, no
  // branch): 8 shared-memory wavefronts per warp where the five word loads of words<4, 2> take 20 with the rows' banks
  // four apart.
  __device__ __forceinline__ void words16(int off, uint32_t (&out)[4]) const {
    const uint32_t a = p + off, base = a & ~15u;
    const uint4 x = lds_v4(base), y = lds_v4(base + 16);
    const bool two = a & 8, one = a & 4;
    const uint32_t v0 = two ? x.z : x.x, v1 = two ? x.w : x.y, v2 = two ? y.x : x.z, v3 = two ? y.y : x.w, v4 = two ? y.z : y.x,
                   v5 = two ? y.w : y.y;
    const uint32_t w0 = one ? v1 : v0, w1 = one ? v2 : v1, w2 = one ? v3 : v2, w3 = one ? v4 : v3, w4 = one ? v5 : v4;
    const uint32_t sh = (a & 2u) << 3;
    out[0] = __funnelshift_r(w0, w1, sh); out[1] = __funnelshift_r(w1, w2, sh);
    out[2] = __funnelshift_r(w2, w3, sh); out[3] = __funnelshift_r(w3, w4, sh);
  }
  template <int NW, int A>
  __device__ __forceinline__ void words(int off, uint32_t (&out)[NW]) const {
    const uint32_t a = p + off;
    if constexpr (A >= 16 && NW % 4 == 0) {
#pragma unroll
      for (int i = 0; i < NW / 4; i++) {
        const uint4 v = lds_v4(a + 16 * i);
        out[4 * i] = v.x; out[4 * i + 1] = v.y; out[4 * i + 2] = v.z; out[4 * i + 3] = v.w;
      }
    } else if constexpr (A >= 8 && NW % 2 == 0) {
#pragma unroll
      for (int i = 0; i < NW / 2; i++) {
        const uint2 v = lds_v2(a + 8 * i);
        out[2 * i] = v.x; out[2 * i + 1] = v.y;
      }
    } else if constexpr (A >= 4) {
#pragma unroll
      for (int i = 0; i < NW; i++) out[i] = lds_u32(a + 4 * i);
    } else {
      // 2-byte aligned: NW + 1 aligned words and a funnel shift by 0 or 16 bits (no branch: a branch
      // here would leave the compiler unsure that the warp is converged at the next mma.sync)
      const uint32_t base = a & ~3u, sh = (a & 2u) << 3;
      uint32_t prev = lds_u32(base);
#pragma unroll
      for (int i = 0; i < NW; i++) { const uint32_t cur = lds_u32(base + 4 + 4 * i); out[i] = __funnelshift_r(prev, cur, sh); prev = cur; }
    }
  }
};
// Per-CTA lookup tables in shared memory.
struct Tables {
  uint32_t grid;           // shared-window address of this lane's copy of the format's grid: 8 (IQ1, IQ2) or 4 (IQ3) code bytes per entry
  uint32_t sign;           // shared-window address of this lane's copy of the sign table (formats with kSignBits)
};
#else
struct BlockLd {
  const uint8_t* p;
  uint32_t u16(int off) const { uint16_t v; memcpy(&v, p + off, 2); return v; }
  void words16(int off, uint32_t (&out)[4]) const { memcpy(out, p + off, 16); }
  template <int NW, int A>
  void words(int off, uint32_t (&out)[NW]) const {
    for (int i = 0; i < NW; i++) memcpy(&out[i], p + off + 4 * i, 4);
  }
};
struct Tables {
  const uint8_t* grid;
  uint32_t kv[4];
};
#endif
struct NoRun {};
// Optional members of a format.
template <class F, class = void> struct KvOf { static constexpr int value = 0; };
template <class F> struct KvOf<F, decltype((void)F::kKv)> { static constexpr int value = F::kKv; };
template <class F, class = void> struct LeanOf { static constexpr bool value = false; };
template <class F> struct LeanOf<F, decltype((void)F::kLean)> { static constexpr bool value = F::kLean; };
template <class F, class = void> struct ScaleExpOf { static constexpr int value = 0; };
template <class F> struct ScaleExpOf<F, decltype((void)F::kScaleExp)> { static constexpr int value = F::kScaleExp; };

// An octet from one word of eight code-book nibbles (pair order 1).  A byte's two codes, one in each half of a word, are
// already an A-operand register: on the device a table of the 256 bytes gives it with one load (32 interleaved
// copies: a lane has its own bank), where four byte permutes, a blend and the widening of each code took seventeen
// instructions of the half-rate integer pipe per octet (IQ4_XS 8192 x 28672 at batch 1: 59.8 -> 51.0 us).
constexpr int kByteTableCopies = 32, kByteTableBytes = 256 * 4 * kByteTableCopies;
TF_HD void lookup_octet(const Tables& tb, uint32_t w, uint32_t (&p)[4]) {
#if TF_DEVICE
#pragma unroll
  for (int j = 0; j < 4; j++) p[j] = lds_u32(tb.grid + 4 * kByteTableCopies * ((w >> (8 * j)) & 0xFF));
#else
  const uint8_t* kv = reinterpret_cast<const uint8_t*>(tb.kv);
  for (int j = 0; j < 4; j++) p[j] = kv[(w >> (8 * j)) & 15] | (uint32_t)kv[(w >> (8 * j + 4)) & 15] << 16;
#endif
}
// An octet from one word of eight plain nibbles (pair order 0: the four low nibbles, then the four high ones).
TF_HD void nibble_octet(uint32_t w, uint32_t (&p)[4]) {
  p[0] = w & 0x000F000Fu; p[1] = (w >> 8) & 0x000F000Fu; p[2] = (w >> 4) & 0x000F000Fu; p[3] = (w >> 12) & 0x000F000Fu;
}
// The same with a fifth bit per weight: bits 0-3 of `h` belong to the low nibbles, bits 16-19 to the high ones.
TF_HD void nibble5_octet(uint32_t w, uint32_t h, uint32_t (&p)[4]) {
  const uint32_t lo = (w & 0x0F0F0F0Fu) | (((h & 15u) * 0x02040810u) & 0x10101010u);
  const uint32_t hi = ((w >> 4) & 0x0F0F0F0Fu) | ((((h >> 16) & 15u) * 0x02040810u) & 0x10101010u);
  p[0] = pair02(lo); p[1] = pair13(lo); p[2] = pair02(hi); p[3] = pair13(hi);
}

// =============================================================================================
// Q4_K  (144 B: d, dmin, 12 packed 6-bit scales/mins, 128 nibble bytes)
// run t = sub-blocks 2t (low nibbles of qs[32t..32t+32)) and 2t+1 (high nibbles); group 0 is the
// low-nibble sub-block, group 1 the high-nibble one (staged times 2^-4, the mask keeps the nibble
// in place).  Contribution of a sub-block: (d * sc) * acc - (dmin * mn) * sum(x).
struct Q4K {
  static constexpr int kQt = 12, kTs = 144, kAlign = 16, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t q[8]; float dl[2], ndm[2]; };
  struct Group { const Run* r; uint32_t mask; float dl, ndm; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int oo) { return oo >= 4 ? -4 : 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    uint32_t h[4];
    ld.words<4, 16>(0, h);
    ld.words<8, 16>(16 + 32 * t, r.q);
    const float d = f16_bits_to_float(h[0] & 0xFFFF), dmin = f16_bits_to_float(h[0] >> 16);
    // 6-bit scale / min of sub-blocks 2t, 2t+1: plain fields for t < 2, split fields for t >= 2
    const int sh = 16 * (t & 1);
    const uint32_t a = h[1] >> sh, m = h[2] >> sh, md = h[3] >> sh;
    const bool low = t < 2;       // selects, not a branch: the warp stays converged for the MMAs
    const uint32_t scp = low ? (a & 0x3F3F) : ((md & 0x0F0F) | ((a >> 2) & 0x3030));
    const uint32_t mnp = low ? (m & 0x3F3F) : (((md >> 4) & 0x0F0F) | ((m >> 2) & 0x3030));
    r.dl[0] = mulf(d, u2f(scp & 0xFF)); r.dl[1] = mulf(d, u2f(scp >> 8));
    r.ndm[0] = -mulf(dmin, u2f(mnp & 0xFF)); r.ndm[1] = -mulf(dmin, u2f(mnp >> 8));
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{&r, grp ? 0x00F000F0u : 0x000F000Fu, r.dl[grp], r.ndm[grp]};
  }
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) {
    const uint32_t w0 = g.r->q[2 * q], w1 = g.r->q[2 * q + 1];
    p[0] = w0 & g.mask; p[1] = (w0 >> 8) & g.mask; p[2] = w1 & g.mask; p[3] = (w1 >> 8) & g.mask;
  }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.ndm, xsum, fmaf_(g.dl, acc, out));
  }
};

// =============================================================================================
// Q2_K  (84 B: 16 scale|min bytes, 64 quant bytes, d, dmin)
// weight e = 128 h + 32 s + p: code = (qs[32 h + p] >> 2 s) & 3, scale byte e / 16.
// run t = (h, u) = (t >> 1, t & 1): the sixteen bytes qs[32 h + 16 u ..+16) at all four shifts;
// group = shift s (16 weights, two octets = the two word pairs), staged times 2^-2s.
struct Q2K {
  static constexpr int kQt = 10, kTs = 84, kAlign = 4, kOct = 8, kGroupOct = 2, kSumOct = 2, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t q[4]; uint32_t sc[4]; float d, ndmin; };
  struct Group { const Run* r; uint32_t mask; float dl, ndm; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) {
    a = 128 * (t >> 1) + 32 * (oo >> 1) + 16 * (t & 1) + 8 * (oo & 1);
    b = a + 4;
  }
  TF_HD static int x_exp(int, int oo) { return -2 * (oo >> 1); }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    ld.words<4, 4>(16 + 16 * t, r.q);
    uint32_t dd[1], s2[2];
    ld.words<1, 4>(80, dd);
    r.d = f16_bits_to_float(dd[0] & 0xFFFF);
    r.ndmin = -f16_bits_to_float(dd[0] >> 16);
    // scale byte of group s: index 8 h + 2 s + u -> byte (2 s + u) of the eight bytes at 8 h
    ld.words<2, 4>(8 * (t >> 1), s2);
    const int u = t & 1;
    r.sc[0] = (s2[0] >> (8 * u)) & 0xFF; r.sc[1] = (s2[0] >> (16 + 8 * u)) & 0xFF;
    r.sc[2] = (s2[1] >> (8 * u)) & 0xFF; r.sc[3] = (s2[1] >> (16 + 8 * u)) & 0xFF;
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{&r, 0x00030003u << (2 * grp), mulf(r.d, u2f(r.sc[grp] & 15)), mulf(r.ndmin, u2f(r.sc[grp] >> 4))};
  }
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) {
    const uint32_t w0 = g.r->q[2 * q], w1 = g.r->q[2 * q + 1];
    p[0] = w0 & g.mask; p[1] = (w0 >> 8) & g.mask; p[2] = w1 & g.mask; p[3] = (w1 >> 8) & g.mask;
  }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.ndm, xsum, fmaf_(g.dl, acc, out));
  }
};

// =============================================================================================
// Q5_K  (176 B: d, dmin, 12 packed 6-bit scales/mins, 32 bytes of fifth bits, 128 nibble bytes)
// code = nibble | bit k of qh[p] << 4 for sub-block k, element p.  Two planes per sub-block: the
// nibbles (as Q4_K) and the fifth bits, kept in place as qh & (0x00010001 << k) = bit * 2^k and
// staged times 2^(4 - k), so that nibble and bit products add up in one accumulator to sum(code * x).
// run t = sub-blocks 2t, 2t+1 = groups 0, 1 of eight octets: four of nibbles, four of fifth bits.
struct Q5K {
  static constexpr int kQt = 13, kTs = 176, kAlign = 16, kOct = 16, kGroupOct = 8, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t q[8], h[8]; float dl[2], ndm[2]; int t; };
  struct Group { const Run* r; uint32_t mask_q, mask_h; float dl, ndm; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 32 * (oo >> 3) + 8 * (oo & 3); b = a + 4; }
  TF_HD static int x_exp(int t, int oo) {
    const int k = 2 * t + (oo >> 3);
    return (oo & 4) ? 4 - k : ((oo >> 3) ? -4 : 0);
  }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    uint32_t h[4];
    ld.words<4, 16>(0, h);
    ld.words<8, 16>(16, r.h);
    ld.words<8, 16>(48 + 32 * t, r.q);
    r.t = t;
    const float d = f16_bits_to_float(h[0] & 0xFFFF), dmin = f16_bits_to_float(h[0] >> 16);
    const int sh = 16 * (t & 1);
    const uint32_t a = h[1] >> sh, m = h[2] >> sh, md = h[3] >> sh;
    const bool low = t < 2;
    const uint32_t scp = low ? (a & 0x3F3F) : ((md & 0x0F0F) | ((a >> 2) & 0x3030));
    const uint32_t mnp = low ? (m & 0x3F3F) : (((md >> 4) & 0x0F0F) | ((m >> 2) & 0x3030));
    r.dl[0] = mulf(d, u2f(scp & 0xFF)); r.dl[1] = mulf(d, u2f(scp >> 8));
    r.ndm[0] = -mulf(dmin, u2f(mnp & 0xFF)); r.ndm[1] = -mulf(dmin, u2f(mnp >> 8));
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{&r, grp ? 0x00F000F0u : 0x000F000Fu, 0x00010001u << (2 * r.t + grp), r.dl[grp], r.ndm[grp]};
  }
  // octets 0-3: the nibbles of the sub-block, octets 4-7: its fifth bits (both add into one accumulator)
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) {
    const uint32_t* w = q < 4 ? g.r->q : g.r->h;
    const uint32_t m = q < 4 ? g.mask_q : g.mask_h;
    const uint32_t w0 = w[2 * (q & 3)], w1 = w[2 * (q & 3) + 1];
    p[0] = w0 & m; p[1] = (w0 >> 8) & m; p[2] = w1 & m; p[3] = (w1 >> 8) & m;
  }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.ndm, xsum, fmaf_(g.dl, acc, out));
  }
};

// =============================================================================================
// Q6_K  (210 B: 128 low-nibble bytes, 64 bytes of 2-bit highs, 16 int8 scales, d)
// element e = 128 h + 32 c + p: low = nibble (c >> 1) of ql[64 h + 32 (c & 1) + p], high = bits 2c, 2c+1 of
// qh[32 h + p], weight = d * sc[8 h + 2 c + (p >> 4)] * (low + 16 high - 32).
// run t = (h, u) = (t >> 1, t & 1): elements p in [16 u, 16 u + 16) of every c, i.e. four scale groups
// of 16.  Two planes per group: the nibbles and the 2-bit highs kept in place (high * 4^c, staged times
// 2^(4 - 2c)) add up in one accumulator to sum((low + 16 high) * x); group c = two octets of nibbles,
// then two of highs.
struct Q6K {
  static constexpr int kQt = 14, kTs = 210, kAlign = 2, kOct = 16, kGroupOct = 4, kSumOct = 2, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t qa[4], qb[4], qh[4]; float dl[4]; };
  struct Group { const uint32_t* lo; const uint32_t* hi; uint32_t mask_lo, mask_hi; float dl; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) {
    a = 128 * (t >> 1) + 32 * (oo >> 2) + 16 * (t & 1) + 8 * (oo & 1);
    b = a + 4;
  }
  TF_HD static int x_exp(int, int oo) {
    const int c = oo >> 2;
    return (oo & 2) ? 4 - 2 * c : ((c >> 1) ? -4 : 0);
  }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    const int h = t >> 1, u = t & 1;
    ld.words<4, 2>(64 * h + 16 * u, r.qa);
    ld.words<4, 2>(64 * h + 32 + 16 * u, r.qb);
    ld.words<4, 2>(128 + 32 * h + 16 * u, r.qh);
    uint32_t sc[2];
    ld.words<2, 2>(192 + 8 * h, sc);
    const float d = f16_bits_to_float(ld.u16(208));
    for (int c = 0; c < 4; c++) {
      const uint32_t byte = (sc[c >> 1] >> (16 * (c & 1) + 8 * u)) & 0xFF;
      r.dl[c] = mulf(d, (float)(int)(int8_t)byte);
    }
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{(grp & 1) ? r.qb : r.qa, r.qh, (grp >> 1) ? 0x00F000F0u : 0x000F000Fu, 0x00030003u << (2 * grp), r.dl[grp]};
  }
  // octets 0-1: the nibbles of the group's sixteen weights, octets 2-3: their 2-bit highs
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) {
    const uint32_t* w = q < 2 ? g.lo : g.hi;
    const uint32_t m = q < 2 ? g.mask_lo : g.mask_hi;
    const uint32_t w0 = w[2 * (q & 1)], w1 = w[2 * (q & 1) + 1];
    p[0] = w0 & m; p[1] = (w0 >> 8) & m; p[2] = w1 & m; p[3] = (w1 >> 8) & m;
  }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.dl, fmaf_(-32.0f, xsum, acc), out);
  }
};

// =============================================================================================
// IQ4_XS  (136 B: d, scales_h, 4 scales_l bytes, 128 nibble bytes)
// sub-block j (32 weights): low nibbles of qs[16 j ..+16) are weights 0-15, high nibbles 16-31;
// weight = d * (ls - 32) * kvalues[nibble].  Codes are kvalues + 128 (1..241), looked up two at a time in the
// table of byte pairs; the fold takes the 128 * sum(x) back out.
// run t = sub-blocks 2t, 2t+1 = groups 0, 1; octet q of a group = word q of the sub-block: its four
// low nibbles (weights 4q..4q+3) and four high nibbles (16+4q..): MMA 1 takes the first two bytes
// of the word, MMA 2 the last two (pair order 1).
struct IQ4XS {
  static constexpr int kQt = 23, kTs = 136, kAlign = 8, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 1, kKv = 1;
  static constexpr bool kSums = true, kUnrollGroups = false;
  static constexpr int kTableBytes = kByteTableBytes;
  typedef NoRun Run;
  struct Group { uint32_t q[4]; float dl; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) {
    a = 64 * t + 32 * (oo >> 2) + 4 * (oo & 3);
    b = a + 16;
  }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd&, int) { return Run{}; }
  TF_HD static Group load_group(const BlockLd& ld, const Run&, int t, int grp) {
    Group g;
    ld.words<4, 8>(8 + 32 * t + 16 * grp, g.q);
    uint32_t h[2];
    ld.words<2, 8>(0, h);                    // d | scales_h << 16, scales_l[0..3]
    const int j = 2 * t + grp;
    const int ls = (int)(((h[1] >> (4 * j)) & 15) | (((h[0] >> (16 + 2 * j)) & 3) << 4)) - 32;
    g.dl = mulf(f16_bits_to_float(h[0] & 0xFFFF), (float)ls);
    return g;
  }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) { lookup_octet(tb, g.q[q], p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.dl, fmaf_(-128.0f, xsum, acc), out);
  }
};

// =============================================================================================
// Grid formats.  Common shape: an octet is one 8-byte grid entry (IQ2, IQ1) or two 4-byte entries
// (IQ3) of unsigned code bytes, times eight sign bits.
// The grid is held kCopies times, entry by entry interleaved, and a lane reads copy lane % kCopies: with 16 copies of
// 8-byte entries (32 of 4-byte ones) every lane of a half-warp (warp) has its own banks and a look-up takes the two (one)
// wavefronts it must; random entries of a single copy collided 3 ways on average, and the shared-memory pipe was what
// these formats waited for.  Fewer copies where 64 KB would not hold them.  With the sign table and runs read at once,
// 8192 x 28672 at batch 1 / 4: IQ2_XS 58.0 / 75.8 -> 48.0 / 60.4 us, IQ3_XXS 59.6 / 71.6 -> 51.0 / 63.4, IQ1_M 67.2 / 79.1 -> 46.0 / 62.7.
template <int ENTRY_BYTES, int COPIES>
TF_HD void grid_words(const Tables& tb, uint32_t i0, uint32_t i1, uint32_t& w0, uint32_t& w1) {
#if TF_DEVICE
  if (ENTRY_BYTES == 8) {
    const uint2 v = lds_v2(tb.grid + 8 * COPIES * i0);
    w0 = v.x; w1 = v.y;
  } else {
    w0 = lds_u32(tb.grid + 4 * COPIES * i0);
    w1 = lds_u32(tb.grid + 4 * COPIES * i1);
  }
#else
  if (ENTRY_BYTES == 8) { memcpy(&w0, tb.grid + 8 * i0, 4); memcpy(&w1, tb.grid + 8 * i0 + 4, 4); }
  else { memcpy(&w0, tb.grid + 4 * i0, 4); memcpy(&w1, tb.grid + 4 * i1, 4); }
#endif
}
// Sign bytes (0x80: negative) of an octet.  On the device they come from a table of 128 (seven-bit indices with a parity
// bit) or 256 (plain bits) 8-byte entries, kept in interleaved copies like the grid: a shift, a mask and a load
// where the parity, its merge and the spreading of eight bits took a dozen instructions of the half-rate integer pipe.
// IQ2_S, whose grid has room for eight copies only, is faster without (8192 x 28672 at 1 / 4 rows 50.6 / 61.1 us, with 52.3 / 67.1).
constexpr int kSignCopies = 16;
TF_HD constexpr int sign_table_bytes(int bits) { return bits ? (1 << bits) * 8 * kSignCopies : 0; }
TF_HD uint32_t sign_bits_of(int bits, uint32_t i) { return bits == 7 ? ksigns(i) : i; }
template <int BITS, bool TABLE>
TF_HD void sign_words(const Tables& tb, uint32_t i, uint32_t& s0, uint32_t& s1) {
#if TF_DEVICE
  if (TABLE) {
    const uint2 v = lds_v2(tb.sign + 8 * kSignCopies * i);
    s0 = v.x; s1 = v.y;
    return;
  }
#endif
  (void)tb;
  const uint32_t b = sign_bits_of(BITS, i);
  s0 = spread_signs4(b); s1 = spread_signs4(b >> 4);
}
TF_HD void signed_octet(uint32_t w0, uint32_t w1, uint32_t s0, uint32_t s1, uint32_t (&p)[4]) {
  p[0] = pair02s(w0, s0); p[1] = pair13s(w0, s0); p[2] = pair02s(w1, s1); p[3] = pair13s(w1, s1);
}
TF_HD void plain_octet(uint32_t w0, uint32_t w1, uint32_t (&p)[4]) {
  p[0] = pair02(w0); p[1] = pair13(w0); p[2] = pair02(w1); p[3] = pair13(w1);
}

// IQ2_XXS (66 B: d, 8 x {4 index bytes, u32 = 4 x 7-bit sign index | 4-bit scale << 28}); group = one of them
struct IQ2XXS {
  static constexpr int kQt = 16, kTs = 66, kAlign = 2, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = false, kUnrollGroups = true;
  static constexpr int kEntries = 256, kEntryBytes = 8, kCopies = 16, kSignBits = 7;
  static constexpr bool kSignTable = true;
  static constexpr int kTableBytes = kEntries * kEntryBytes * kCopies + sign_table_bytes(kSignTable ? kSignBits : 0);
  struct Run { uint32_t q[4]; float d4; };
  struct Group { uint32_t q, aux; float db; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    ld.words16(2 + 16 * t, r.q);
    r.d4 = mulf(f16_bits_to_float(ld.u16(0)), 0.25f);
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{r.q[2 * grp], r.q[2 * grp + 1], mulf(r.d4, 0.5f + u2f(r.q[2 * grp + 1] >> 28))};
  }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) {
    uint32_t w0, w1, s0, s1;
    grid_words<8, kCopies>(tb, (g.q >> (8 * q)) & 0xFF, 0, w0, w1);
    sign_words<kSignBits, kSignTable>(tb, (g.aux >> (7 * q)) & 127, s0, s1);
    signed_octet(w0, w1, s0, s1, p);
  }
  TF_HD static float fold(const Group& g, float acc, float, float out) { return fmaf_(g.db, acc, out); }
};

// IQ2_XS (74 B: d, 32 x u16 = 9-bit grid index | 7-bit sign index << 9, 8 scale bytes of two nibbles)
struct IQ2XS {
  static constexpr int kQt = 17, kTs = 74, kAlign = 2, kOct = 8, kGroupOct = 2, kSumOct = 2, kPairOrder = 0;
  static constexpr bool kSums = false, kUnrollGroups = true;
  static constexpr int kEntries = 512, kEntryBytes = 8, kCopies = 16, kSignBits = 7;
  static constexpr bool kSignTable = true;
  static constexpr int kTableBytes = kEntries * kEntryBytes * kCopies + sign_table_bytes(kSignTable ? kSignBits : 0);
  struct Run { uint32_t q[4], sc; float d4; };
  struct Group { uint32_t q; float db; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    ld.words16(2 + 16 * t, r.q);
    r.sc = ld.u16(66 + 2 * t);
    r.d4 = mulf(f16_bits_to_float(ld.u16(0)), 0.25f);
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{r.q[grp], mulf(r.d4, 0.5f + u2f((r.sc >> (4 * grp)) & 15))};
  }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) {
    uint32_t w0, w1, s0, s1;
    grid_words<8, kCopies>(tb, (g.q >> (16 * q)) & 511, 0, w0, w1);
    sign_words<kSignBits, kSignTable>(tb, (g.q >> (16 * q + 9)) & 127, s0, s1);
    signed_octet(w0, w1, s0, s1, p);
  }
  TF_HD static float fold(const Group& g, float acc, float, float out) { return fmaf_(g.db, acc, out); }
};

// IQ2_S (82 B: d, 32 index bytes, 32 sign bytes, 8 bytes of 2 high index bits, 8 scale bytes)
struct IQ2S {
  static constexpr int kQt = 22, kTs = 82, kAlign = 2, kOct = 8, kGroupOct = 2, kSumOct = 2, kPairOrder = 0;
  static constexpr bool kSums = false, kUnrollGroups = true;
  static constexpr int kEntries = 1024, kEntryBytes = 8, kCopies = 8, kSignBits = 8;
  static constexpr bool kSignTable = false;
  static constexpr int kTableBytes = kEntries * kEntryBytes * kCopies + sign_table_bytes(kSignTable ? kSignBits : 0);
  struct Run { uint32_t qs[2], sg[2], qh, sc; float d4; };
  struct Group { uint32_t qs, sg, qh; float db; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    ld.words<2, 2>(2 + 8 * t, r.qs);
    ld.words<2, 2>(34 + 8 * t, r.sg);
    r.qh = ld.u16(66 + 2 * t);
    r.sc = ld.u16(74 + 2 * t);
    r.d4 = mulf(f16_bits_to_float(ld.u16(0)), 0.25f);
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    const int sh = 16 * (grp & 1);
    return Group{r.qs[grp >> 1] >> sh, r.sg[grp >> 1] >> sh, r.qh >> (4 * grp), mulf(r.d4, 0.5f + u2f((r.sc >> (4 * grp)) & 15))};
  }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) {
    const uint32_t idx = ((g.qs >> (8 * q)) & 0xFF) | (((g.qh >> (2 * q)) & 3) << 8);
    uint32_t w0, w1, s0, s1;
    grid_words<8, kCopies>(tb, idx, 0, w0, w1);
    sign_words<kSignBits, kSignTable>(tb, (g.sg >> (8 * q)) & 0xFF, s0, s1);
    signed_octet(w0, w1, s0, s1, p);
  }
  TF_HD static float fold(const Group& g, float acc, float, float out) { return fmaf_(g.db, acc, out); }
};

// IQ3_XXS (98 B: d, 64 index bytes (one per 4 weights), 8 x u32 = 4 x 7-bit sign index | scale << 28)
struct IQ3XXS {
  static constexpr int kQt = 18, kTs = 98, kAlign = 2, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = false, kUnrollGroups = true;
  static constexpr int kEntries = 256, kEntryBytes = 4, kCopies = 32, kSignBits = 7;
  static constexpr bool kSignTable = true;
  static constexpr int kTableBytes = kEntries * kEntryBytes * kCopies + sign_table_bytes(kSignTable ? kSignBits : 0);
  struct Run { uint32_t q[4], aux[2]; float d2; };
  struct Group { uint32_t q[2], aux; float db; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    ld.words16(2 + 16 * t, r.q);
    ld.words<2, 2>(66 + 8 * t, r.aux);
    r.d2 = mulf(f16_bits_to_float(ld.u16(0)), 0.5f);
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{{r.q[2 * grp], r.q[2 * grp + 1]}, r.aux[grp], mulf(r.d2, 0.5f + u2f(r.aux[grp] >> 28))};
  }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) {
    const uint32_t q16 = g.q[q >> 1] >> (16 * (q & 1));
    uint32_t w0, w1, s0, s1;
    grid_words<4, kCopies>(tb, q16 & 0xFF, (q16 >> 8) & 0xFF, w0, w1);
    sign_words<kSignBits, kSignTable>(tb, (g.aux >> (7 * q)) & 127, s0, s1);
    signed_octet(w0, w1, s0, s1, p);
  }
  TF_HD static float fold(const Group& g, float acc, float, float out) { return fmaf_(g.db, acc, out); }
};

// IQ3_S (110 B: d, 64 index bytes, 8 bytes of ninth index bits, 32 sign bytes, 4 scale bytes of two nibbles)
struct IQ3S {
  static constexpr int kQt = 21, kTs = 110, kAlign = 2, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = false, kUnrollGroups = true;
  static constexpr int kEntries = 512, kEntryBytes = 4, kCopies = 16, kSignBits = 8;
  static constexpr bool kSignTable = true;
  static constexpr int kTableBytes = kEntries * kEntryBytes * kCopies + sign_table_bytes(kSignTable ? kSignBits : 0);
  struct Run { uint32_t q[4], sg[2], qh, sc; float d; };
  struct Group { uint32_t q[2], sg, qh; float db; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    ld.words16(2 + 16 * t, r.q);
    ld.words<2, 2>(74 + 8 * t, r.sg);
    r.qh = ld.u16(66 + 2 * t);
    r.sc = ld.u16(106 + (t & 2)) >> (8 * (t & 1));
    r.d = f16_bits_to_float(ld.u16(0));
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{{r.q[2 * grp], r.q[2 * grp + 1]}, r.sg[grp], r.qh >> (8 * grp), mulf(r.d, u2f(1 + 2 * ((r.sc >> (4 * grp)) & 15)))};
  }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) {
    const uint32_t q16 = g.q[q >> 1] >> (16 * (q & 1));
    const uint32_t i0 = (q16 & 0xFF) | (((g.qh >> (2 * q)) & 1) << 8);
    const uint32_t i1 = ((q16 >> 8) & 0xFF) | (((g.qh >> (2 * q + 1)) & 1) << 8);
    uint32_t w0, w1, s0, s1;
    grid_words<4, kCopies>(tb, i0, i1, w0, w1);
    sign_words<kSignBits, kSignTable>(tb, (g.sg >> (8 * q)) & 0xFF, s0, s1);
    signed_octet(w0, w1, s0, s1, p);
  }
  TF_HD static float fold(const Group& g, float acc, float, float out) { return fmaf_(g.db, acc, out); }
};

// IQ1_S (50 B: d, 32 index bytes, 8 x u16 = 4 x 3 high index bits | 3-bit scale << 12 | delta sign << 15)
// weight = d (2 s + 1) (grid + delta), grid in {-1, 0, 1}, delta = -+1/8.  The shared-memory table
// holds the codes 8 grid + 9 (1, 9, 17); adding or subtracting 1 in every byte applies delta, the
// fold removes the 9 and the factor 8:  (dl / 8) * (sum(code x) - 9 sum(x)).
struct IQ1S {
  static constexpr int kQt = 19, kTs = 50, kAlign = 2, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kEntries = 2048, kEntryBytes = 8, kCopies = 4, kSignBits = 0;
  static constexpr bool kSignTable = false;
  static constexpr int kTableBytes = kEntries * kEntryBytes * kCopies + sign_table_bytes(kSignTable ? kSignBits : 0);
  struct Run { uint32_t qs[2], qh[1]; float d8; };
  struct Group { uint32_t qs, qh, dlt; float dl8; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    ld.words<2, 2>(2 + 8 * t, r.qs);
    ld.words<1, 2>(34 + 4 * t, r.qh);
    r.d8 = mulf(f16_bits_to_float(ld.u16(0)), 0.125f);
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    Group g;
    g.qs = r.qs[grp];
    g.qh = r.qh[0] >> (16 * grp);
    g.dlt = (g.qh & 0x8000) ? 0xFEFEFEFFu : 0x01010101u;      // -1 / +1 in every byte
    g.dl8 = mulf(r.d8, u2f(2 * ((g.qh >> 12) & 7) + 1));
    return g;
  }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) {
    const uint32_t idx = ((g.qs >> (8 * q)) & 0xFF) | (((g.qh >> (3 * q)) & 7) << 8);
    uint32_t w0, w1;
    grid_words<8, kCopies>(tb, idx, 0, w0, w1);
    plain_octet(w0 + g.dlt, w1 + g.dlt, p);
  }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.dl8, fmaf_(-9.0f, xsum, acc), out);
  }
};

// IQ1_M (56 B: 32 index bytes, 16 bytes of 2 x {3 high index bits, delta sign}, 4 x u16 = 4 x 3-bit scale |
// a nibble of the f16 super-scale << 12)
struct IQ1M {
  static constexpr int kQt = 29, kTs = 56, kAlign = 8, kOct = 8, kGroupOct = 2, kSumOct = 2, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kEntries = 2048, kEntryBytes = 8, kCopies = 4, kSignBits = 0;
  static constexpr bool kSignTable = false;
  static constexpr int kTableBytes = kEntries * kEntryBytes * kCopies + sign_table_bytes(kSignTable ? kSignBits : 0);
  struct Run { uint32_t qs[2], qh[1], w; float d8; };
  struct Group { uint32_t qs, qh; float dl8; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    uint32_t sc[2];
    ld.words<2, 8>(8 * t, r.qs);
    ld.words<1, 4>(32 + 4 * t, r.qh);
    ld.words<2, 8>(48, sc);
    const uint32_t dbits = ((sc[0] >> 12) & 0x000F) | ((sc[0] >> 24) & 0x00F0) | ((sc[1] >> 4) & 0x0F00) | ((sc[1] >> 16) & 0xF000);
    r.w = ((t & 2) ? sc[1] : sc[0]) >> (16 * (t & 1));
    r.d8 = mulf(f16_bits_to_float(dbits), 0.125f);
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{r.qs[grp >> 1] >> (16 * (grp & 1)), r.qh[0] >> (8 * grp), mulf(r.d8, u2f(2 * ((r.w >> (3 * grp)) & 7) + 1))};
  }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) {
    const uint32_t n = (g.qh >> (4 * q)) & 15;
    const uint32_t idx = ((g.qs >> (8 * q)) & 0xFF) | ((n & 7) << 8);
    uint32_t w0, w1;
    grid_words<8, kCopies>(tb, idx, 0, w0, w1);
    const uint32_t dlt = (n & 8) ? 0xFEFEFEFFu : 0x01010101u;
    plain_octet(w0 + dlt, w1 + dlt, p);
  }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.dl8, fmaf_(-9.0f, xsum, acc), out);
  }
};

// =============================================================================================
// Q3_K  (110 B: 32 bytes of third bits, 64 quant bytes, 12 bytes of 6-bit scales, d)
// weight e = 128 h + 32 s + p: code = (qs[32 h + p] >> 2 s) & 3 | third bit << 2 (bit 4 h + s of hmask[p]), value
// d * (scale - 32) * (code - 4), scale index 8 h + 2 s + (p >> 4).
// run t = (h, u) = (t >> 1, t & 1): p in [16 u, 16 u + 16); group = shift s, as in Q2_K.
struct Q3K {
  static constexpr int kQt = 11, kTs = 110, kAlign = 2, kOct = 8, kGroupOct = 2, kSumOct = 2, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t q[4], hm[4]; float dl[4]; int h4; };
  struct Group { const Run* r; int s; float dl; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { Q2K::src_quads(t, oo, a, b); }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    const int h = t >> 1, u = t & 1;
    ld.words<4, 2>(32 + 32 * h + 16 * u, r.q);
    ld.words<4, 2>(16 * u, r.hm);
    r.h4 = 4 * h;
    uint32_t sc[3];
    ld.words<3, 2>(96, sc);
    const float d = f16_bits_to_float(ld.u16(108));
    for (int s = 0; s < 4; s++) {
      // low four bits: nibble h of byte j = 2 s + u; high two bits: field 2 h + (s >> 1) of byte 8 + (j & 3)
      const uint32_t lo = (sc[s >> 1] >> (16 * (s & 1) + 8 * u + 4 * h)) & 15;
      const uint32_t hi = (sc[2] >> (16 * (s & 1) + 8 * u + 4 * h + 2 * (s >> 1))) & 3;
      r.dl[s] = mulf(d, (float)((int)(lo | (hi << 4)) - 32));
    }
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) { return Group{&r, grp, r.dl[grp]}; }
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) {
    for (int i = 0; i < 2; i++) {
      const uint32_t c = ((g.r->q[2 * q + i] >> (2 * g.s)) & 0x03030303u) |
                         (((g.r->hm[2 * q + i] >> (g.r->h4 + g.s)) & 0x01010101u) << 2);
      p[2 * i] = pair02(c); p[2 * i + 1] = pair13(c);
    }
  }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.dl, fmaf_(-4.0f, xsum, acc), out);
  }
};

// =============================================================================================
// TQ2_0  (66 B: 64 bytes of 2-bit fields laid out as in Q2_K, d): value d * (code - 1), one scale per superblock
struct TQ20 {
  static constexpr int kQt = 35, kTs = 66, kAlign = 2, kOct = 8, kGroupOct = 8, kSumOct = 8, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t q[4]; float d; };
  typedef const Run& Group;
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { Q2K::src_quads(t, oo, a, b); }
  TF_HD static int x_exp(int, int oo) { return -2 * (oo >> 1); }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    ld.words<4, 2>(16 * t, r.q);
    r.d = f16_bits_to_float(ld.u16(64));
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int) { return r; }
  TF_HD static void octet(Group g, int q, const Tables&, uint32_t (&p)[4]) {
    const uint32_t m = 0x00030003u << (2 * (q >> 1)), w0 = g.q[2 * (q & 1)], w1 = g.q[2 * (q & 1) + 1];
    p[0] = w0 & m; p[1] = (w0 >> 8) & m; p[2] = w1 & m; p[3] = (w1 >> 8) & m;
  }
  TF_HD static float fold(Group g, float acc, float xsum, float out) { return fmaf_(g.d, fmaf_(-1.0f, xsum, acc), out); }
};

// TQ1_0  (54 B: 48 + 4 bytes of base-3 digits, d): digit n of a byte v is (((v * 3^n) & 255) * 3) >> 8, value d * (digit - 1).
// Octet g = 8 t + q (elements 8 g ..): g < 20 bytes 8 (g & 3).., digit g >> 2; g < 30 bytes 32 + 8 (g & 1).., digit
// (g - 20) >> 1; the last two octets hold bytes 48..51 twice each, digits 2 (g - 30) and 2 (g - 30) + 1.
struct TQ10 {
  static constexpr int kQt = 34, kTs = 54, kAlign = 2, kOct = 8, kGroupOct = 8, kSumOct = 8, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { float d; int t; };
  struct Group { BlockLd ld; float d; int t; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) { return Run{f16_bits_to_float(ld.u16(52)), t}; }
  TF_HD static Group load_group(const BlockLd& ld, const Run& r, int, int) { return Group{ld, r.d, r.t}; }
  TF_HD static uint32_t digits(uint32_t bytes02, uint32_t pow3) {
    return ((((bytes02 & 0x00FF00FFu) * pow3) & 0x00FF00FFu) * 3u >> 8) & 0x00030003u;
  }
  TF_HD static uint32_t pow3(int n) { return n < 4 ? (0x1B090301u >> (8 * n)) & 0xFFu : 81u; }
  TF_HD static void octet(const Group& gr, int q, const Tables&, uint32_t (&p)[4]) {
    const int g = 8 * gr.t + q;
    const int off = g < 20 ? 8 * (g & 3) : g < 30 ? 32 + 8 * (g & 1) : 48;
    const int n = g < 20 ? g >> 2 : g < 30 ? (g - 20) >> 1 : 2 * (g - 30);
    const int last = g >= 30 ? 1 : 0;
    uint32_t w0[1], w1[1];
    gr.ld.template words<1, 2>(off, w0);
    gr.ld.template words<1, 2>(last ? off : off + 4, w1);
    const uint32_t pa = pow3(n), pb = pow3(n + last);
    p[0] = digits(w0[0], pa); p[1] = digits(w0[0] >> 8, pa); p[2] = digits(w1[0], pb); p[3] = digits(w1[0] >> 8, pb);
  }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) { return fmaf_(g.d, fmaf_(-1.0f, xsum, acc), out); }
};

// =============================================================================================
// Formats that ran on kernels decoding byte by byte to float32 before (streaming at batch 1, three bf16 terms per weight above).
// Measured on B200, 14336 x 4096, us at batch 1 / 4 / 8, before -> here: Q8_0 26 / 55 / 57 -> 20 / 22 / 30, Q4_0 31 / 86 / 87 -> 16 /
// 19 / 27, Q5_1 38 / 131 / 133 -> 18 / 21 / 35, MXFP4 36 / 90 / 92 -> 21 / 23 / 34, Q3_K 42 / 102 / 102 -> 21 / 24 / 39, TQ1_0
// 68 / 92 / 92 -> 23 / 28 / 36.
//
// The 32-element formats: eight blocks make a superblock (kTs = 8 x block bytes), run t = blocks 2 t and 2 t + 1
// = groups 0 and 1.  The run is read as aligned words; the block that starts two bytes into a word is shifted.

// Q8_0 (34 B: d, 32 int8): codes q + 128
struct Q80 {
  static constexpr int kQt = 8, kTs = 272, kAlign = 16, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t q[16]; float d[2]; };
  struct Group { const uint32_t* q; float d; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 8 * oo; b = a + 4; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    uint32_t w[17];
    ld.words<17, 4>(68 * t, w);
    r.d[0] = f16_bits_to_float(w[0] & 0xFFFF);
    r.d[1] = f16_bits_to_float(w[8] >> 16);
    for (int i = 0; i < 8; i++) {
      r.q[i] = funnel16(w[i], w[i + 1]) ^ 0x80808080u;
      r.q[8 + i] = w[9 + i] ^ 0x80808080u;
    }
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) { return Group{r.q + 8 * grp, r.d[grp]}; }
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) { plain_octet(g.q[2 * q], g.q[2 * q + 1], p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.d, fmaf_(-128.0f, xsum, acc), out);
  }
};

// Nibble blocks: element e < 16 is the low nibble of byte e, element 16 + e its high nibble; octet q of a block is its
// word q (weights 4 q.. and 16 + 4 q..).
TF_HD void nibble_src(int t, int oo, int& a, int& b) { a = 64 * t + 32 * (oo >> 2) + 4 * (oo & 3); b = a + 16; }

// Q4_0 (18 B: d, 16 nibble bytes): d * (code - 8)
struct Q40 {
  static constexpr int kQt = 2, kTs = 144, kAlign = 16, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t q[8]; float d[2]; };
  struct Group { const uint32_t* q; float d; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { nibble_src(t, oo, a, b); }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    uint32_t w[9];
    ld.words<9, 4>(36 * t, w);
    r.d[0] = f16_bits_to_float(w[0] & 0xFFFF);
    r.d[1] = f16_bits_to_float(w[4] >> 16);
    for (int i = 0; i < 4; i++) { r.q[i] = funnel16(w[i], w[i + 1]); r.q[4 + i] = w[5 + i]; }
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) { return Group{r.q + 4 * grp, r.d[grp]}; }
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) { nibble_octet(g.q[q], p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.d, fmaf_(-8.0f, xsum, acc), out);
  }
};

// IQ4_NL (18 B, laid out as Q4_0): nibbles select one of sixteen values, codes value + 128
struct IQ4NL : Q40 {
  static constexpr int kQt = 20, kPairOrder = 1, kKv = 1, kTableBytes = kByteTableBytes;
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) { lookup_octet(tb, g.q[q], p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.d, fmaf_(-128.0f, xsum, acc), out);
  }
};

// Q4_1 (20 B: d, m, 16 nibble bytes): d * code + m
struct Q41 {
  static constexpr int kQt = 3, kTs = 160, kAlign = 16, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  static constexpr bool kLean = true;
  struct Run { uint32_t w[10]; };
  struct Group { uint32_t q[4]; float d, m; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { nibble_src(t, oo, a, b); }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) { Run r; ld.words<10, 8>(40 * t, r.w); return r; }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    const uint32_t* w = r.w + 5 * grp;
    return Group{{w[1], w[2], w[3], w[4]}, f16_bits_to_float(w[0] & 0xFFFF), f16_bits_to_float(w[0] >> 16)};
  }
  TF_HD static Group load_group_lean(const BlockLd& ld, int t, int grp) {
    uint32_t w[5];
    ld.words<5, 4>(40 * t + 20 * grp, w);
    return Group{{w[1], w[2], w[3], w[4]}, f16_bits_to_float(w[0] & 0xFFFF), f16_bits_to_float(w[0] >> 16)};
  }
  template <bool = false>
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) { nibble_octet(g.q[q], p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) { return fmaf_(g.m, xsum, fmaf_(g.d, acc, out)); }
};

// Q5_0 (22 B: d, 32 fifth bits, 16 nibble bytes): d * (code - 16)
struct Q50 {
  static constexpr int kQt = 6, kTs = 176, kAlign = 16, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  struct Run { uint32_t q[8], h[2]; float d[2]; };
  struct Group { const uint32_t* q; uint32_t h; float d; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { nibble_src(t, oo, a, b); }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    uint32_t w[11];
    ld.words<11, 4>(44 * t, w);
    r.d[0] = f16_bits_to_float(w[0] & 0xFFFF);
    r.h[0] = funnel16(w[0], w[1]);
    r.d[1] = f16_bits_to_float(w[5] >> 16);
    r.h[1] = w[6];
    for (int i = 0; i < 4; i++) { r.q[i] = funnel16(w[1 + i], w[2 + i]); r.q[4 + i] = w[7 + i]; }
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) { return Group{r.q + 4 * grp, r.h[grp], r.d[grp]}; }
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) { nibble5_octet(g.q[q], g.h >> (4 * q), p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.d, fmaf_(-16.0f, xsum, acc), out);
  }
};

// Q5_1 (24 B: d, m, 32 fifth bits, 16 nibble bytes): d * code + m
struct Q51 {
  static constexpr int kQt = 7, kTs = 192, kAlign = 16, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 0;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = 0;
  static constexpr bool kLean = true;
  struct Run { uint32_t w[12]; };
  struct Group { uint32_t q[4], h; float d, m; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { nibble_src(t, oo, a, b); }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) { Run r; ld.words<12, 16>(48 * t, r.w); return r; }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    const uint32_t* w = r.w + 6 * grp;
    return Group{{w[2], w[3], w[4], w[5]}, w[1], f16_bits_to_float(w[0] & 0xFFFF), f16_bits_to_float(w[0] >> 16)};
  }
  TF_HD static Group load_group_lean(const BlockLd& ld, int t, int grp) {
    uint32_t w[6];
    ld.words<6, 8>(48 * t + 24 * grp, w);
    return Group{{w[2], w[3], w[4], w[5]}, w[1], f16_bits_to_float(w[0] & 0xFFFF), f16_bits_to_float(w[0] >> 16)};
  }
  template <bool = false>
  TF_HD static void octet(const Group& g, int q, const Tables&, uint32_t (&p)[4]) { nibble5_octet(g.q[q], g.h >> (4 * q), p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) { return fmaf_(g.m, xsum, fmaf_(g.d, acc, out)); }
};

// MXFP4 (17 B: an exponent byte e, 16 nibble bytes): 2^(e - 128) * value, codes value + 12.  Blocks have no alignment: the
// run's 34 bytes start at 2 t (mod 4) and its blocks at bytes 0 and 17.  The scale reaches down to 2^-128 and meets sums
// staged times 2^-37: it is carried times 2^37, so that no product leaves the float32 range sooner than the result does.
struct MXFP4 {
  static constexpr int kQt = 39, kTs = 136, kAlign = 8, kOct = 8, kGroupOct = 4, kSumOct = 4, kPairOrder = 1, kKv = 2, kScaleExp = 37;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = kByteTableBytes;
  struct Run { uint32_t q[8]; float d[2]; };
  struct Group { const uint32_t* q; float d; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { nibble_src(t, oo, a, b); }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static float scale(uint32_t e) {
    const uint32_t bits = e < 2 ? 0x00200000u << e : (e - 1) << 23;
#if TF_DEVICE
    return mulf(__uint_as_float(bits), 0x1p37f);
#else
    float d;
    memcpy(&d, &bits, 4);
    return mulf(d, 0x1p37f);
#endif
  }
  TF_HD static Run load_run(const BlockLd& ld, int t) {
    Run r;
    uint32_t v[8], tail;
    ld.words<8, 2>(34 * t, v);
    tail = ld.u16(34 * t + 32);
    r.d[0] = scale(v[0] & 0xFF);
    r.d[1] = scale((v[4] >> 8) & 0xFF);
    for (int i = 0; i < 4; i++) r.q[i] = prmt(v[i], v[i + 1], 0x4321u);
    for (int i = 0; i < 4; i++) r.q[4 + i] = funnel16(v[4 + i], i == 3 ? tail : v[5 + i]);
    return r;
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) { return Group{r.q + 4 * grp, r.d[grp]}; }
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) { lookup_octet(tb, g.q[q], p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.d, fmaf_(-12.0f, xsum, acc), out);
  }
};

// NVFP4 (36 B per 64 weights: four UE4M3 scales, 32 nibble bytes): group s = 16 weights, elements 16 s + j (low nibble of
// byte 8 s + j) and 16 s + 8 + j (high nibble), codes value + 12.  A superblock is four blocks, run t is block t.
struct NVFP4 {
  static constexpr int kQt = 40, kTs = 144, kAlign = 16, kOct = 8, kGroupOct = 2, kSumOct = 2, kPairOrder = 1, kKv = 2;
  static constexpr bool kSums = true, kUnrollGroups = true;
  static constexpr int kTableBytes = kByteTableBytes;
  static constexpr bool kLean = true;
  struct Run { uint32_t w[9]; };
  struct Group { uint32_t q[2]; float d; };
  TF_HD static void src_quads(int t, int oo, int& a, int& b) { a = 64 * t + 16 * (oo >> 1) + 4 * (oo & 1); b = a + 8; }
  TF_HD static int x_exp(int, int) { return 0; }
  TF_HD static Run load_run(const BlockLd& ld, int t) { Run r; ld.words<9, 4>(36 * t, r.w); return r; }
  TF_HD static float scale(uint32_t x) {       // half the UE4M3 value; 0 and 0x7F stand for 0
    const int ex = (int)(x >> 3) & 15;
    const float man = u2f(x & 7);
    const float raw = ex == 0 ? mulf(man, 0x1p-9f) : mulf(8.0f + man, u2f(1u << ex) * 0x1p-10f);
    return (x == 0 || x == 0x7F) ? 0.0f : mulf(raw, 0.5f);
  }
  TF_HD static Group load_group(const BlockLd&, const Run& r, int, int grp) {
    return Group{{r.w[1 + 2 * grp], r.w[2 + 2 * grp]}, scale((r.w[0] >> (8 * grp)) & 0xFF)};
  }
  TF_HD static Group load_group_lean(const BlockLd& ld, int t, int grp) {
    uint32_t w[1], q[2];
    ld.words<1, 4>(36 * t, w);
    ld.words<2, 4>(36 * t + 4 + 8 * grp, q);
    return Group{{q[0], q[1]}, scale((w[0] >> (8 * grp)) & 0xFF)};
  }
  template <bool = false>
  TF_HD static void octet(const Group& g, int q, const Tables& tb, uint32_t (&p)[4]) { lookup_octet(tb, g.q[q], p); }
  TF_HD static float fold(const Group& g, float acc, float xsum, float out) {
    return fmaf_(g.d, fmaf_(-12.0f, xsum, acc), out);
  }
};

}  // namespace tf
}  // namespace ggq
