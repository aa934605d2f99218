// Block formats of the batch kernel (gemv_batch.cuh): how one lane turns raw block bytes into tensor-core operands that already
// carry their group's integer scale.
//
// Formats with one float scale per block of 256 weights write a weight as d * (s * q) [- dmin * m], with a small integer scale s per
// group of 16 or 32 weights and a small integer q.  s * q is an integer of at most 11 significant bits in most of them, which a
// float16 holds exactly, so the group scale goes into the A operand (one packed multiply per two weights) and a whole block of 256
// weights adds up in one accumulator: d is applied once per block, whatever the number of batch rows.  (The kernels of
// tile_formats.cuh keep the codes bare and the groups apart in the columns of the MMA, which leaves two of eight columns for batch rows.)
//
// Codes are the ones of tile_formats.cuh: bits 0x00vv / 0x80vv of a half word, as float16 +-v * 2^-24 (exact, v < 1024), times a scale
// of s * 2^(24 - kExp), gives +-v * s * 2^-kExp.  kExp = 20 keeps every product a multiple of 2^-20 (float16 resolves 2^-24) and every
// scale below 65504.  Q6_K (8-bit scale, 6-bit code) and IQ4_XS (6-bit, 8-bit) have up to 13 bits and take two planes of operands,
// each exact, multiplied by the same activations.
//
// A format provides
//   Base                the tile format whose block geometry, activation order (src_quads, kPairOrder) and tables it shares
//   kPlanes             1, or 2 operands per weight that add up
//   kMins               integer offsets per run (0, 2 or 4): the block's second sum is dmin * sum over groups of m * sum(x)
//   src_quads(t, o)     first weight of the two quads of octet o (0..7) of run t, in the order of Base::kPairOrder
//   Run, load(ld, t)    raw fields and packed scales of run t of one row (or load(ld0, ld1, t, r0, r1) of two)
//   octet(run, q, tb, a, b)   operands of octet q: a[0], a[1] = first MMA (k-slots 2t.., 2t+8..), a[2], a[3] = second; b = second plane
//   Run::d, Run::nd     float scale of the block's sum and, with kMins, of the second sum (-dmin)
//   Run::mn[kMins / 2]  pairs of the offsets as bfloat16
// Host and device code, checked on the CPU like tile_formats.cuh.
#pragma once

#include "tile_formats.cuh"

namespace ggq {
namespace bf {

using namespace tf;
constexpr int kExp = 20;

// ---- packed float16 / bfloat16 arithmetic
#if !TF_DEVICE
inline float half_at(uint32_t v, int i) { return f16_bits_to_float((v >> (16 * i)) & 0xFFFF); }
inline uint32_t to_half(double d) { _Float16 h = (_Float16)d; uint16_t u; memcpy(&u, &h, 2); return u; }
inline float bhalf_at(uint32_t v, int i) { uint32_t u = ((v >> (16 * i)) & 0xFFFF) << 16; float f; memcpy(&f, &u, 4); return f; }
#endif
TF_HD uint32_t hmul2(uint32_t a, uint32_t b) {
#if TF_DEVICE
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
#else
  return to_half((double)half_at(a, 0) * half_at(b, 0)) | to_half((double)half_at(a, 1) * half_at(b, 1)) << 16;
#endif
}
TF_HD uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
#if TF_DEVICE
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
#else
  return to_half((double)half_at(a, 0) * half_at(b, 0) + half_at(c, 0)) | to_half((double)half_at(a, 1) * half_at(b, 1) + half_at(c, 1)) << 16;
#endif
}
constexpr uint32_t dup(uint32_t h) { return h | h << 16; }
constexpr uint32_t half_pow2(int e) { return e >= -14 ? (uint32_t)(e + 15) << 10 : 1u << (e + 24); }        // 2^e, -24 <= e <= 15
constexpr uint32_t kNeg = 0x8000;
// Both halves (byte SEL of w + BIAS) * 2^E, BIAS 0 or -128 (the subtraction of 1024 - BIAS is exact).
template <int SEL, int E, int BIAS = 0>
TF_HD uint32_t byte_scale(uint32_t w) {
  // half bits 0x64bb are 1024 + b; (1024 - BIAS) * 2^E has at most four significant bits
  constexpr uint32_t c = BIAS == 0 ? half_pow2(10 + E) : half_pow2(10 + E) | (uint32_t)(-BIAS / 128) << 7;
  static_assert(BIAS == 0 || BIAS == -128, "");
  return hfma2(prmt(w, 0x64646464u, SEL * 0x0101 + 0x4040), dup(half_pow2(E)), dup(c | kNeg));
}
TF_HD uint32_t small_scale(uint32_t v) {         // both halves v * 2^4, v < 1024
  return hfma2((v * 0x00010001u) | 0x64006400u, dup(half_pow2(4)), dup(half_pow2(14) | kNeg));
}
// The pair of bytes of w that sel picks, each below 128, as two bfloat16: 0x43vv is 128 + v.
TF_HD uint32_t bf16_pair(uint32_t w, uint32_t sel) {
  const uint32_t v = prmt(w, 0x43434343u, sel);
#if TF_DEVICE
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(v), "r"(0x3F803F80u), "r"(0xC300C300u));
  return r;
#else
  uint32_t r = 0;
  for (int i = 0; i < 2; i++) { const float f = bhalf_at(v, i) - 128.0f; uint32_t u; memcpy(&u, &f, 4); r |= (u >> 16) << (16 * i); }
  return r;
#endif
}
TF_HD void scale4(const uint32_t (&p)[4], uint32_t s, uint32_t (&a)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) a[i] = hmul2(p[i], s);
}
TF_HD void scale4(const uint32_t (&p)[4], uint32_t s, uint32_t o, uint32_t (&a)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) a[i] = hfma2(p[i], s, o);
}
TF_HD uint32_t rotl(uint32_t v, int n) {
#if TF_DEVICE
  return __funnelshift_l(v, v, n);
#else
  n &= 31;
  return n ? v << n | v >> (32 - n) : v;
#endif
}

// The 6-bit scales and mins of sub-blocks 2t, 2t + 1 from the headers of two rows: bytes 0 and 1 of scp and mnp are the first row's,
// bytes 2 and 3 the second's (both rows in one word: half the operations of unpacking each).
TF_HD void k_scales(const uint32_t (&h0)[4], const uint32_t (&h1)[4], int t, uint32_t& scp, uint32_t& mnp) {
  const uint32_t sel = t & 1 ? 0x7632u : 0x5410u;
  const uint32_t a = prmt(h0[1], h1[1], sel), m = prmt(h0[2], h1[2], sel), md = prmt(h0[3], h1[3], sel);
  const bool low = t < 2;
  scp = low ? (a & 0x3F3F3F3Fu) : ((md & 0x0F0F0F0Fu) | ((a >> 2) & 0x30303030u));
  mnp = low ? (m & 0x3F3F3F3Fu) : (((md >> 4) & 0x0F0F0F0Fu) | ((m >> 2) & 0x30303030u));
}

struct Q4K {
  typedef tf::Q4K Base;
  static constexpr int kPlanes = 1, kMins = 2;
  struct Run { uint32_t q[8], s[2], mn[1]; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) { Base::src_quads(t, o, a, b); }
  TF_HD static void load(const BlockLd& ld0, const BlockLd& ld1, int t, Run& r0, Run& r1) {
    uint32_t h0[4], h1[4], scp, mnp;
    ld0.words<4, 16>(0, h0);
    ld1.words<4, 16>(0, h1);
    ld0.words<8, 16>(16 + 32 * t, r0.q);
    ld1.words<8, 16>(16 + 32 * t, r1.q);
    r0.d = f16_bits_to_float(h0[0] & 0xFFFF); r0.nd = -f16_bits_to_float(h0[0] >> 16);
    r1.d = f16_bits_to_float(h1[0] & 0xFFFF); r1.nd = -f16_bits_to_float(h1[0] >> 16);
    k_scales(h0, h1, t, scp, mnp);
    // high nibbles stay in place: code * 16
    r0.s[0] = byte_scale<0, 4>(scp); r0.s[1] = byte_scale<1, 0>(scp); r0.mn[0] = bf16_pair(mnp, 0x4140);
    r1.s[0] = byte_scale<2, 4>(scp); r1.s[1] = byte_scale<3, 0>(scp); r1.mn[0] = bf16_pair(mnp, 0x4342);
  }
  TF_HD static void octet(const Run& r, int q, const Tables&, uint32_t (&a)[4], uint32_t (&)[4]) {
    const uint32_t m = q >= 4 ? 0x00F000F0u : 0x000F000Fu, w0 = r.q[2 * (q & 3)], w1 = r.q[2 * (q & 3) + 1];
    const uint32_t p[4] = {w0 & m, (w0 >> 8) & m, w1 & m, (w1 >> 8) & m};
    scale4(p, r.s[q >> 2], a);
  }
};

struct Q5K {
  typedef tf::Q5K Base;
  static constexpr int kPlanes = 1, kMins = 2;
  struct Run { uint32_t q[8], h[8], s[2], mn[1]; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) { a = 64 * t + 8 * o; b = a + 4; }
  TF_HD static void load(const BlockLd& ld0, const BlockLd& ld1, int t, Run& r0, Run& r1) {
    uint32_t h0[4], h1[4], scp, mnp;
    ld0.words<4, 16>(0, h0);
    ld1.words<4, 16>(0, h1);
    ld0.words<8, 16>(16, r0.h);
    ld1.words<8, 16>(16, r1.h);
    ld0.words<8, 16>(48 + 32 * t, r0.q);
    ld1.words<8, 16>(48 + 32 * t, r1.q);
    r0.d = f16_bits_to_float(h0[0] & 0xFFFF); r0.nd = -f16_bits_to_float(h0[0] >> 16);
    r1.d = f16_bits_to_float(h1[0] & 0xFFFF); r1.nd = -f16_bits_to_float(h1[0] >> 16);
    k_scales(h0, h1, t, scp, mnp);
    r0.s[0] = byte_scale<0, 4>(scp); r0.s[1] = byte_scale<1, 4>(scp); r0.mn[0] = bf16_pair(mnp, 0x4140);
    r1.s[0] = byte_scale<2, 4>(scp); r1.s[1] = byte_scale<3, 4>(scp); r1.mn[0] = bf16_pair(mnp, 0x4342);
    // the fifth bits of sub-blocks 2t and 2t + 1 to bits 4 and 5 of every byte
#pragma unroll
    for (int i = 0; i < 8; i++) { r0.h[i] = rotl(r0.h[i], 4 - 2 * t); r1.h[i] = rotl(r1.h[i], 4 - 2 * t); }
  }
  TF_HD static void octet(const Run& r, int q, const Tables&, uint32_t (&a)[4], uint32_t (&)[4]) {
    uint32_t p[4];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint32_t w = q >= 4 ? r.q[2 * (q & 3) + i] >> 4 : r.q[2 * (q & 3) + i], h = q >= 4 ? r.h[2 * (q & 3) + i] >> 1 : r.h[2 * (q & 3) + i];
      const uint32_t u = (w & 0x0F0F0F0Fu) | (h & 0x10101010u);
      p[2 * i] = pair02(u); p[2 * i + 1] = pair13(u);
    }
    scale4(p, r.s[q >> 2], a);
  }
};

// Group c of the run: low nibbles in plane a, (2-bit high - 2) * 16 in plane b.
struct Q6K {
  typedef tf::Q6K Base;
  static constexpr int kPlanes = 2, kMins = 0;
  struct Run { uint32_t qa[4], qb[4], qh[4], s[4]; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) {
    a = 128 * (t >> 1) + 32 * (o >> 1) + 16 * (t & 1) + 8 * (o & 1);
    b = a + 4;
  }
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    const int h = t >> 1, u = t & 1;
    ld.words16(64 * h + 16 * u, r.qa);
    ld.words16(64 * h + 32 + 16 * u, r.qb);
    ld.words16(128 + 32 * h + 16 * u, r.qh);
    uint32_t sc[2];
    ld.words<2, 2>(192 + 8 * h, sc);
    r.d = f16_bits_to_float(ld.u16(208));
    r.nd = 0.f;
    // scale bytes 2c + u of the eight, flipped to unsigned: 128 + scale
    const uint32_t s0 = (sc[0] >> (8 * u)) ^ 0x00800080u, s1 = (sc[1] >> (8 * u)) ^ 0x00800080u;
    r.s[0] = byte_scale<0, 4, -128>(s0); r.s[1] = byte_scale<2, 4, -128>(s0);
    r.s[2] = byte_scale<0, 4, -128>(s1); r.s[3] = byte_scale<2, 4, -128>(s1);
    return r;
  }
  TF_HD static void octet(const Run& r, int q, const Tables&, uint32_t (&a)[4], uint32_t (&b)[4]) {
    const int c = q >> 1, i = 2 * (q & 1);
    const uint32_t ml = c >= 2 ? 0x00F000F0u : 0x000F000Fu, mh = 0x00030003u << (2 * c);
    const uint32_t w0 = (c & 1) ? r.qb[i] : r.qa[i], w1 = (c & 1) ? r.qb[i + 1] : r.qa[i + 1], h0 = r.qh[i], h1 = r.qh[i + 1];
    const uint32_t pl[4] = {w0 & ml, (w0 >> 8) & ml, w1 & ml, (w1 >> 8) & ml}, ph[4] = {h0 & mh, (h0 >> 8) & mh, h1 & mh, (h1 >> 8) & mh};
    scale4(pl, c >= 2 ? hmul2(r.s[c], dup(half_pow2(-4))) : r.s[c], a);
    scale4(ph, c == 2 ? r.s[c] : hmul2(r.s[c], dup(half_pow2(4 - 2 * c))), hmul2(r.s[c], dup(half_pow2(-19) | kNeg)), b);      // -32 * scale * 2^-20
  }
};

struct Q2K {
  typedef tf::Q2K Base;
  static constexpr int kPlanes = 1, kMins = 4;
  struct Run { uint32_t q[4], s[4], mn[2]; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) { Base::src_quads(t, o, a, b); }
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    uint32_t dd[1], s2[2];
    ld.words<4, 4>(16 + 16 * t, r.q);
    ld.words<1, 4>(80, dd);
    ld.words<2, 4>(8 * (t >> 1), s2);
    r.d = f16_bits_to_float(dd[0] & 0xFFFF);
    r.nd = -f16_bits_to_float(dd[0] >> 16);
    // bytes 0 and 2: the scale bytes of groups 0, 1 (2, 3)
    const uint32_t b0 = (s2[0] >> (8 * (t & 1))) & 0x00FF00FFu, b1 = (s2[1] >> (8 * (t & 1))) & 0x00FF00FFu;
    const uint32_t c0 = b0 & 0x000F000Fu, c1 = b1 & 0x000F000Fu;
    r.s[0] = byte_scale<0, 4>(c0); r.s[1] = byte_scale<2, 2>(c0); r.s[2] = byte_scale<0, 0>(c1); r.s[3] = byte_scale<2, -2>(c1);
    r.mn[0] = bf16_pair(b0 >> 4, 0x4240); r.mn[1] = bf16_pair(b1 >> 4, 0x4240);
    return r;
  }
  TF_HD static void octet(const Run& r, int q, const Tables&, uint32_t (&a)[4], uint32_t (&)[4]) {
    const uint32_t m = 0x00030003u << (2 * (q >> 1)), w0 = r.q[2 * (q & 1)], w1 = r.q[2 * (q & 1) + 1];
    const uint32_t p[4] = {w0 & m, (w0 >> 8) & m, w1 & m, (w1 >> 8) & m};
    scale4(p, r.s[q >> 1], a);
  }
};

struct Q3K {
  typedef tf::Q3K Base;
  static constexpr int kPlanes = 1, kMins = 0;
  struct Run { uint32_t q[4], hm[4], s[4]; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) { Base::src_quads(t, o, a, b); }
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    const int h = t >> 1, u = t & 1;
    ld.words16(32 + 32 * h + 16 * u, r.q);
    ld.words16(16 * u, r.hm);
    uint32_t sc[3];
    ld.words<3, 2>(96, sc);
    r.d = f16_bits_to_float(ld.u16(108));
    r.nd = 0.f;
    // third bit of group s (bit 4 h + s) to bit 2 + s of every byte
#pragma unroll
    for (int i = 0; i < 4; i++) r.hm[i] = rotl(r.hm[i], 2 - 4 * h);
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const uint32_t lo = (sc[s >> 1] >> (16 * (s & 1) + 8 * u + 4 * h)) & 15;
      const uint32_t hi = (sc[2] >> (16 * (s & 1) + 8 * u + 4 * h + 2 * (s >> 1))) & 3;
      // 16 * (scale - 32): 0x6400 | v is 1024 + v, 1056 * 16 has six significant bits
      r.s[s] = hfma2(((lo | (hi << 4)) * 0x00010001u) | 0x64006400u, dup(half_pow2(4)), dup((half_pow2(14) | 32) | kNeg));
    }
    return r;
  }
  TF_HD static void octet(const Run& r, int q, const Tables&, uint32_t (&a)[4], uint32_t (&)[4]) {
    const int s = q >> 1;
    uint32_t p[4];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint32_t c = ((r.q[2 * (q & 1) + i] >> (2 * s)) & 0x03030303u) | ((r.hm[2 * (q & 1) + i] >> s) & 0x04040404u);
      p[2 * i] = pair02(c); p[2 * i + 1] = pair13(c);
    }
    scale4(p, r.s[s], hmul2(r.s[s], dup(half_pow2(-22) | kNeg)), a);      // -4 * scale * 2^-20
  }
};

// Grid formats: the tile format's run and group, the scale d * (2 s + 1) split into 2 s + 1 and a power-of-two multiple of d.
template <class B, int GROUP_OCT>
struct GridFormat {
  typedef B Base;
  static constexpr int kPlanes = 1, kMins = 0, kGroups = 8 / GROUP_OCT;
  struct Run { typename B::Run r; uint32_t s[kGroups]; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) { B::src_quads(t, o, a, b); }
  TF_HD static void octet(const Run& r, int q, const Tables& tb, uint32_t (&a)[4], uint32_t (&)[4]) {
    uint32_t p[4];
    B::octet(B::load_group(BlockLd{}, r.r, 0, q / GROUP_OCT), q % GROUP_OCT, tb, p);
    scale4(p, r.s[q / GROUP_OCT], a);
  }
};
struct IQ2XXS : GridFormat<tf::IQ2XXS, 4> {
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    r.r = Base::load_run(ld, t);
    r.d = mulf(r.r.d4, 0.5f); r.nd = 0.f;
    for (int g = 0; g < 2; g++) r.s[g] = small_scale(2 * (r.r.q[2 * g + 1] >> 28) + 1);
    return r;
  }
};
struct IQ2XS : GridFormat<tf::IQ2XS, 2> {
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    r.r = Base::load_run(ld, t);
    r.d = mulf(r.r.d4, 0.5f); r.nd = 0.f;
    for (int g = 0; g < 4; g++) r.s[g] = small_scale(2 * ((r.r.sc >> (4 * g)) & 15) + 1);
    return r;
  }
};
struct IQ2S : GridFormat<tf::IQ2S, 2> {
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    r.r = Base::load_run(ld, t);
    r.d = mulf(r.r.d4, 0.5f); r.nd = 0.f;
    for (int g = 0; g < 4; g++) r.s[g] = small_scale(2 * ((r.r.sc >> (4 * g)) & 15) + 1);
    return r;
  }
};
struct IQ3XXS : GridFormat<tf::IQ3XXS, 4> {
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    r.r = Base::load_run(ld, t);
    r.d = mulf(r.r.d2, 0.5f); r.nd = 0.f;
    for (int g = 0; g < 2; g++) r.s[g] = small_scale(2 * (r.r.aux[g] >> 28) + 1);
    return r;
  }
};
struct IQ3S : GridFormat<tf::IQ3S, 4> {
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    r.r = Base::load_run(ld, t);
    r.d = r.r.d; r.nd = 0.f;
    for (int g = 0; g < 2; g++) r.s[g] = small_scale(2 * ((r.r.sc >> (4 * g)) & 15) + 1);
    return r;
  }
};
// IQ1: codes 8 * grid + 9 + delta; the 9 comes out with the scale.
template <class B, int GROUP_OCT>
struct Iq1Format : GridFormat<B, GROUP_OCT> {
  typedef typename GridFormat<B, GROUP_OCT>::Run Run;
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    r.r = B::load_run(ld, t);
    r.d = r.r.d8; r.nd = 0.f;
    for (int g = 0; g < 8 / GROUP_OCT; g++) {
      uint32_t s;
      if constexpr (GROUP_OCT == 4) s = r.r.qh[0] >> (16 * g + 12);
      else s = r.r.w >> (3 * g);
      r.s[g] = small_scale(2 * (s & 7) + 1);
    }
    return r;
  }
  TF_HD static void octet(const Run& r, int q, const Tables& tb, uint32_t (&a)[4], uint32_t (&)[4]) {
    uint32_t p[4];
    B::octet(B::load_group(BlockLd{}, r.r, 0, q / GROUP_OCT), q % GROUP_OCT, tb, p);
    const uint32_t s = r.s[q / GROUP_OCT];
    scale4(p, s, hmul2(s, dup(9u | kNeg)), a);           // half bits 0x8009 are -9 * 2^-24
  }
};
struct IQ1S : Iq1Format<tf::IQ1S, 4> {};
struct IQ1M : Iq1Format<tf::IQ1M, 2> {};

// Code book values as signed codes (the batch kernel's table of byte pairs); ls * value rounded to float16 and what that left out.
struct IQ4XS {
  typedef tf::IQ4XS Base;
  static constexpr int kPlanes = 2, kMins = 0;
  struct Run { uint32_t q[8], s[2]; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) { Base::src_quads(t, o, a, b); }
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    uint32_t h[2];
    ld.words<2, 8>(0, h);                    // d | scales_h << 16, scales_l[0..3]
    ld.words<8, 8>(8 + 32 * t, r.q);
    r.d = f16_bits_to_float(h[0] & 0xFFFF);
    r.nd = 0.f;
#pragma unroll
    for (int g = 0; g < 2; g++) {
      const int j = 2 * t + g;
      const uint32_t ls = ((h[1] >> (4 * j)) & 15) | (((h[0] >> (16 + 2 * j)) & 3) << 4);
      r.s[g] = hfma2((ls * 0x00010001u) | 0x64006400u, dup(half_pow2(4)), dup((half_pow2(14) | 32) | kNeg));
    }
    return r;
  }
  TF_HD static void octet(const Run& r, int q, const Tables& tb, uint32_t (&a)[4], uint32_t (&b)[4]) {
    uint32_t p[4];
    lookup_octet(tb, r.q[q], p);
#if !TF_DEVICE
    for (int i = 0; i < 4; i++) {            // the host's table holds value + 128 bytes
      uint32_t v = 0;
      for (int h = 0; h < 2; h++) { const int c = (int)((p[i] >> (16 * h)) & 0xFF) - 128; v |= (uint32_t)(c < 0 ? 0x8000 - c : c) << (16 * h); }
      p[i] = v;
    }
#endif
    const uint32_t s = r.s[q >> 2];
    scale4(p, s, a);
#pragma unroll
    for (int i = 0; i < 4; i++) b[i] = hfma2(p[i], s, a[i] ^ 0x80008000u);
  }
};

struct TQ20 {
  typedef tf::TQ20 Base;
  static constexpr int kPlanes = 1, kMins = 0;
  struct Run { uint32_t q[4]; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) { Base::src_quads(t, o, a, b); }
  TF_HD static Run load(const BlockLd& ld, int t) {
    Run r;
    ld.words16(16 * t, r.q);
    r.d = f16_bits_to_float(ld.u16(64));
    r.nd = 0.f;
    return r;
  }
  TF_HD static void octet(const Run& r, int q, const Tables&, uint32_t (&a)[4], uint32_t (&)[4]) {
    const int s = q >> 1;
    const uint32_t m = 0x00030003u << (2 * s), w0 = r.q[2 * (q & 1)], w1 = r.q[2 * (q & 1) + 1];
    const uint32_t p[4] = {w0 & m, (w0 >> 8) & m, w1 & m, (w1 >> 8) & m};
    scale4(p, dup(half_pow2(4 - 2 * s)), dup(half_pow2(-kExp) | kNeg), a);
  }
};
struct TQ10 {
  typedef tf::TQ10 Base;
  static constexpr int kPlanes = 1, kMins = 0;
  struct Run { BlockLd ld; int t; float d, nd; };
  TF_HD static void src_quads(int t, int o, int& a, int& b) { Base::src_quads(t, o, a, b); }
  TF_HD static Run load(const BlockLd& ld, int t) { return Run{ld, t, f16_bits_to_float(ld.u16(52)), 0.f}; }
  TF_HD static void octet(const Run& r, int q, const Tables& tb, uint32_t (&a)[4], uint32_t (&)[4]) {
    uint32_t p[4];
    Base::octet(Base::Group{r.ld, r.d, r.t}, q, tb, p);
    scale4(p, dup(half_pow2(4)), dup(half_pow2(-kExp) | kNeg), a);
  }
};

// Run t of two rows.
template <class F>
TF_HD void load_pair(const BlockLd& ld0, const BlockLd& ld1, int t, typename F::Run& r0, typename F::Run& r1) {
  if constexpr (F::kMins == 2) F::load(ld0, ld1, t, r0, r1);
  else { r0 = F::load(ld0, t); r1 = F::load(ld1, t); }
}

}  // namespace bf
}  // namespace ggq
