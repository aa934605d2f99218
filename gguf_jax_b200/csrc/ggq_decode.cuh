// Per-qtype block decoders: decode8<QT>(block, g, tables, out) writes the eight
// consecutive elements 8g .. 8g+7 of one block as float32.
//
// The arithmetic is the float32 arithmetic of gguf.quants / gguf-jax
// (src/gguf_jax/quants.py:125-712) in the same association, written with __fmul_rn /
// __fadd_rn / __fsub_rn so the compiler can neither contract nor reassociate it.  Every
// product is exact in float32 (f16 scale x small integer), so the only rounding is the
// final add/sub of Q4_1, Q5_1, Q2_K, Q4_K and Q5_K -- which is why the result is
// bit-identical to the numpy decode.  No flush-to-zero: MXFP4 scales below 2^-126 are
// float32 subnormals.
//
// Most block sizes (18, 22, 34, 50, 66, 110, 210 ...) give no alignment beyond two bytes, MXFP4's 17 none: loads are
// as wide as a block's alignment allows.
#pragma once

#include "ggq_common.cuh"

// Where the block bytes live.  By default they are read from global memory through the
// read-only path (__ldg).  A translation unit that stages raw blocks in shared memory first
// (gemm_tcgen05.cu) defines GGQ_DECODE_GENERIC_LOADS before including this header and gets the
// same decoders with plain generic loads, which work on shared and global addresses alike.
// The two flavours live in different inline namespaces, so they are different entities.
#ifdef GGQ_DECODE_GENERIC_LOADS
#define GGQ_LD(p) (*(p))
#define GGQ_DEC_NS dec_generic_loads
#else
#define GGQ_LD(p) __ldg(p)
#define GGQ_DEC_NS dec_global_loads
#endif

namespace ggq {
inline namespace GGQ_DEC_NS {

__device__ __forceinline__ uint32_t ldb(const uint8_t* p) { return GGQ_LD(p); }
__device__ __forceinline__ uint32_t ld16(const uint8_t* p) { return ldb(p) | (ldb(p + 1) << 8); }
__device__ __forceinline__ uint32_t ld32(const uint8_t* p) {
  return ldb(p) | (ldb(p + 1) << 8) | (ldb(p + 2) << 16) | (ldb(p + 3) << 24);
}
// Eight consecutive block bytes as two little-endian words, with loads as wide as the block's
// alignment allows.  ALIGN is the guaranteed alignment of p: a tensor starts 16-byte aligned and
// every block starts a multiple of its size further on, so ALIGN = gcd(block bytes, 16) combined
// with the (even) offset inside the block.
template <int ALIGN>
__device__ __forceinline__ uint2 ld8(const uint8_t* p) {
  if constexpr (ALIGN >= 8) {
    return GGQ_LD(reinterpret_cast<const uint2*>(p));
  } else if constexpr (ALIGN >= 4) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p);
    return make_uint2(GGQ_LD(q), GGQ_LD(q + 1));
  } else if constexpr (ALIGN >= 2) {
#ifdef GGQ_DECODE_GENERIC_LOADS
    // staged blocks: four short loads of shared memory (2048 x 2048 Q8_0 at batch 1 3.9 us, as words 4.4)
    const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
    return make_uint2((uint32_t)GGQ_LD(q) | ((uint32_t)GGQ_LD(q + 1) << 16),
                      (uint32_t)GGQ_LD(q + 2) | ((uint32_t)GGQ_LD(q + 3) << 16));
#else
    // the two or three aligned words that hold the bytes (never one that holds none of them)
    const uint32_t sh = ((uintptr_t)p & 2) * 8;
    const uint32_t* q = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
    const uint32_t a = GGQ_LD(q), b = GGQ_LD(q + 1), c = sh ? GGQ_LD(q + 2) : 0u;
    return make_uint2(__funnelshift_r(a, b, sh), __funnelshift_r(b, c, sh));
#endif
  } else {
    return make_uint2(ld32(p), ld32(p + 4));
  }
}

// Eight bytes at any address, as the aligned words that hold them (never one that holds none of them).
__device__ __forceinline__ uint2 ld8_any(const uint8_t* p) {
  const uint32_t sh = 8 * ((uintptr_t)p & 3);
  const uint32_t* q = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
  const uint32_t a = GGQ_LD(q), b = GGQ_LD(q + 1), c = sh ? GGQ_LD(q + 2) : 0u;
  return make_uint2(__funnelshift_r(a, b, sh), __funnelshift_r(b, c, sh));
}
// Two and four bytes at an even address.
__device__ __forceinline__ uint32_t ld16a(const uint8_t* p) { return GGQ_LD(reinterpret_cast<const unsigned short*>(p)); }
__device__ __forceinline__ uint32_t ld32a(const uint8_t* p) { return ld16a(p) | (ld16a(p + 2) << 16); }

// Float32 arithmetic on pairs.  Written as instructions, so nothing is contracted or reassociated: a product and a sum are
// rounded on their own, fma_pair rounds once (used only where the product is exact, so that it equals product then sum).
__device__ __forceinline__ void add_pair(float& a, float& b, float c) {
  asm("{ .reg .b64 x, k;\n mov.b64 x, {%0, %1};\n mov.b64 k, {%2, %2};\n add.rn.f32x2 x, x, k;\n mov.b64 {%0, %1}, x; }" : "+f"(a), "+f"(b) : "f"(c));
}
__device__ __forceinline__ void mul_pair(float& a, float& b, float c) {
  asm("{ .reg .b64 x, k;\n mov.b64 x, {%0, %1};\n mov.b64 k, {%2, %2};\n mul.rn.f32x2 x, x, k;\n mov.b64 {%0, %1}, x; }" : "+f"(a), "+f"(b) : "f"(c));
}
__device__ __forceinline__ void fma_pair(float& a, float& b, float m, float c) {
  asm("{ .reg .b64 x, k, l;\n mov.b64 x, {%0, %1};\n mov.b64 k, {%2, %2};\n mov.b64 l, {%3, %3};\n fma.rn.f32x2 x, x, k, l;\n mov.b64 {%0, %1}, x; }"
      : "+f"(a), "+f"(b) : "f"(m), "f"(c));
}
// The eight code bytes of (w0, w1) minus `bias` as exact floats: the bits 0x4B0000vv are 2^23 + v.
__device__ __forceinline__ void codes8(uint32_t w0, uint32_t w1, float bias, float* o) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    o[i] = __uint_as_float(__byte_perm(w0, 0x4B000000u, 0x7440 + i));
    o[4 + i] = __uint_as_float(__byte_perm(w1, 0x4B000000u, 0x7440 + i));
  }
#pragma unroll
  for (int i = 0; i < 8; i += 2) add_pair(o[i], o[i + 1], -(8388608.0f + bias));
}
__device__ __forceinline__ void mul8(float* o, float d) {
#pragma unroll
  for (int i = 0; i < 8; i += 2) mul_pair(o[i], o[i + 1], d);
}
__device__ __forceinline__ void fma8(float* o, float d, float m) {
#pragma unroll
  for (int i = 0; i < 8; i += 2) fma_pair(o[i], o[i + 1], d, m);
}
// Four bits (bit j of the low nibble of v) spread to bit 4 of byte j, and to 0x80 in byte j.
__device__ __forceinline__ uint32_t spread_bit4(uint32_t v) { return ((v & 15u) * 0x02040810u) & 0x10101010u; }
__device__ __forceinline__ uint32_t spread_sign(uint32_t v) { return (((v & 15u) * 0x00204081u) << 7) & 0x80808080u; }
// Four code bytes g < 128 with signs (0x80 in byte j of s: negative) as bytes 128 + g or 128 - g.
__device__ __forceinline__ uint32_t signed_bytes(uint32_t g, uint32_t s) {
  const uint32_t m = (s >> 7) * 255u;
  return 0x80808080u + (g & ~m) - (g & m);
}
// Sixteen-entry table lookup (four registers of bytes) of the four low nibbles of w's bytes.
__device__ __forceinline__ uint32_t lookup_bytes(const uint4& kv, uint32_t w) {
  const uint32_t x = w | (w >> 4);
  const uint32_t sel = __byte_perm(x, 0u, 0x4420);
  const uint32_t s7 = sel & 0x7777u;
  const uint32_t lo = __byte_perm(kv.x, kv.y, s7), hi = __byte_perm(kv.z, kv.w, s7);
  return __byte_perm(lo, hi, ((sel >> 1) & 0x4444u) | 0x3210u);
}
__device__ __forceinline__ uint4 table16(const uint8_t* tab, int offset) {     // int8 values + 128
  const uint4 v = GGQ_LD(reinterpret_cast<const uint4*>(tab + offset));
  return make_uint4(v.x ^ 0x80808080u, v.y ^ 0x80808080u, v.z ^ 0x80808080u, v.w ^ 0x80808080u);
}

// IEEE half bits -> float (exact; cvt.f32.f16 keeps subnormals).
__device__ __forceinline__ float h2f(uint32_t bits) {
  return __half2float(__ushort_as_half((unsigned short)bits));
}
__device__ __forceinline__ float i2f(int v) { return (float)v; }
// ksigns[i] = i | parity(i) << 7 (gguf/quants.py IQ2_XXS.ksigns).
__device__ __forceinline__ uint32_t ksign(uint32_t i) { return i | ((__popc(i) & 1) << 7); }

// Compile-time block geometry (elements, bytes) of the block qtypes.
constexpr int block_elems_of(int qt) {
  return (qt == QT_Q4_0 || qt == QT_Q4_1 || qt == QT_Q5_0 || qt == QT_Q5_1 || qt == QT_Q8_0 ||
          qt == QT_IQ4_NL || qt == QT_MXFP4) ? 32 : (qt == QT_NVFP4 ? 64 : 256);
}
constexpr int block_bytes_of(int qt) {
  return qt == QT_Q4_0 ? 18 : qt == QT_Q4_1 ? 20 : qt == QT_Q5_0 ? 22 : qt == QT_Q5_1 ? 24 : qt == QT_Q8_0 ? 34 :
         qt == QT_Q2_K ? 84 : qt == QT_Q3_K ? 110 : qt == QT_Q4_K ? 144 : qt == QT_Q5_K ? 176 : qt == QT_Q6_K ? 210 :
         qt == QT_IQ2_XXS ? 66 : qt == QT_IQ2_XS ? 74 : qt == QT_IQ3_XXS ? 98 : qt == QT_IQ1_S ? 50 :
         qt == QT_IQ4_NL ? 18 : qt == QT_IQ3_S ? 110 : qt == QT_IQ2_S ? 82 : qt == QT_IQ4_XS ? 136 :
         qt == QT_IQ1_M ? 56 : qt == QT_TQ1_0 ? 54 : qt == QT_TQ2_0 ? 66 : qt == QT_MXFP4 ? 17 : 36;
}

template <int QT>
struct Dec;  // Dec<QT>::run(block, g, tables, out[8])

// Common shape: the eight codes are gathered as bytes of two words, turned into exact floats by codes8 and scaled in
// pairs, about four instructions per weight (byte-wise extraction with integer conversion took six to twenty).

// ---- legacy 32-element blocks ------------------------------------------------------
// nibble order: elements 0-15 = low nibbles of qs[0..15], 16-31 = high nibbles.
__device__ __forceinline__ uint32_t nibbles(uint32_t w, int g_hi) { return (w >> (4 * g_hi)) & 0x0F0F0F0Fu; }

template <> struct Dec<QT_Q4_0> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const float d = h2f(ld16a(b));
    const uint2 q = ld8<2>(b + 2 + 8 * (g & 1));
    codes8(nibbles(q.x, g >> 1), nibbles(q.y, g >> 1), 8.f, o);
    mul8(o, d);
  }
};
template <> struct Dec<QT_Q4_1> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const uint32_t dm = GGQ_LD(reinterpret_cast<const uint32_t*>(b));
    const uint2 q = ld8<4>(b + 4 + 8 * (g & 1));
    codes8(nibbles(q.x, g >> 1), nibbles(q.y, g >> 1), 0.f, o);
    fma8(o, h2f(dm & 0xFFFF), h2f(dm >> 16));          // d * q is exact: 11 x 4 bits
  }
};
template <> struct Dec<QT_Q5_0> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const float d = h2f(ld16a(b));
    const uint32_t qh = ld32a(b + 2) >> (8 * g);
    const uint2 q = ld8<2>(b + 6 + 8 * (g & 1));
    codes8(nibbles(q.x, g >> 1) | spread_bit4(qh), nibbles(q.y, g >> 1) | spread_bit4(qh >> 4), 16.f, o);
    mul8(o, d);
  }
};
template <> struct Dec<QT_Q5_1> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const uint2 h = ld8<8>(b);                          // d | m, fifth bits
    const uint32_t qh = h.y >> (8 * g);
    const uint2 q = ld8<8>(b + 8 + 8 * (g & 1));
    codes8(nibbles(q.x, g >> 1) | spread_bit4(qh), nibbles(q.y, g >> 1) | spread_bit4(qh >> 4), 0.f, o);
    fma8(o, h2f(h.x & 0xFFFF), h2f(h.x >> 16));         // d * q is exact: 11 x 5 bits
  }
};
template <> struct Dec<QT_Q8_0> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const float d = h2f(ld16a(b));
    const uint2 q = ld8<2>(b + 2 + 8 * g);
    codes8(q.x ^ 0x80808080u, q.y ^ 0x80808080u, 128.f, o);
    mul8(o, d);
  }
};
template <> struct Dec<QT_IQ4_NL> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const uint4 kv = table16(tab, TAB_KV_IQ4);
    const float d = h2f(ld16a(b));
    const uint2 q = ld8<2>(b + 2 + 8 * (g & 1));
    codes8(lookup_bytes(kv, nibbles(q.x, g >> 1)), lookup_bytes(kv, nibbles(q.y, g >> 1)), 128.f, o);
    mul8(o, d);
  }
};
template <> struct Dec<QT_MXFP4> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const uint4 kv = table16(tab, TAB_KV_MXFP4);
    const uint32_t e = ldb(b);
    const float d = __uint_as_float(e < 2 ? (0x00200000u << e) : ((e - 1) << 23));
    const uint2 q = ld8_any(b + 1 + 8 * (g & 1));
    codes8(lookup_bytes(kv, nibbles(q.x, g >> 1)), lookup_bytes(kv, nibbles(q.y, g >> 1)), 128.f, o);
    mul8(o, d);
  }
};
// NVFP4: 64 elements, four UE4M3 sub-scales; elements 16s+j (low nibble of qs[8s+j]) and
// 16s+8+j (high nibble).
template <> struct Dec<QT_NVFP4> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const uint4 kv = table16(tab, TAB_KV_MXFP4);
    const int s = g >> 1;
    const uint32_t x = ldb(b + s);
    const int ex = (x >> 3) & 15;
    const float man = i2f(x & 7);
    const float raw = ex == 0 ? __fmul_rn(man, 0.001953125f)
                              : __fmul_rn(__fadd_rn(1.0f, __fmul_rn(man, 0.125f)),
                                          __uint_as_float((uint32_t)(ex - 7 + 127) << 23));
    const float d = (x == 0 || x == 0x7F) ? 0.0f : __fmul_rn(raw, 0.5f);
    const uint2 q = ld8<4>(b + 4 + 8 * s);
    codes8(lookup_bytes(kv, nibbles(q.x, g & 1)), lookup_bytes(kv, nibbles(q.y, g & 1)), 128.f, o);
    mul8(o, d);
  }
};

// ---- K-quants -----------------------------------------------------------------------
template <> struct Dec<QT_Q2_K> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const uint32_t dd = GGQ_LD(reinterpret_cast<const uint32_t*>(b + 80)), sc = ldb(b + (g >> 1));
    const float dl = __fmul_rn(h2f(dd & 0xFFFF), i2f(sc & 15)), ml = __fmul_rn(h2f(dd >> 16), i2f(sc >> 4));
    const uint2 q = ld8<4>(b + 16 + 32 * (g >> 4) + 8 * (g & 3));
    const int sh = 2 * ((g >> 2) & 3);
    codes8((q.x >> sh) & 0x03030303u, (q.y >> sh) & 0x03030303u, 0.f, o);
    fma8(o, dl, -ml);                                   // dl * q is exact: 15 x 2 bits
  }
};
template <> struct Dec<QT_Q3_K> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const uint8_t* s = b + 96;
    const float d = h2f(ld16a(b + 108));
    const int i16 = g >> 1;
    const int lo = (ldb(s + (i16 & 7)) >> (4 * (i16 >> 3))) & 15;
    const int hi = (ldb(s + 8 + (i16 & 3)) >> (2 * (i16 >> 2))) & 3;
    const float dl = __fmul_rn(d, i2f((lo | (hi << 4)) - 32));
    const uint2 q = ld8<2>(b + 32 + 32 * (g >> 4) + 8 * (g & 3));
    const uint2 hm = ld8<2>(b + 8 * (g & 3));
    const int sh = 2 * ((g >> 2) & 3), hb = g >> 2;
    codes8(((q.x >> sh) & 0x03030303u) | (((hm.x >> hb) & 0x01010101u) << 2),
           ((q.y >> sh) & 0x03030303u) | (((hm.y >> hb) & 0x01010101u) << 2), 4.f, o);
    mul8(o, dl);
  }
};
// Q4_K / Q5_K blocks are 144 / 176 bytes: always 16-byte aligned, so the header is one
// 128-bit load and the eight quant bytes one 64-bit load.
__device__ __forceinline__ void scale_min_k4_words(const uint4& h, int k, int& sc, int& mn) {
  // h = (d|dmin, s0-3, s4-7, s8-11); 6-bit scale and min of sub-block k (src/gguf_jax/quants.py:275-283)
  const int sh = 8 * (k & 3);
  const uint32_t a = (h.y >> sh) & 0xFF, m = (h.z >> sh) & 0xFF, md = (h.w >> sh) & 0xFF;
  if (k < 4) { sc = a & 63; mn = m & 63; }
  else { sc = (md & 15) | ((a >> 6) << 4); mn = (md >> 4) | ((m >> 6) << 4); }
}
template <> struct Dec<QT_Q4_K> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const uint4 h = GGQ_LD(reinterpret_cast<const uint4*>(b));
    const float d = h2f(h.x & 0xFFFF), dmin = h2f(h.x >> 16);
    int k = g >> 2, sc, mn;
    scale_min_k4_words(h, k, sc, mn);
    const float dl = __fmul_rn(d, i2f(sc)), dm = __fmul_rn(dmin, i2f(mn));
    const uint2 q = ld8<8>(b + 16 + 32 * (k >> 1) + 8 * (g & 3));
    codes8(nibbles(q.x, k & 1), nibbles(q.y, k & 1), 0.f, o);
    fma8(o, dl, -dm);                                   // dl * q is exact: 17 x 4 bits
  }
};
template <> struct Dec<QT_Q5_K> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const uint4 h = GGQ_LD(reinterpret_cast<const uint4*>(b));
    const float d = h2f(h.x & 0xFFFF), dmin = h2f(h.x >> 16);
    int k = g >> 2, sc, mn;
    scale_min_k4_words(h, k, sc, mn);
    const float dl = __fmul_rn(d, i2f(sc)), dm = __fmul_rn(dmin, i2f(mn));
    const uint2 qh = ld8<8>(b + 16 + 8 * (g & 3));
    const uint2 q = ld8<8>(b + 48 + 32 * (k >> 1) + 8 * (g & 3));
    codes8(nibbles(q.x, k & 1) | (((qh.x >> k) & 0x01010101u) << 4), nibbles(q.y, k & 1) | (((qh.y >> k) & 0x01010101u) << 4), 0.f, o);
    fma8(o, dl, -dm);                                   // dl * q is exact: 17 x 5 bits
  }
};
// Q6_K blocks are 210 bytes: 2-byte aligned, all offsets below are even.
template <> struct Dec<QT_Q6_K> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const float d = h2f(ld16a(b + 208));
    const float dl = __fmul_rn(d, i2f((int8_t)ldb(b + 192 + (g >> 1))));
    const int c = g >> 2, t0 = 8 * (g & 3);
    const uint2 ql = ld8<2>(b + 64 * (c >> 2) + 32 * (c & 1) + t0);
    const uint2 qh = ld8<2>(b + 128 + 32 * (c >> 2) + t0);
    const int n = (c >> 1) & 1, shh = 2 * (c & 3);
    codes8(nibbles(ql.x, n) | (((qh.x >> shh) & 0x03030303u) << 4), nibbles(ql.y, n) | (((qh.y >> shh) & 0x03030303u) << 4), 32.f, o);
    mul8(o, dl);
  }
};

// ---- ternary --------------------------------------------------------------------------
template <> struct Dec<QT_TQ1_0> {
  // base-3 digits of four bytes at a time, as the bytes (0, 2) and (1, 3) of two words
  __device__ static uint32_t digits(uint32_t bytes02, uint32_t pow3) {
    return ((((bytes02 & 0x00FF00FFu) * pow3) & 0x00FF00FFu) * 3u >> 8) & 0x00030003u;
  }
  __device__ static uint32_t pow3(int n) { return n < 4 ? (0x1B090301u >> (8 * n)) & 0xFFu : 81u; }
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const float d = h2f(ld16a(b + 52));
    const int last = g >= 30 ? 1 : 0;
    const int off = g < 20 ? 8 * (g & 3) : last ? 48 : 32 + 8 * (g & 1);
    const int n = g < 20 ? g >> 2 : last ? 2 * (g - 30) : (g - 20) >> 1;
    const uint32_t w0 = ld32a(b + off), w1 = last ? w0 : ld32a(b + off + 4);
    const uint32_t pa = pow3(n), pb = pow3(n + last);
    codes8(digits(w0, pa) | (digits(w0 >> 8, pa) << 8), digits(w1, pb) | (digits(w1 >> 8, pb) << 8), 1.f, o);
    mul8(o, d);
  }
};
template <> struct Dec<QT_TQ2_0> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t*, float* o) {
    const float d = h2f(ld16a(b + 64));
    const uint2 q = ld8<2>(b + 32 * (g >> 4) + 8 * (g & 3));
    const int sh = 2 * ((g >> 2) & 3);
    codes8((q.x >> sh) & 0x03030303u, (q.y >> sh) & 0x03030303u, 1.f, o);
    mul8(o, d);
  }
};

// ---- codebook (I-quant) types ------------------------------------------------------------
// db * grid is exact (at most 17 x 6 bits), so a negative weight is the negated grid value times db.
__device__ __forceinline__ void signed_grid8(uint32_t g0, uint32_t g1, uint32_t signs, float db, float* o) {
  codes8(signed_bytes(g0, spread_sign(signs)), signed_bytes(g1, spread_sign(signs >> 4)), 128.f, o);
  mul8(o, db);
}
__device__ __forceinline__ uint2 grid8(const uint8_t* tab, int offset, uint32_t i) { return GGQ_LD(reinterpret_cast<const uint2*>(tab + offset) + i); }
__device__ __forceinline__ uint32_t grid4(const uint8_t* tab, int offset, uint32_t i) { return GGQ_LD(reinterpret_cast<const uint32_t*>(tab + offset) + i); }

template <> struct Dec<QT_IQ2_XXS> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const float d = h2f(ld16a(b));
    const int ib = g >> 2, l = g & 3;
    const uint32_t aux = ld32a(b + 2 + 8 * ib + 4);
    const float db = __fmul_rn(__fmul_rn(d, __fadd_rn(0.5f, i2f(aux >> 28))), 0.25f);
    const uint2 gr = grid8(tab, TAB_IQ2_XXS, ldb(b + 2 + 8 * ib + l));
    signed_grid8(gr.x, gr.y, ksign((aux >> (7 * l)) & 127), db, o);
  }
};
template <> struct Dec<QT_IQ2_XS> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const float d = h2f(ld16a(b));
    const uint32_t q = ld16a(b + 2 + 2 * g);
    const uint32_t s = (ldb(b + 66 + (g >> 2)) >> (4 * ((g >> 1) & 1))) & 15;
    const float db = __fmul_rn(__fmul_rn(d, __fadd_rn(0.5f, i2f(s))), 0.25f);
    const uint2 gr = grid8(tab, TAB_IQ2_XS, q & 511);
    signed_grid8(gr.x, gr.y, ksign(q >> 9), db, o);
  }
};
template <> struct Dec<QT_IQ2_S> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const float d = h2f(ld16a(b));
    const uint32_t s = (ldb(b + 74 + (g >> 2)) >> (4 * ((g >> 1) & 1))) & 15;
    const float db = __fmul_rn(__fmul_rn(d, __fadd_rn(0.5f, i2f(s))), 0.25f);
    const uint32_t idx = ldb(b + 2 + g) | (((ldb(b + 66 + (g >> 2)) >> (2 * (g & 3))) & 3) << 8);
    const uint2 gr = grid8(tab, TAB_IQ2_S, idx);
    signed_grid8(gr.x, gr.y, ldb(b + 34 + g), db, o);
  }
};
template <> struct Dec<QT_IQ3_XXS> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const float d = h2f(ld16a(b));
    const int ib = g >> 2, l = g & 3;
    const uint32_t aux = ld32a(b + 66 + 4 * ib);
    const float db = __fmul_rn(__fmul_rn(d, __fadd_rn(0.5f, i2f(aux >> 28))), 0.5f);
    const uint32_t q = ld16a(b + 2 + 2 * g);
    signed_grid8(grid4(tab, TAB_IQ3_XXS, q & 0xFF), grid4(tab, TAB_IQ3_XXS, q >> 8), ksign((aux >> (7 * l)) & 127), db, o);
  }
};
template <> struct Dec<QT_IQ3_S> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const float d = h2f(ld16a(b));
    const uint32_t s = (ldb(b + 106 + (g >> 3)) >> (4 * ((g >> 2) & 1))) & 15;
    const float db = __fmul_rn(d, i2f(1 + 2 * s));
    const uint32_t qh = ldb(b + 66 + (g >> 2)) >> (2 * (g & 3));
    const uint32_t q = ld16a(b + 2 + 2 * g);
    const uint32_t i0 = (q & 0xFF) | ((qh & 1) << 8), i1 = (q >> 8) | (((qh >> 1) & 1) << 8);
    signed_grid8(grid4(tab, TAB_IQ3_S, i0), grid4(tab, TAB_IQ3_S, i1), ldb(b + 74 + g), db, o);
  }
};
// dl * (grid + delta), both factors exact; the int8 grid values are biased to bytes
__device__ __forceinline__ void delta_grid8(const uint2& gr, float delta, float dl, float* o) {
  codes8(gr.x ^ 0x80808080u, gr.y ^ 0x80808080u, 128.f, o);
#pragma unroll
  for (int i = 0; i < 8; i += 2) add_pair(o[i], o[i + 1], delta);
  mul8(o, dl);
}
template <> struct Dec<QT_IQ1_S> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const float d = h2f(ld16a(b));
    const int ib = g >> 2, l = g & 3;
    const uint32_t qh = ld16a(b + 34 + 2 * ib);
    const float dl = __fmul_rn(d, i2f(2 * ((qh >> 12) & 7) + 1));
    const float delta = (qh & 0x8000) ? -0.125f : 0.125f;
    const uint32_t idx = ldb(b + 2 + 4 * ib + l) | (((qh >> (3 * l)) & 7) << 8);
    delta_grid8(grid8(tab, TAB_IQ1, idx), delta, dl, o);
  }
};
template <> struct Dec<QT_IQ1_M> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const uint2 sw = ld8<8>(b + 48);                    // four u16: 3-bit scales, and a nibble of the super-scale each
    const uint32_t dbits = ((sw.x >> 12) & 0x000F) | ((sw.x >> 24) & 0x00F0) | ((sw.y >> 4) & 0x0F00) | ((sw.y >> 16) & 0xF000);
    const float d = h2f(dbits);
    const uint32_t w = (g >> 4 ? sw.y : sw.x) >> (16 * ((g >> 3) & 1));
    const uint32_t s = (w >> (3 * ((g >> 1) & 3))) & 7;
    const float dl = __fmul_rn(d, i2f(2 * s + 1));
    const uint32_t n = (ldb(b + 32 + (g >> 1)) >> (4 * (g & 1))) & 15;
    const uint32_t idx = ldb(b + g) | ((n & 7) << 8);
    delta_grid8(grid8(tab, TAB_IQ1, idx), (n & 8) ? -0.125f : 0.125f, dl, o);
  }
};
template <> struct Dec<QT_IQ4_XS> {
  __device__ static void run(const uint8_t* b, int g, const uint8_t* tab, float* o) {
    const uint4 kv = table16(tab, TAB_KV_IQ4);
    const uint2 h = ld8<8>(b);                          // d | high scale bits, low scale nibbles
    const float d = h2f(h.x & 0xFFFF);
    const int j = g >> 2;
    const int sc = (int)(((h.y >> (4 * j)) & 15) | (((h.x >> (16 + 2 * j)) & 3) << 4)) - 32;
    const float dl = __fmul_rn(d, i2f(sc));
    const uint2 q = ld8<8>(b + 8 + 16 * j + 8 * (g & 1));
    const int hi = (g >> 1) & 1;
    codes8(lookup_bytes(kv, nibbles(q.x, hi)), lookup_bytes(kv, nibbles(q.y, hi)), 128.f, o);
    mul8(o, dl);
  }
};

// Calls f.template operator()<QT>() for the block qtype `qtype`; returns false for the
// float passthrough types and unknown codes.
template <class F>
inline bool dispatch_block_qtype(int qtype, F&& f) {
  switch (qtype) {
#define GGQ_CASE(T) case T: f.template operator()<T>(); return true;
    GGQ_CASE(QT_Q4_0) GGQ_CASE(QT_Q4_1) GGQ_CASE(QT_Q5_0) GGQ_CASE(QT_Q5_1) GGQ_CASE(QT_Q8_0)
    GGQ_CASE(QT_Q2_K) GGQ_CASE(QT_Q3_K) GGQ_CASE(QT_Q4_K) GGQ_CASE(QT_Q5_K) GGQ_CASE(QT_Q6_K)
    GGQ_CASE(QT_IQ2_XXS) GGQ_CASE(QT_IQ2_XS) GGQ_CASE(QT_IQ3_XXS) GGQ_CASE(QT_IQ1_S)
    GGQ_CASE(QT_IQ4_NL) GGQ_CASE(QT_IQ3_S) GGQ_CASE(QT_IQ2_S) GGQ_CASE(QT_IQ4_XS)
    GGQ_CASE(QT_IQ1_M) GGQ_CASE(QT_TQ1_0) GGQ_CASE(QT_TQ2_0) GGQ_CASE(QT_MXFP4) GGQ_CASE(QT_NVFP4)
#undef GGQ_CASE
    default: return false;
  }
}

}  // inline namespace
}  // namespace ggq
