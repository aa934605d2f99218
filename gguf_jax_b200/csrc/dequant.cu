// Block-decode kernels: quantized bytes -> float32 / bfloat16 / float16.
//
// HBM-bound on the WRITE side (a Q4_K block is 144 bytes in, 1024 bytes of float32 out),
// so the mapping is chosen for the stores: one thread produces sixteen consecutive output
// elements and writes them as one (bf16/f16) or two (f32) 32-byte stores, a whole memory sector each;
// consecutive threads own consecutive groups, so a warp writes 1 / 2 KiB contiguous.  The block
// bytes come through the read-only path and are reused by the threads of a superblock out of L1; what the two
// octets of a thread share (scales, header words) is unpacked once.
// The kernel is a programmatic dependent of the launch before it, which hides its launch (decode + GEMM of seven weights of 3 to 48 MB at 32
// rows: 191 -> 183 us).
//
// Measured on B200, 14336 x 4096, us to bf16 / float32, eight weights per thread with byte-wise decoders before -> here:
// Q4_K 41 / 56 -> 27 / 43 (5.7 / 6.2 TB/s read and written), Q5_K 51 / 56 -> 29 / 45, Q2_K 42 / 70 -> 25 / 42, IQ2_XS 59 / 72 ->
// 27 / 43, IQ1_S 73 / 83 -> 25 / 41, MXFP4 41 / 65 -> 29 / 43, TQ1_0 101 / 103 -> 28 / 45; instructions, not memory, were the bound.
// The 2-byte aligned formats read their codes as aligned words (four 2-byte loads per octet: Q6_K 39, Q8_0 34, Q3_K 36 us;
// two or three words: 33, 31, 31; before all of this 46, 34, 55).
#include "gemv.cuh"
#include "ggq_decode.cuh"

namespace ggq {

template <int OUT> struct OutT;
template <> struct OutT<GGQ_F32> { using type = float; };
template <> struct OutT<GGQ_BF16> { using type = __nv_bfloat16; };
template <> struct OutT<GGQ_F16> { using type = __half; };

// 32 bytes at p (16-byte aligned): one store when p is 32-byte aligned, which `wide` says for the whole launch.
__device__ __forceinline__ void store32(uint8_t* p, const uint32_t (&u)[8], bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]) : "memory");
  } else {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(u[0], u[1], u[2], u[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(u[4], u[5], u[6], u[7]);
  }
}
// Elements 16 group .. + 15 of the output.
template <int OUT>
__device__ __forceinline__ void store16(void* out, int64_t group, const float (&v)[16], bool wide) {
  uint32_t u[8];
  if constexpr (OUT == GGQ_F32) {
    uint8_t* p = reinterpret_cast<uint8_t*>(out) + 64 * group;
#pragma unroll
    for (int h = 0; h < 2; h++) {
#pragma unroll
      for (int i = 0; i < 8; i++) u[i] = __float_as_uint(v[8 * h + i]);
      store32(p + 32 * h, u, wide);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if constexpr (OUT == GGQ_BF16) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        u[i] = *reinterpret_cast<const uint32_t*>(&a);
      } else {
        const __half2 a = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
        u[i] = *reinterpret_cast<const uint32_t*>(&a);
      }
    }
    store32(reinterpret_cast<uint8_t*>(out) + 32 * group, u, wide);
  }
}

template <int QT, int BS, int TS, int OUT>
__global__ void __launch_bounds__(256)
dequant_kernel(const uint8_t* __restrict__ blocks, int64_t n_groups, void* __restrict__ out,
               const uint8_t* __restrict__ tab, const bool wide) {
  pdl_wait();                   // the launch before this one may still be reading what is about to be written
  constexpr int GPB = BS / 16;  // groups of 16 elements per block
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= n_groups) return;
  const int64_t blk = gid / GPB;
  const int g = (int)(gid - blk * GPB);
  float v[16];
  Dec<QT>::run(blocks + blk * TS, 2 * g, tab, v);
  Dec<QT>::run(blocks + blk * TS, 2 * g + 1, tab, v + 8);
  store16<OUT>(out, gid, v, wide);
  pdl_trigger();
}

// F32 / F16 / BF16 "qtypes": widen (or copy) element-wise, bit-exact
// (src/gguf_jax/quants.py:125-138).
template <int QT, int OUT>
__global__ void __launch_bounds__(256)
passthrough_kernel(const uint8_t* __restrict__ in, int64_t n, void* __restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float v;
  if constexpr (QT == QT_F32) v = __uint_as_float(ld32(in + 4 * i));
  else if constexpr (QT == QT_F16) v = h2f(ld16(in + 2 * i));
  else v = __uint_as_float(ld16(in + 2 * i) << 16);
  if constexpr (OUT == GGQ_F32) reinterpret_cast<float*>(out)[i] = v;
  else if constexpr (OUT == GGQ_BF16) reinterpret_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(v);
  else reinterpret_cast<__half*>(out)[i] = __float2half_rn(v);
}

template <int QT, int OUT>
static cudaError_t launch_block(const TypeInfo* ti, const uint8_t* blocks, int64_t n_blocks, void* out,
                                const uint8_t* tab, cudaStream_t st) {
  constexpr int BS = block_elems_of(QT), TS = block_bytes_of(QT);
  if (ti->block_elems != BS || ti->block_bytes != TS) return cudaErrorInvalidValue;
  int64_t n_groups = n_blocks * (BS / 16);
  if (n_groups == 0) return cudaSuccess;
  int64_t grid = (n_groups + 255) / 256;
  const cudaError_t err = launch_pdl(dequant_kernel<QT, BS, TS, OUT>, (int)grid, 256, 0, st, blocks, n_groups, out, tab, (uintptr_t)out % 32 == 0);
  return err != cudaSuccess ? err : cudaPeekAtLastError();
}

template <int OUT>
static cudaError_t launch_out(const TypeInfo* ti, const uint8_t* blocks, int64_t n_blocks, void* out,
                              const uint8_t* tab, cudaStream_t st) {
  int qt = ti->qtype;
  if (qt == QT_F32 || qt == QT_F16 || qt == QT_BF16) {
    if (n_blocks == 0) return cudaSuccess;
    unsigned grid = (unsigned)((n_blocks + 255) / 256);
    if (qt == QT_F32) passthrough_kernel<QT_F32, OUT><<<grid, 256, 0, st>>>(blocks, n_blocks, out);
    else if (qt == QT_F16) passthrough_kernel<QT_F16, OUT><<<grid, 256, 0, st>>>(blocks, n_blocks, out);
    else passthrough_kernel<QT_BF16, OUT><<<grid, 256, 0, st>>>(blocks, n_blocks, out);
    return cudaPeekAtLastError();
  }
  cudaError_t err = cudaErrorInvalidValue;
  dispatch_block_qtype(qt, [&]<int QT>() { err = launch_block<QT, OUT>(ti, blocks, n_blocks, out, tab, st); });
  return err;
}

}  // namespace ggq

extern "C" int32_t ggq_dequant(int32_t qtype, const void* blocks, int64_t n_blocks, void* out,
                               int32_t out_dtype, void* stream) {
  using namespace ggq;
  const TypeInfo* ti = type_info(qtype);
  if (!ti) return fail(GGQ_BAD_QTYPE, "ggq_dequant: qtype %d is not decodable", qtype);
  if (n_blocks < 0) return fail(GGQ_BAD_SHAPE, "ggq_dequant: n_blocks %lld < 0", (long long)n_blocks);
  if (n_blocks * (int64_t)(ti->block_elems >= 8 ? ti->block_elems / 8 : 1) > (int64_t)0x7FFFFFFF * 256)
    return fail(GGQ_BAD_SHAPE, "ggq_dequant: %lld blocks exceed one launch", (long long)n_blocks);
  if (n_blocks == 0) return GGQ_OK;
  if (!blocks || !out) return fail(GGQ_MISALIGNED, "ggq_dequant: null pointer");
  if ((uintptr_t)out % 16) return fail(GGQ_MISALIGNED, "ggq_dequant: out must be 16-byte aligned");
  if ((uintptr_t)blocks % block_alignment(ti))
    return fail(GGQ_MISALIGNED, "ggq_dequant: blocks must be %d-byte aligned for qtype %d", block_alignment(ti), qtype);
  int dev = 0;
  cudaGetDevice(&dev);
  const uint8_t* tab = device_tables(dev);
  if (ti->needs_tables && !tab)
    return fail(GGQ_NO_TABLES, "ggq_dequant: call ggq_set_tables(%d, ...) before decoding qtype %d", dev, qtype);
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t err;
  switch (out_dtype) {
    case GGQ_F32: err = launch_out<GGQ_F32>(ti, (const uint8_t*)blocks, n_blocks, out, tab, st); break;
    case GGQ_BF16: err = launch_out<GGQ_BF16>(ti, (const uint8_t*)blocks, n_blocks, out, tab, st); break;
    case GGQ_F16: err = launch_out<GGQ_F16>(ti, (const uint8_t*)blocks, n_blocks, out, tab, st); break;
    default: return fail(GGQ_BAD_DTYPE, "ggq_dequant: out_dtype %d", out_dtype);
  }
  if (err != cudaSuccess) return fail(GGQ_LAUNCH_FAILED, "ggq_dequant: %s", cudaGetErrorString(err));
  return GGQ_OK;
}
