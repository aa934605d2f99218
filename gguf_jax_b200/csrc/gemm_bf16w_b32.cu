// Fused decode + GEMM with bf16 weights: the formats of 32 and 64 weights a block.
#include "gemm_bf16w_generic.cuh"

namespace ggq {
namespace gemmb {

cudaError_t launch_b32(int qtype, const Call& c) {
  switch (qtype) {
    case QT_Q4_0: return launch_generic<QT_Q4_0>(c);
    case QT_Q4_1: return launch_generic<QT_Q4_1>(c);
    case QT_Q5_0: return launch_generic<QT_Q5_0>(c);
    case QT_Q5_1: return launch_generic<QT_Q5_1>(c);
    case QT_Q8_0: return launch_generic<QT_Q8_0>(c);
    case QT_IQ4_NL: return launch_generic<QT_IQ4_NL>(c);
    case QT_MXFP4: return launch_generic<QT_MXFP4>(c);
    case QT_NVFP4: return launch_generic<QT_NVFP4>(c);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gemmb
}  // namespace ggq
