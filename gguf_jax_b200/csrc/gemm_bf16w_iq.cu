// Fused decode + GEMM with bf16 weights: the low-bit formats of 256 weights a block.
#include "gemm_bf16w_generic.cuh"

namespace ggq {
namespace gemmb {

cudaError_t launch_iq(int qtype, const Call& c) {
  switch (qtype) {
    case QT_Q6_K: return launch_generic<QT_Q6_K>(c);          // rows off 16 bytes
    case QT_Q2_K: return launch_generic<QT_Q2_K>(c);
    case QT_Q3_K: return launch_generic<QT_Q3_K>(c);
    case QT_IQ4_XS: return launch_generic<QT_IQ4_XS>(c);
    case QT_IQ2_XXS: return launch_generic<QT_IQ2_XXS>(c);
    case QT_IQ2_XS: return launch_generic<QT_IQ2_XS>(c);
    case QT_IQ2_S: return launch_generic<QT_IQ2_S>(c);
    case QT_IQ3_XXS: return launch_generic<QT_IQ3_XXS>(c);
    case QT_IQ3_S: return launch_generic<QT_IQ3_S>(c);
    case QT_IQ1_S: return launch_generic<QT_IQ1_S>(c);
    case QT_IQ1_M: return launch_generic<QT_IQ1_M>(c);
    case QT_TQ1_0: return launch_generic<QT_TQ1_0>(c);
    case QT_TQ2_0: return launch_generic<QT_TQ2_0>(c);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gemmb
}  // namespace ggq
