// Instantiations of the batch kernel (gemv_batch.cuh): the IQ formats with one scale per 256 weights.
#include "gemv_batch.cuh"

namespace ggq {
namespace batch {

cudaError_t launch_iq(int qtype, const Args& a) {
  switch (qtype) {
    case QT_IQ4_XS: return launch_tiles<bf::IQ4XS>(a);
    case QT_IQ2_XXS: return launch_tiles<bf::IQ2XXS>(a);
    case QT_IQ2_XS: return launch_tiles<bf::IQ2XS>(a);
    case QT_IQ2_S: return launch_tiles<bf::IQ2S>(a);
    case QT_IQ3_XXS: return launch_tiles<bf::IQ3XXS>(a);
    case QT_IQ3_S: return launch_tiles<bf::IQ3S>(a);
    case QT_IQ1_S: return launch_tiles<bf::IQ1S>(a);
    case QT_IQ1_M: return launch_tiles<bf::IQ1M>(a);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace batch
}  // namespace ggq
