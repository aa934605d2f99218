// Instantiations of the tiled fused multiply (gemv_tile.cuh): the IQ formats with 256-weight blocks.
#include "gemv_tile.cuh"

namespace ggq {
namespace tile {

cudaError_t launch_iq(int qtype, const Args& a) {
  switch (qtype) {
    case QT_IQ4_XS: return launch_args<tf::IQ4XS>(a);
    case QT_IQ2_XS: return launch_args<tf::IQ2XS>(a);
    case QT_IQ2_S: return launch_args<tf::IQ2S>(a);
    case QT_IQ3_XXS: return launch_args<tf::IQ3XXS>(a);
    case QT_IQ3_S: return launch_args<tf::IQ3S>(a);
    case QT_IQ1_S: return launch_args<tf::IQ1S>(a);
    case QT_IQ1_M: return launch_args<tf::IQ1M>(a);
    case QT_IQ2_XXS: return launch_args<tf::IQ2XXS>(a);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace tile
}  // namespace ggq
