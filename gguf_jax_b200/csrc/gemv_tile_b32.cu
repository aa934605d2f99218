// Instantiations of the tiled fused multiply (gemv_tile.cuh): the formats with blocks of 32 or 64 weights.
#include "gemv_tile.cuh"

namespace ggq {
namespace tile {

cudaError_t launch_b32(int qtype, const Args& a) {
  switch (qtype) {
    case QT_Q8_0: return launch_args<tf::Q80>(a);
    case QT_Q4_0: return launch_args<tf::Q40>(a);
    case QT_Q4_1: return launch_args<tf::Q41>(a);
    case QT_Q5_0: return launch_args<tf::Q50>(a);
    case QT_Q5_1: return launch_args<tf::Q51>(a);
    case QT_IQ4_NL: return launch_args<tf::IQ4NL>(a);
    case QT_MXFP4: return launch_args<tf::MXFP4>(a);
    case QT_NVFP4: return launch_args<tf::NVFP4>(a);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace tile
}  // namespace ggq
