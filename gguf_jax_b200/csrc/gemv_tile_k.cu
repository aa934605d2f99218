// Instantiations of the tiled fused multiply (gemv_tile.cuh): the K-quants and the ternary formats.
#include "gemv_tile.cuh"

namespace ggq {
namespace tile {

cudaError_t launch_k(int qtype, const Args& a) {
  switch (qtype) {
    case QT_Q4_K: return launch_args<tf::Q4K>(a);
    case QT_Q5_K: return launch_args<tf::Q5K>(a);
    case QT_Q6_K: return launch_args<tf::Q6K>(a);
    case QT_Q2_K: return launch_args<tf::Q2K>(a);
    case QT_Q3_K: return launch_args<tf::Q3K>(a);
    case QT_TQ1_0: return launch_args<tf::TQ10>(a);
    case QT_TQ2_0: return launch_args<tf::TQ20>(a);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace tile
}  // namespace ggq
