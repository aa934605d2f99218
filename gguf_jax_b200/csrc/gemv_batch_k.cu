// Instantiations of the batch kernel (gemv_batch.cuh): the K-quants and the ternary formats.
#include "gemv_batch.cuh"

namespace ggq {
namespace batch {

int max_clusters(int Q) {
  const auto kernel = gemv_batch_kernel<bf::Q4K, 1>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)Q);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = 128 << 10;        // one CTA per SM, like every launch
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)Q;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tile::kSmemLimit) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

cudaError_t launch_k(int qtype, const Args& a) {
  switch (qtype) {
    case QT_Q2_K: return launch_tiles<bf::Q2K>(a);
    case QT_Q3_K: return launch_tiles<bf::Q3K>(a);
    case QT_Q4_K: return launch_tiles<bf::Q4K>(a);
    case QT_Q5_K: return launch_tiles<bf::Q5K>(a);
    case QT_Q6_K: return launch_tiles<bf::Q6K>(a);
    case QT_TQ1_0: return launch_tiles<bf::TQ10>(a);
    case QT_TQ2_0: return launch_tiles<bf::TQ20>(a);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace batch
}  // namespace ggq
