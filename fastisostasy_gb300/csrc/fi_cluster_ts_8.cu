// fi_cluster_ts_8.cu — cluster kernels of reference-compatible tsit54, up to eight rows a thread (fi_cluster.cuh).
#include "fi_cluster.cuh"

namespace fi {
template cudaError_t cluster_go<CLU_TSIT, 512, 8>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
}  // namespace fi
