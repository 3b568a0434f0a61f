// fi_cluster_ts.cu — cluster kernels of reference-compatible tsit54, up to four rows a thread (fi_cluster.cuh).
#include "fi_cluster.cuh"

namespace fi {
template cudaError_t cluster_go<CLU_TSIT, 256, 2>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
template cudaError_t cluster_go<CLU_TSIT, 512, 4>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
}  // namespace fi
