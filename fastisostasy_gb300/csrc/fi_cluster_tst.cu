// fi_cluster_tst.cu — cluster kernels of true-stage tsit54, up to four rows a thread (fi_cluster.cuh).
#include "fi_cluster.cuh"

namespace fi {
template cudaError_t cluster_go<CLU_TSIT_TRUE, 256, 2>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
template cudaError_t cluster_go<CLU_TSIT_TRUE, 512, 4>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
}  // namespace fi
