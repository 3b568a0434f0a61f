// fi_cluster_rk4.cu — cluster kernels of RK4, up to four rows a thread (fi_cluster.cuh).
#include "fi_cluster.cuh"

namespace fi {
template cudaError_t cluster_go<CLU_RK4, 256, 2>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
template cudaError_t cluster_go<CLU_RK4, 512, 4>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
}  // namespace fi
