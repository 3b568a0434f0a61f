// fi_cluster_rk4_8.cu — cluster kernels of RK4, up to eight rows a thread (fi_cluster.cuh).
#include "fi_cluster.cuh"

namespace fi {
template cudaError_t cluster_go<CLU_RK4, 512, 8>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
}  // namespace fi
