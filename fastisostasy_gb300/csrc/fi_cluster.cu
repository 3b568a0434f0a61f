// fi_cluster.cu — which domains run in a cluster (fi_cluster.cuh).  The kernels
// are in translation units of their own (fi_cluster_*.cu): together they
// compile for minutes.
#include "fi_cluster.cuh"

namespace fi {

extern template cudaError_t cluster_go<CLU_RK4, 256, 2>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
extern template cudaError_t cluster_go<CLU_RK4, 512, 4>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
extern template cudaError_t cluster_go<CLU_RK4, 512, 8>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
extern template cudaError_t cluster_go<CLU_TSIT, 256, 2>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
extern template cudaError_t cluster_go<CLU_TSIT, 512, 4>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
extern template cudaError_t cluster_go<CLU_TSIT, 512, 8>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
extern template cudaError_t cluster_go<CLU_TSIT_TRUE, 256, 2>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
extern template cudaError_t cluster_go<CLU_TSIT_TRUE, 512, 4>(const ClusterArgs&, int, size_t, cudaStream_t, bool);
extern template cudaError_t cluster_go<CLU_TSIT_TRUE, 512, 8>(const ClusterArgs&, int, size_t, cudaStream_t, bool);

template <int MODE>
static cudaError_t cluster_any(const ClusterArgs& a, int nc, int threads, int run, size_t smem, cudaStream_t s,
                               bool probe)
{
    if (threads == 256) return cluster_go<MODE, 256, 2>(a, nc, smem, s, probe);
    return run <= 4 ? cluster_go<MODE, 512, 4>(a, nc, smem, s, probe) : cluster_go<MODE, 512, 8>(a, nc, smem, s, probe);
}


int cluster_config(const Plan2D& p, int mode, int* nc, int* threads, int* stages, size_t* smem)
{
    if (p.nx < 16 || p.ny < 16) return 0;
    // A length without a register line takes the shared-memory stages, on 8 or
    // 16 multiprocessors: faster than the grid-wide engine on the smallest
    // domains (an RK4 update of ten steps: 34^2 371 against 584 us, 50^2 379
    // against 549).  The line was drawn with direct sums for the odd radices
    // (80^2 567 against 608 alone, 3 % slower in a served mix; 100^2 721
    // against 711, 122 = 2 61 1368 against 892); with the present stages the
    // cluster leads above it as well (80^2 436 against 563, 100^2 469 against
    // 598, 122^2 651 against 713), which a served mix has not been timed for.
    if ((!CluLay::line_ok(p.h) || !CluLay::line_ok(p.ny)) && p.nx * p.ny > 4096) return 0;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    for (int n : {8, 16}) {
        const int rpc = clu_rpc(p.ny, n), cpc = clu_cpc(p.h, n);
        if (n == 8 && rpc * p.nx > 1024) continue;   // more cells than two a thread: spread over 16 blocks
        auto bytes = [&](int k) { return (size_t)CluLay(p.nx, p.h, p.ny, rpc, cpc, k).total * sizeof(float) + 2048; };
        if (bytes(0) > (size_t)optin) continue;   // (2 KB: the static shared state)
        *stages = mode == CLU_TSIT_TRUE && bytes(7) <= (size_t)optin ? 7 : 0;
        const size_t b = bytes(*stages) - 2048;
        *nc = n;
        // 256 threads where they own two rows at most: two such blocks fit a
        // multiprocessor
        *threads = p.nx <= 256 && clu_run(p.nx, rpc, 256) <= 2 ? 256 : 512;
        if (p.nx > *threads || clu_run(p.nx, rpc, *threads) > 8) continue;
        *smem = b;
        ClusterArgs a;
        memset(&a, 0, sizeof(a));
        a.p = p;
        if (cluster_launch(a, mode, n, *threads, *smem, nullptr, true) == cudaSuccess) return 1;
    }
    return 0;
}

void cluster_split(ClusterArgs& a, int nc)
{
    a.rpc = clu_rpc(a.p.ny, nc);
    a.cpc = clu_cpc(a.p.h, nc);
}

cudaError_t cluster_launch(const ClusterArgs& a, int mode, int nc, int threads, size_t smem, cudaStream_t s, bool probe)
{
    const int run = clu_run(a.p.nx, clu_rpc(a.p.ny, nc), threads);
    switch (mode) {
    case CLU_RK4: return cluster_any<CLU_RK4>(a, nc, threads, run, smem, s, probe);
    case CLU_TSIT: return cluster_any<CLU_TSIT>(a, nc, threads, run, smem, s, probe);
    default: return cluster_any<CLU_TSIT_TRUE>(a, nc, threads, run, smem, s, probe);
    }
}

}  // namespace fi
