// fi_cluster.h — small mixed domains advanced by one thread-block cluster each
// (fi_cluster.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fi_common.cuh"
#include "fi_kernels.h"

namespace fi {

enum { CLU_RK4 = 0, CLU_TSIT = 1, CLU_TSIT_TRUE = 2 };

struct ClusterArgs {
    Plan2D p;
    FlexCoefF fcf;
    double* x;                       // integrator state
    double* w;                       // now%w
    const float* wrhi;               // w_ref as a float pair (true stages)
    const float* wrlo;
    const float* q0;                 // load term
    const float* D;
    const float* inv2eta;
    const float* mAT;                // 1/(kappa R) factors, column-major (k*ny + l)
    const float* mBT;
    int even;
    const uint8_t* mask;
    float* raw[7];                   // stage outputs; the last one evaluated is left in raw[0] (raw[3] in RK4)
    Ctl* ctl;
    int nsteps;                      // RK4: steps of this update
    int rpc, cpc;                    // rows and spectrum columns per block
    double spy, atol, rtol, q, dt_max;
    int max_iter;                    // adaptive: attempts per update
    int stages;                      // stage outputs kept in shared memory
    float norm_scale_f;
};

// Blocks per cluster, threads, stage outputs kept in shared memory (true-stage
// tsit54) and its size for a domain of this plan;
// 0 where it does not fit (then the other paths take it).
int cluster_config(const Plan2D& p, int mode, int* nc, int* threads, int* stages, size_t* smem);
void cluster_split(ClusterArgs& a, int nc);
// probe: no launch, only whether such a cluster can be resident
cudaError_t cluster_launch(const ClusterArgs& a, int mode, int nc, int threads, size_t smem, cudaStream_t s,
                           bool probe = false);

}  // namespace fi
