// fi_tableau.cuh — coefficients of the integrators, for every kernel that steps
// a domain (a translation unit has its own copy).
#pragma once

namespace fi {

// RK4: y_s = x + a_s h k_{s-1}
static __constant__ double c_rk4_a[4] = {0.0, 0.5, 0.5, 1.0};

// Tsitouras 5(4), reference-compatible (tsit54, src/integrators.f90): weights of
// the two solutions
static __constant__ double c_ts_b[6] = {0.0845, 0.0, 0.0, 0.5179, 0.1276, 0.2700};
static __constant__ double c_ts_bh[6] = {0.0845, 0.0, 0.0, 0.5179, 0.1276, 0.2700 - 1 / 5.0};

// the Dormand-Prince 5(4) pair: stages, and weights of the embedded solution
static __constant__ double c_dp_a[7][6] = {
    {0, 0, 0, 0, 0, 0},
    {1.0 / 5, 0, 0, 0, 0, 0},
    {3.0 / 40, 9.0 / 40, 0, 0, 0, 0},
    {44.0 / 45, -56.0 / 15, 32.0 / 9, 0, 0, 0},
    {19372.0 / 6561, -25360.0 / 2187, 64448.0 / 6561, -212.0 / 729, 0, 0},
    {9017.0 / 3168, -355.0 / 33, 46732.0 / 5247, 49.0 / 176, -5103.0 / 18656, 0},
    {35.0 / 384, 0, 500.0 / 1113, 125.0 / 192, -2187.0 / 6784, 11.0 / 84}};
static __constant__ double c_dp_bs[7] = {5179.0 / 57600, 0, 7571.0 / 16695, 393.0 / 640, -92097.0 / 339200,
                                         187.0 / 2100, 1.0 / 40};

}  // namespace fi
