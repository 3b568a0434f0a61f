// fi_rhs.cu — the LV-ELVA viscous-rate pipeline and the FFT convolution
// passes (calc_lvelva, src/lv_elva.f90:31-126; precomputed_fftconvolution,
// src/convolutions.f90:59-91).
//
// RHS = four kernels:
//   k_flexure*     finite-difference flexure moments and load -> f (one pass over the grid)
//   rows_fwd       real FFT of every row of f -> half spectrum S
//   cols_hartley   column FFT, multiply by 1/(kappa R) in the Hartley basis, inverse column FFT
//   rows_inv       inverse real FFT of the rows, scaled by 1/(nx*ny) -> raw
// The transforms of lengths that have a register line are in fi_lines*.cu;
// the shared-memory forms here take every other length.
// The corner boundary condition and the sec_per_year factor are applied by
// whichever kernel consumes raw (it reads the four corner values).
//
// The reference transforms with FFTW's separable DHT.  The Hartley
// coefficients are formed from the DFT in the column kernel,
//   H[k,l] = Re F[k,-l] - Im F[k,l],
// multiplied by m = 1/(kappa R) at all four (+-k, +-l), and turned back into
// the DFT of DHT^-1(m H); when m is even in both indices this reduces to
// F' = m F (flag `even`).
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "fi_fft.cuh"

#include "fi_batch.h"
#include "fi_kernels.h"
#include "fi_lines.cuh"

namespace fi {

template <typename T> __device__ __forceinline__ const typename vec2<T>::type* twp(const FftLen& L);
template <> __device__ __forceinline__ const double2* twp<double>(const FftLen& L) { return L.tw64; }
template <> __device__ __forceinline__ const float2* twp<float>(const FftLen& L) { return L.tw32; }
template <typename T> __device__ __forceinline__ const typename vec2<T>::type* rtwp(const Plan2D& p);
template <> __device__ __forceinline__ const double2* rtwp<double>(const Plan2D& p) { return p.rtw64; }
template <> __device__ __forceinline__ const float2* rtwp<float>(const Plan2D& p) { return p.rtw32; }

// Raise a kernel's dynamic shared-memory limit when a larger launch needs it
// (the limit belongs to the kernel and is shared by every handle, so it only
// ever grows).
template <typename K> static void set_smem(K kern, size_t bytes)
{
    static std::mutex mu;
    static const void* fn[64];
    static size_t done[64];
    static int nfn = 0;
    if (bytes <= 48 * 1024) return;
    std::lock_guard<std::mutex> lk(mu);
    const void* key = (const void*)kern;
    for (int i = 0; i < nfn; ++i)
        if (fn[i] == key) {
            if (done[i] >= bytes) return;
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            done[i] = bytes;
            return;
        }
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (nfn < 64) { fn[nfn] = key; done[nfn] = bytes; ++nfn; }
}

// ---------------------------------------------------------------------------
// Flexure stencil of the mixed form on a distorted grid (1/(dx K), 1/(dy K) per
// cell).  Tile TX x TY outputs with a halo of 2; the first-level differences
// are taken on the double state, then rounded to float.
// ---------------------------------------------------------------------------
constexpr int TX = 32, TY = 8, RX = TX + 4, RY = TY + 4;

__global__ void __launch_bounds__(TX* TY)
k_flexure(const double* __restrict__ y, const double* __restrict__ wref, const float* __restrict__ q0,
          const uint8_t* __restrict__ mask, const float* __restrict__ D, const float* __restrict__ inv2eta,
          float* __restrict__ f, int nx, int ny, FlexCoef c, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    typedef float T;
    __shared__ double ys[RY][RX];
    __shared__ T wx[RY][RX];
    __shared__ T Mxx[RY][RX];
    __shared__ T Myy[RY][RX];
    __shared__ T Mxy[RY][RX];
    __shared__ T Mxyx[RY][RX];
    const int tid = threadIdx.x + TX * threadIdx.y;
    const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;

    // per-cell spacings: 1/(2 d) and 1/d^2 from the stored 1/d (an FP64
    // division is a chain of a dozen FP64 instructions, and a cell took eight)
    auto idx1 = [&](int i, int j) -> double { return c.ixm[(size_t)j * nx + i]; };
    auto idx2h = [&](int i, int j) -> double { return 0.5 * c.ixm[(size_t)j * nx + i]; };
    auto idxx = [&](int i, int j) -> double {
        const double d = c.ixm[(size_t)j * nx + i];
        return d * d;
    };
    auto idy1 = [&](int i, int j) -> double { return c.iym[(size_t)j * nx + i]; };
    auto idy2h = [&](int i, int j) -> double { return 0.5 * c.iym[(size_t)j * nx + i]; };
    auto idyy = [&](int i, int j) -> double {
        const double d = c.iym[(size_t)j * nx + i];
        return d * d;
    };

    for (int e = tid; e < RX * RY; e += TX * TY) {
        const int lx = e % RX, ly = e / RX;
        const int gi = i0 - 2 + lx, gj = j0 - 2 + ly;
        ys[ly][lx] = (gi >= 0 && gi < nx && gj >= 0 && gj < ny) ? y[(size_t)gj * nx + gi] : 0.0;
    }
    __syncthreads();
    // w_x on lx in [1, RX-1), all rows
    for (int e = tid; e < RX * RY; e += TX * TY) {
        const int lx = e % RX, ly = e / RX;
        const int gi = i0 - 2 + lx, gj = j0 - 2 + ly;
        if (lx < 1 || lx >= RX - 1 || gi < 0 || gi >= nx || gj < 0 || gj >= ny) continue;
        double v;
        if (gi == 0) v = (ys[ly][lx + 1] - ys[ly][lx]) * idx1(gi, gj);
        else if (gi == nx - 1) v = (ys[ly][lx] - ys[ly][lx - 1]) * idx1(gi, gj);
        else v = (ys[ly][lx + 1] - ys[ly][lx - 1]) * idx2h(gi, gj);
        wx[ly][lx] = (T)v;
    }
    __syncthreads();
    // level 1: w_xy, w_xx, w_yy -> moments, on lx, ly in [1, R-1)
    for (int e = tid; e < RX * RY; e += TX * TY) {
        const int lx = e % RX, ly = e / RX;
        const int gi = i0 - 2 + lx, gj = j0 - 2 + ly;
        if (lx < 1 || lx >= RX - 1 || ly < 1 || ly >= RY - 1 || gi < 0 || gi >= nx || gj < 0 || gj >= ny) continue;
        T wxy;
        if (gj == 0) wxy = (wx[ly + 1][lx] - wx[ly][lx]) * (T)idy1(gi, gj);
        else if (gj == ny - 1) wxy = (wx[ly][lx] - wx[ly - 1][lx]) * (T)idy1(gi, gj);
        else wxy = (wx[ly + 1][lx] - wx[ly - 1][lx]) * (T)idy2h(gi, gj);
        double dxx, dyy;
        if (gi == 0) dxx = ((ys[ly][lx + 2] - 2 * ys[ly][lx + 1]) + ys[ly][lx]) * idxx(0, gj);
        else if (gi == nx - 1) dxx = ((ys[ly][lx] - 2 * ys[ly][lx - 1]) + ys[ly][lx - 2]) * idxx(0, gj);
        else dxx = ((ys[ly][lx + 1] - 2 * ys[ly][lx]) + ys[ly][lx - 1]) * idxx(gi, gj);
        if (gj == 0) dyy = ((ys[ly + 2][lx] - 2 * ys[ly + 1][lx]) + ys[ly][lx]) * idyy(gi, 0);
        else if (gj == ny - 1) dyy = ((ys[ly][lx] - 2 * ys[ly - 1][lx]) + ys[ly - 2][lx]) * idyy(gi, gj);
        else dyy = ((ys[ly + 1][lx] - 2 * ys[ly][lx]) + ys[ly - 1][lx]) * idyy(gi, gj);
        const T wxx = (T)dxx, wyy = (T)dyy;
        const T Dl = D[(size_t)gj * nx + gi];
        const T nu = (T)c.nu;
        Mxx[ly][lx] = -Dl * (wxx + nu * wyy);
        Myy[ly][lx] = -Dl * (wyy + nu * wxx);
        Mxy[ly][lx] = (-Dl * (T)c.one_minus_nu) * wxy;
    }
    __syncthreads();
    // d/dx of Mxy on lx in [2, RX-2), ly in [1, RY-1)
    for (int e = tid; e < RX * RY; e += TX * TY) {
        const int lx = e % RX, ly = e / RX;
        const int gi = i0 - 2 + lx, gj = j0 - 2 + ly;
        if (lx < 2 || lx >= RX - 2 || ly < 1 || ly >= RY - 1 || gi < 0 || gi >= nx || gj < 0 || gj >= ny) continue;
        T v;
        if (gi == 0) v = (Mxy[ly][lx + 1] - Mxy[ly][lx]) * (T)idx1(gi, gj);
        else if (gi == nx - 1) v = (Mxy[ly][lx] - Mxy[ly][lx - 1]) * (T)idx1(gi, gj);
        else v = (Mxy[ly][lx + 1] - Mxy[ly][lx - 1]) * (T)idx2h(gi, gj);
        Mxyx[ly][lx] = v;
    }
    __syncthreads();
    {
        const int lx = threadIdx.x + 2, ly = threadIdx.y + 2;
        const int gi = i0 + threadIdx.x, gj = j0 + threadIdx.y;
        if (gi < nx && gj < ny) {
            T mxy_xy, mx_xx, my_yy;
            if (gj == 0) mxy_xy = (Mxyx[ly + 1][lx] - Mxyx[ly][lx]) * (T)idy1(gi, gj);
            else if (gj == ny - 1) mxy_xy = (Mxyx[ly][lx] - Mxyx[ly - 1][lx]) * (T)idy1(gi, gj);
            else mxy_xy = (Mxyx[ly + 1][lx] - Mxyx[ly - 1][lx]) * (T)idy2h(gi, gj);
            if (gi == 0) mx_xx = ((Mxx[ly][lx + 2] - (T)2 * Mxx[ly][lx + 1]) + Mxx[ly][lx]) * (T)idxx(0, gj);
            else if (gi == nx - 1) mx_xx = ((Mxx[ly][lx] - (T)2 * Mxx[ly][lx - 1]) + Mxx[ly][lx - 2]) * (T)idxx(0, gj);
            else mx_xx = ((Mxx[ly][lx + 1] - (T)2 * Mxx[ly][lx]) + Mxx[ly][lx - 1]) * (T)idxx(gi, gj);
            if (gj == 0) my_yy = ((Myy[ly + 2][lx] - (T)2 * Myy[ly + 1][lx]) + Myy[ly][lx]) * (T)idyy(gi, 0);
            else if (gj == ny - 1) my_yy = ((Myy[ly][lx] - (T)2 * Myy[ly - 1][lx]) + Myy[ly - 2][lx]) * (T)idyy(gi, gj);
            else my_yy = ((Myy[ly + 1][lx] - (T)2 * Myy[ly][lx]) + Myy[ly - 1][lx]) * (T)idyy(gi, gj);
            const size_t e = (size_t)gj * nx + gi;
            T p = (T)0;
            if (mask[e]) {
                double pm = (double)q0[e];
                if (wref) pm += c.coef_mantle * (ys[ly][lx] - wref[e]);
                p = (T)pm;
            }
            f[e] = (((p + mx_xx) + (T)2 * mxy_xy) + my_yy) * inv2eta[e];
        }
    }
}

// Mixed form, uniform spacing.  The only double work per cell is the pair of
// forward differences of the double state, dX = y[i+1]-y[i] and
// dY = y[j+1]-y[j] (taken before rounding to float, so the second
// differences keep the small curvature of a large smooth field), and the
// mantle term y - w_ref.  Central and second differences are rebuilt
// exactly from them: y[i+1]-y[i-1] = dX[i]+dX[i-1],
// y[i+1]-2y[i]+y[i-1] = dX[i]-dX[i-1].
__device__ __forceinline__ void flexure_f32_body(const double* __restrict__ y, const double* __restrict__ wref,
                                                 const float* __restrict__ q0, const uint8_t* __restrict__ mask,
                                                 const float* __restrict__ D, const float* __restrict__ inv2eta,
                                                 float* __restrict__ f, int nx, int ny, FlexCoefF c, int bx, int by)
{
    __shared__ double ys[RY][RX];
    __shared__ float dX[RY][RX];
    __shared__ float dY[RY][RX];
    __shared__ float Wx[RY][RX];
    __shared__ float Mxx[RY][RX];
    __shared__ float Myy[RY][RX];
    __shared__ float Mxy[RY][RX];
    __shared__ float Mxyx[RY][RX];
    __shared__ float Ds[RY][RX];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int i0 = bx * TX - 2, j0 = by * TY - 2;   // global index of lx = ly = 0
    // every global input is requested up front, so their latencies overlap:
    // this thread's output cell ...
    const int go_i = i0 + tx + 2, go_j = j0 + ty + 2;
    const bool own = go_i < nx && go_j < ny;
    const size_t eo = own ? (size_t)go_j * nx + go_i : 0;
    const uint8_t own_m = own ? mask[eo] : (uint8_t)0;
    const float own_q = own ? q0[eo] : 0.f, own_ie = own ? inv2eta[eo] : 0.f;
    // ... and the state and rigidity tiles with their halo
    for (int ly = ty; ly < RY; ly += TY)
        for (int lx = tx; lx < RX; lx += TX) {
            const int gi = i0 + lx, gj = j0 + ly;
            const bool in = gi >= 0 && gi < nx && gj >= 0 && gj < ny;
            Ds[ly][lx] = in ? D[(size_t)gj * nx + gi] : 0.f;
            ys[ly][lx] = in ? y[(size_t)gj * nx + gi] : 0.0;
        }
    __syncthreads();
    for (int ly = ty; ly < RY; ly += TY)
        for (int lx = tx; lx < RX; lx += TX) {
            if (lx < RX - 1) dX[ly][lx] = (float)(ys[ly][lx + 1] - ys[ly][lx]);
            if (ly < RY - 1) dY[ly][lx] = (float)(ys[ly + 1][lx] - ys[ly][lx]);
        }
    __syncthreads();
    for (int ly = ty; ly < RY; ly += TY)
        for (int lx = tx + 1; lx < RX - 1; lx += TX) {
            const int gi = i0 + lx, gj = j0 + ly;
            if (gi < 0 || gi >= nx || gj < 0 || gj >= ny) continue;
            float v;
            if (gi == 0) v = dX[ly][lx] * c.inv_dx;
            else if (gi == nx - 1) v = dX[ly][lx - 1] * c.inv_dx;
            else v = (dX[ly][lx] + dX[ly][lx - 1]) * c.inv_2dx;
            Wx[ly][lx] = v;
        }
    __syncthreads();
    for (int ly = ty + 1; ly < RY - 1; ly += TY)
        for (int lx = tx + 1; lx < RX - 1; lx += TX) {
            const int gi = i0 + lx, gj = j0 + ly;
            if (gi < 0 || gi >= nx || gj < 0 || gj >= ny) continue;
            float wxy, wxx, wyy;
            if (gj == 0) wxy = (Wx[ly + 1][lx] - Wx[ly][lx]) * c.inv_dy;
            else if (gj == ny - 1) wxy = (Wx[ly][lx] - Wx[ly - 1][lx]) * c.inv_dy;
            else wxy = (Wx[ly + 1][lx] - Wx[ly - 1][lx]) * c.inv_2dy;
            if (gi == 0) wxx = (dX[ly][lx + 1] - dX[ly][lx]) * c.inv_dx2;
            else if (gi == nx - 1) wxx = (dX[ly][lx - 1] - dX[ly][lx - 2]) * c.inv_dx2;
            else wxx = (dX[ly][lx] - dX[ly][lx - 1]) * c.inv_dx2;
            if (gj == 0) wyy = (dY[ly + 1][lx] - dY[ly][lx]) * c.inv_dy2;
            else if (gj == ny - 1) wyy = (dY[ly - 1][lx] - dY[ly - 2][lx]) * c.inv_dy2;
            else wyy = (dY[ly][lx] - dY[ly - 1][lx]) * c.inv_dy2;
            const float Dl = Ds[ly][lx];
            Mxx[ly][lx] = -Dl * (wxx + c.nu * wyy);
            Myy[ly][lx] = -Dl * (wyy + c.nu * wxx);
            Mxy[ly][lx] = (-Dl * c.one_minus_nu) * wxy;
        }
    __syncthreads();
    for (int ly = ty + 1; ly < RY - 1; ly += TY)
        for (int lx = tx + 2; lx < RX - 2; lx += TX) {
            const int gi = i0 + lx, gj = j0 + ly;
            if (gi < 0 || gi >= nx || gj < 0 || gj >= ny) continue;
            float v;
            if (gi == 0) v = (Mxy[ly][lx + 1] - Mxy[ly][lx]) * c.inv_dx;
            else if (gi == nx - 1) v = (Mxy[ly][lx] - Mxy[ly][lx - 1]) * c.inv_dx;
            else v = (Mxy[ly][lx + 1] - Mxy[ly][lx - 1]) * c.inv_2dx;
            Mxyx[ly][lx] = v;
        }
    __syncthreads();
    const int lx = tx + 2, ly = ty + 2;
    const int gi = i0 + lx, gj = j0 + ly;
    if (gi >= nx || gj >= ny) return;
    float mxy_xy, mx_xx, my_yy;
    if (gj == 0) mxy_xy = (Mxyx[ly + 1][lx] - Mxyx[ly][lx]) * c.inv_dy;
    else if (gj == ny - 1) mxy_xy = (Mxyx[ly][lx] - Mxyx[ly - 1][lx]) * c.inv_dy;
    else mxy_xy = (Mxyx[ly + 1][lx] - Mxyx[ly - 1][lx]) * c.inv_2dy;
    if (gi == 0) mx_xx = ((Mxx[ly][lx + 2] - 2.f * Mxx[ly][lx + 1]) + Mxx[ly][lx]) * c.inv_dx2;
    else if (gi == nx - 1) mx_xx = ((Mxx[ly][lx] - 2.f * Mxx[ly][lx - 1]) + Mxx[ly][lx - 2]) * c.inv_dx2;
    else mx_xx = ((Mxx[ly][lx + 1] - 2.f * Mxx[ly][lx]) + Mxx[ly][lx - 1]) * c.inv_dx2;
    if (gj == 0) my_yy = ((Myy[ly + 2][lx] - 2.f * Myy[ly + 1][lx]) + Myy[ly][lx]) * c.inv_dy2;
    else if (gj == ny - 1) my_yy = ((Myy[ly][lx] - 2.f * Myy[ly - 1][lx]) + Myy[ly - 2][lx]) * c.inv_dy2;
    else my_yy = ((Myy[ly + 1][lx] - 2.f * Myy[ly][lx]) + Myy[ly - 1][lx]) * c.inv_dy2;
    const size_t e = eo;
    float p = 0.f;
    if (own_m) {
        p = own_q;
        if (wref) p += c.coef_mantle * (float)(ys[ly][lx] - wref[e]);
    }
    f[e] = (((p + mx_xx) + 2.f * mxy_xy) + my_yy) * own_ie;
}

// ---------------------------------------------------------------------------
// Flexure by column strips (mixed form, uniform spacing, the FP64 state: its
// first differences taken in double and rounded, as in flexure_f32_body, and
// with wref the mantle term coef_mantle (y - wref) at masked cells).  One
// warp task = SW output columns [SW g, SW g + SW) by `seg` output rows
// [seg s, seg s + seg): lane l holds column SW g - 2 + l and walks down the
// rows with the vertical stencil window in registers, taking x-neighbours by
// warp shuffles, so there is no shared memory and no block barrier.  Moments
// of row m are formed when input row m + 2 has been read, f of row o when
// moments of row o + 2 exist (the one-sided formulas of the first and last
// rows reach two rows further than the interior ones).
// ---------------------------------------------------------------------------
constexpr int SW = 28;                     // output columns per warp task

__device__ __forceinline__ int strip_tasks(int nx, int ny, int seg)
{
    return ((nx + SW - 1) / SW) * ((ny + seg - 1) / seg);
}

__device__ __forceinline__ void flexure_strip(const double* __restrict__ y, const double* __restrict__ wref,
                                              const float* __restrict__ q0, const uint8_t* __restrict__ mask,
                                              const float* __restrict__ D, const float* __restrict__ inv2eta,
                                              float* __restrict__ f, int nx, int ny, const FlexCoefF& c, int seg,
                                              int task)
{
    const unsigned FULL = 0xffffffffu;
    const int ncg = (nx + SW - 1) / SW;
    const int g = task % ncg, sg = task / ncg;
    const int lane = (int)(threadIdx.x + threadIdx.y * blockDim.x) & 31;   // 1D or 32 x 8 blocks
    const int col = g * SW - 2 + lane;
    const bool cin = col >= 0 && col < nx;
    const bool outl = cin && lane >= 2 && lane < 2 + SW;
    const bool left = col == 0, right = col == nx - 1;
    const bool edge = g == 0 || g == ncg - 1;   // warp-uniform: a lane may sit on x = 0 or x = nx - 1
    const int o0 = sg * seg, o1 = min(o0 + seg, ny);
    const int cc = cin ? col : 0;
    double yp = 0.0;                                    // state of row r - 1
    float Wx1 = 0.f, Wx2 = 0.f, Wx3 = 0.f;              // Wx of rows r-1, r-2, r-3
    float wxx1 = 0.f, wxx2 = 0.f;                       // wxx of rows r-1, r-2
    float dY1 = 0.f, dY2 = 0.f, dY3 = 0.f, dY4 = 0.f;   // dY of rows r-1 .. r-4 (dY_j = y_{j+1} - y_j)
    float My0 = 0.f, My1 = 0.f, My2 = 0.f, My3 = 0.f, My4 = 0.f;   // Myy of rows m .. m-4
    float Mq0 = 0.f, Mq1 = 0.f, Mq2 = 0.f, Mq3 = 0.f;              // Mxyx of rows m .. m-3
    float mx0 = 0.f, mx1 = 0.f, mx2 = 0.f;                         // mx_xx of rows m .. m-2
    // the next row's loads are issued one iteration ahead
    int r = o0 - 4;
    auto ld = [&](int rr) { return cin && rr >= 0 && rr < ny ? __ldg(y + (size_t)rr * nx + cc) : 0.0; };
    double yn = ld(r);
    for (; r < o1 + 4; ++r) {
        const double yv = yn;
        yn = ld(r + 1);
        const int m = r - 2, o = r - 4;
        const bool orow = outl && o >= o0 && o < o1;
        const size_t eo = orow ? (size_t)o * nx + cc : 0;
        const bool mrow = cin && m >= 0 && m < ny;
        const float Dm = mrow ? __ldg(D + (size_t)m * nx + cc) : 0.f;
        const uint32_t om = orow ? (uint32_t)__ldg(mask + eo) : 0u;
        const float oq = orow ? __ldg(q0 + eo) : 0.f, oie = orow ? __ldg(inv2eta + eo) : 0.f;
        // row r: first differences, Wx, wxx
        const double yr = __shfl_down_sync(FULL, yv, 1);
        const float dX = (float)(yr - yv);
        const float dXm = __shfl_up_sync(FULL, dX, 1);
        float Wx, wxx;
        if (edge) {
            const float dXp = __shfl_down_sync(FULL, dX, 1), dXmm = __shfl_up_sync(FULL, dX, 2);
            Wx = left ? dX * c.inv_dx : right ? dXm * c.inv_dx : (dX + dXm) * c.inv_2dx;
            wxx = left ? (dXp - dX) * c.inv_dx2 : right ? (dXm - dXmm) * c.inv_dx2 : (dX - dXm) * c.inv_dx2;
        } else {
            Wx = (dX + dXm) * c.inv_2dx;
            wxx = (dX - dXm) * c.inv_dx2;
        }
        const float dYn = (float)(yv - yp);   // dY of row r - 1
        yp = yv;
        dY4 = dY3; dY3 = dY2; dY2 = dY1; dY1 = dYn;
        // moments of row m = r - 2 (Wx1..3 are still those of rows r-1..r-3)
        float wxy, wyy;
        if (m == 0) {
            wxy = (Wx1 - Wx2) * c.inv_dy;
            wyy = (dY1 - dY2) * c.inv_dy2;
        } else if (m == ny - 1) {
            wxy = (Wx2 - Wx3) * c.inv_dy;
            wyy = (dY3 - dY4) * c.inv_dy2;
        } else {
            wxy = (Wx1 - Wx3) * c.inv_2dy;
            wyy = (dY2 - dY3) * c.inv_dy2;
        }
        const float wxm = wxx2;
        const float Mxx = -Dm * (wxm + c.nu * wyy);
        const float Myy = -Dm * (wyy + c.nu * wxm);
        const float Mxy = (-Dm * c.one_minus_nu) * wxy;
        Wx3 = Wx2; Wx2 = Wx1; Wx1 = Wx;
        wxx2 = wxx1; wxx1 = wxx;
        // x-derivatives of the moments of row m
        const float Mxyp = __shfl_down_sync(FULL, Mxy, 1), Mxym = __shfl_up_sync(FULL, Mxy, 1);
        const float Mxxp = __shfl_down_sync(FULL, Mxx, 1), Mxxm = __shfl_up_sync(FULL, Mxx, 1);
        float Mxyx, mxx;
        if (edge) {
            const float Mxxp2 = __shfl_down_sync(FULL, Mxx, 2), Mxxm2 = __shfl_up_sync(FULL, Mxx, 2);
            Mxyx = left ? (Mxyp - Mxy) * c.inv_dx : right ? (Mxy - Mxym) * c.inv_dx : (Mxyp - Mxym) * c.inv_2dx;
            mxx = left ? ((Mxxp2 - 2.f * Mxxp) + Mxx) * c.inv_dx2
                : right ? ((Mxx - 2.f * Mxxm) + Mxxm2) * c.inv_dx2
                : ((Mxxp - 2.f * Mxx) + Mxxm) * c.inv_dx2;
        } else {
            Mxyx = (Mxyp - Mxym) * c.inv_2dx;
            mxx = ((Mxxp - 2.f * Mxx) + Mxxm) * c.inv_dx2;
        }
        My4 = My3; My3 = My2; My2 = My1; My1 = My0; My0 = Myy;
        Mq3 = Mq2; Mq2 = Mq1; Mq1 = Mq0; Mq0 = Mxyx;
        mx2 = mx1; mx1 = mx0; mx0 = mxx;
        // f of row o = m - 2
        if (orow) {
            float mxy_xy, my_yy;
            if (o == 0) {
                mxy_xy = (Mq1 - Mq2) * c.inv_dy;
                my_yy = ((My0 - 2.f * My1) + My2) * c.inv_dy2;
            } else if (o == ny - 1) {
                mxy_xy = (Mq2 - Mq3) * c.inv_dy;
                my_yy = ((My2 - 2.f * My3) + My4) * c.inv_dy2;
            } else {
                mxy_xy = (Mq1 - Mq3) * c.inv_2dy;
                my_yy = ((My1 - 2.f * My2) + My3) * c.inv_dy2;
            }
            float p = om ? oq : 0.f;
            if (om && wref) p += c.coef_mantle * (float)(__ldg(y + eo) - __ldg(wref + eo));
            f[eo] = (((p + mx2) + 2.f * mxy_xy) + my_yy) * oie;
        }
    }
}

__global__ void __launch_bounds__(256)
k_flexure_strip_y(const double* __restrict__ y, const double* __restrict__ wref, const float* __restrict__ q0,
                  const uint8_t* __restrict__ mask, const float* __restrict__ D, const float* __restrict__ inv2eta,
                  float* __restrict__ f, int nx, int ny, FlexCoefF c, int seg, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    const int task = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (task >= strip_tasks(nx, ny, seg)) return;   // whole warps
    flexure_strip(y, wref, q0, mask, D, inv2eta, f, nx, ny, c, seg, task);
}

// rows per warp task for a single domain: enough tasks to fill the GPU
static int strip_seg_single(int nx, int ny)
{
    const long long ncg = (nx + SW - 1) / SW;
    long long seg = (long long)ny * ncg / (152 * 16);
    if (seg > 32) seg = 32;
    if (seg < 8) seg = 8;
    return (int)seg;
}

// ---------------------------------------------------------------------------
// FP64 flexure of the plain form on uniform spacing.  GB300 issues one FP64
// warp instruction every 64 clocks per SM quarter, whatever the instruction-
// level parallelism, so the stencil costs their number.  The tile form with
// per-cell spacing (k_flexure) executes about 70 per cell: its 32 x 8 tiles
// take every level on a halo of two, and every difference is scaled where it
// is taken.  Here the tile is 32 x 16, moments are formed straight from the
// stage state, all differences are left unscaled (the spacings sit in five
// factors, FlexCoef64), and the RK4 stage state x + sc raw is one FMA on the
// way into the tile instead of a kernel and a field of its own: 30 per cell.
// A walk down column strips as in flexure_strip needs 25 a lane and row but
// ran slower (512^2 50 us against 31 of the old tiles): at one or two warps a
// quarter nothing covers its loads, shuffles and addressing (FP64 pipe 39 %).
// STAGE: y = x + sc rprev; `off` = sc times the corner mean of rprev, which the
// differences drop and the mantle term takes off.
// R output rows of a tile: 16, or fewer where that fills the chip better.  A
// tile costs R + 2 rows of moments and R of outputs one after the other on its
// SM, which the rounds of tiles multiply (the last term: what a round cannot
// overlap of its first loads).  Plain / distorted, 16, 8, 4 rows: 122^2 12.9,
// 10.2, 8.4 / 15.6, 10.5, 8.7 us; 192^2 13.1, 10.1, 10.2 / 15.9, 10.9, 11.7;
// 256^2 12.8, 12.6, 13.5 / 15.9, 14.4, 16.0; 384^2 18.3, 18.1, 20.0 / 22.4,
// 23.3, 26.2; 512^2 28.6, 26.5, 30.3 / 38.6, 36.4, 40.6.
// ---------------------------------------------------------------------------
constexpr int TY64 = 16;                              // 32 x R outputs, 32 x 8 threads
constexpr int YC = TX + 4, MC = TX + 2;
constexpr int SMS = 152;   // multiprocessors of a GB300
static int tile64_rows(int nx, int ny)
{
    int best = 16;
    long long least = -1;
    for (int r : {16, 8, 4}) {
        const long long tiles = (long long)((nx + TX - 1) / TX) * ((ny + r - 1) / r);
        const long long cost = (tiles + SMS - 1) / SMS * (2 * r + 2) + r / 2;
        if (least < 0 || cost < least) { least = cost; best = r; }
    }
    return best;
}

template <bool STAGE, int R>
__device__ __forceinline__ void flexure_tile64(const double* __restrict__ x, const double* __restrict__ rprev,
                                               const double* __restrict__ wref, const double* __restrict__ q0,
                                               const uint8_t* __restrict__ mask, const double* __restrict__ D,
                                               const double* __restrict__ inv2eta, double* __restrict__ f, int nx,
                                               int ny, const FlexCoef64& c, int bx, int by, double sc = 0.0,
                                               double off = 0.0)
{
    __shared__ double ys[R + 4][YC];
    __shared__ double Mxx[R + 2][MC], Myy[R + 2][MC], Mxy[R + 2][MC];
    const int tid = (int)(threadIdx.x + threadIdx.y * blockDim.x);   // 1D or 32 x 8 blocks
    const int i0 = bx * TX, j0 = by * R;
    // tiles that touch no edge of the grid carry none of the one-sided forms
    const bool inner = i0 >= 2 && i0 + TX + 2 <= nx && j0 >= 2 && j0 + R + 2 <= ny;
    for (int e = tid; e < (R + 4) * YC; e += TX * TY) {
        const int ly = e / YC, lx = e - ly * YC;
        const int gi = i0 - 2 + lx, gj = j0 - 2 + ly;
        double v = 0.0;
        if (inner || (gi >= 0 && gi < nx && gj >= 0 && gj < ny)) {
            const size_t g = (size_t)gj * nx + gi;
            v = __ldg(x + g);
            if (STAGE) v += sc * __ldg(rprev + g);
        }
        ys[ly][lx] = v;
    }
    __syncthreads();
    if (inner) {
        for (int e = tid; e < (R + 2) * MC; e += TX * TY) {
            const int my = e / MC, mx = e - my * MC;
            const int ly = my + 1, lx = mx + 1;
            const double Dl = __ldg(D + (size_t)(j0 - 1 + my) * nx + (i0 - 1 + mx));
            const double y = ys[ly][lx];
            // differences of first differences, which are exact between
            // neighbours of a smooth field (a sum of neighbours less 2 y saves
            // two instructions and rounds at the size of y)
            const double wxx = (ys[ly][lx + 1] - y) - (y - ys[ly][lx - 1]);
            const double wyy = (ys[ly + 1][lx] - y) - (y - ys[ly - 1][lx]);
            const double wxy = (ys[ly + 1][lx + 1] - ys[ly + 1][lx - 1]) - (ys[ly - 1][lx + 1] - ys[ly - 1][lx - 1]);
            Mxx[my][mx] = Dl * (wxx + c.rxy * wyy);
            Myy[my][mx] = Dl * (wyy + c.ryx * wxx);
            Mxy[my][mx] = Dl * wxy;
        }
    } else {
        for (int e = tid; e < (R + 2) * MC; e += TX * TY) {
            const int my = e / MC, mx = e - my * MC;
            const int gi = i0 - 1 + mx, gj = j0 - 1 + my;
            if (gi < 0 || gi >= nx || gj < 0 || gj >= ny) continue;
            const int ly = my + 1, lx = mx + 1;
            // the one-sided second differences are the central ones one cell
            // inside, a one-sided first difference counts twice
            const int cx = lx + (gi == 0) - (gi == nx - 1), cy = ly + (gj == 0) - (gj == ny - 1);
            const int xl = lx - (gi > 0), xr = lx + (gi < nx - 1), yl = ly - (gj > 0), yr = ly + (gj < ny - 1);
            const double tw = (xr - xl == 2 ? 1.0 : 2.0) * (yr - yl == 2 ? 1.0 : 2.0);
            const double Dl = __ldg(D + (size_t)gj * nx + gi);
            const double wxx = (ys[ly][cx + 1] - ys[ly][cx]) - (ys[ly][cx] - ys[ly][cx - 1]);
            const double wyy = (ys[cy + 1][lx] - ys[cy][lx]) - (ys[cy][lx] - ys[cy - 1][lx]);
            const double wxy = tw * ((ys[yr][xr] - ys[yr][xl]) - (ys[yl][xr] - ys[yl][xl]));
            Mxx[my][mx] = Dl * (wxx + c.rxy * wyy);
            Myy[my][mx] = Dl * (wyy + c.ryx * wxx);
            Mxy[my][mx] = Dl * wxy;
        }
    }
    __syncthreads();
    for (int e = tid; e < TX * R; e += TX * TY) {
        const int ly = e / TX, lx = e - ly * TX;
        const int gi = i0 + lx, gj = j0 + ly;
        if (!inner && (gi >= nx || gj >= ny)) continue;
        const size_t g = (size_t)gj * nx + gi;
        double p = __ldg(q0 + g);
        const uint32_t on = __ldg(mask + g);
        const double ie = __ldg(inv2eta + g);
        const int my = ly + 1, mx = lx + 1;
        double mxx, myy, mxy;
        if (inner) {
            mxx = (Mxx[my][mx + 1] + Mxx[my][mx - 1]) - 2.0 * Mxx[my][mx];
            myy = (Myy[my + 1][mx] + Myy[my - 1][mx]) - 2.0 * Myy[my][mx];
            mxy = (Mxy[my + 1][mx + 1] - Mxy[my + 1][mx - 1]) - (Mxy[my - 1][mx + 1] - Mxy[my - 1][mx - 1]);
        } else {
            const int cx = mx + (gi == 0) - (gi == nx - 1), cy = my + (gj == 0) - (gj == ny - 1);
            const int xl = mx - (gi > 0), xr = mx + (gi < nx - 1), yl = my - (gj > 0), yr = my + (gj < ny - 1);
            const double tw = (xr - xl == 2 ? 1.0 : 2.0) * (yr - yl == 2 ? 1.0 : 2.0);
            mxx = (Mxx[my][cx + 1] + Mxx[my][cx - 1]) - 2.0 * Mxx[my][cx];
            myy = (Myy[cy + 1][mx] + Myy[cy - 1][mx]) - 2.0 * Myy[cy][mx];
            mxy = tw * ((Mxy[yr][xr] - Mxy[yr][xl]) - (Mxy[yl][xr] - Mxy[yl][xl]));
        }
        if (wref) p += c.cm * ((STAGE ? ys[ly + 2][lx + 2] - off : ys[ly + 2][lx + 2]) - __ldg(wref + g));
        if (on == 0) p = 0.0;
        f[g] = (((p + c.cxx * mxx) + c.cxy * mxy) + c.cyy * myy) * ie;
    }
}

// The same tile on a distorted grid: 1/(dx K), 1/(dy K) per cell (ixm, iym).
// A first difference takes the spacing of the cell it is taken at, a second
// one that cell's squared; the last column's second x-difference takes the
// first column's, as the reference does (src/finite_differences.f90:90-91).
// (256^2: 26.5 us with a division per difference on 32 x 8 tiles, 17 with the
// stored inverses, 14 on these tiles.)
template <int R>
__device__ __forceinline__ void flexure_tile64k(const double* __restrict__ x, const double* __restrict__ wref,
                                                const double* __restrict__ q0, const uint8_t* __restrict__ mask,
                                                const double* __restrict__ D, const double* __restrict__ inv2eta,
                                                double* __restrict__ f, int nx, int ny, const FlexCoef& c, int bx,
                                                int by)
{
    __shared__ double ys[R + 4][YC];
    __shared__ double Mxx[R + 2][MC], Myy[R + 2][MC], Mxy[R + 2][MC];
    const int tid = (int)(threadIdx.x + threadIdx.y * blockDim.x);   // 1D or 32 x 8 blocks
    const int i0 = bx * TX, j0 = by * R;
    for (int e = tid; e < (R + 4) * YC; e += TX * TY) {
        const int ly = e / YC, lx = e - ly * YC;
        const int gi = i0 - 2 + lx, gj = j0 - 2 + ly;
        ys[ly][lx] = gi >= 0 && gi < nx && gj >= 0 && gj < ny ? __ldg(x + (size_t)gj * nx + gi) : 0.0;
    }
    __syncthreads();
    // neighbours of grid cell (gi, gj) and its spacings: centre of the second
    // differences, ends of the first ones, 1/span of those in x at the two
    // rows and in y
    struct Nb {
        int cx, cy, xl, xr, yl, yr;
        double sl, sr, sy, ixx, iyy;
    };
    auto nb = [&](int gi, int gj) {
        Nb n;
        n.cx = (gi == 0) - (gi == nx - 1);
        n.cy = (gj == 0) - (gj == ny - 1);
        n.xl = -(gi > 0);
        n.xr = gi < nx - 1;
        n.yl = -(gj > 0);
        n.yr = gj < ny - 1;
        const size_t g = (size_t)gj * nx + gi;
        const double hx = n.xr - n.xl == 2 ? 0.5 : 1.0, hy = n.yr - n.yl == 2 ? 0.5 : 1.0;
        n.sl = hx * __ldg(c.ixm + (ptrdiff_t)g + (ptrdiff_t)n.yl * nx);
        n.sr = hx * __ldg(c.ixm + (ptrdiff_t)g + (ptrdiff_t)n.yr * nx);
        const double iy = __ldg(c.iym + g), ix = __ldg(c.ixm + (gi == nx - 1 ? g - gi : g));
        n.sy = hy * iy;
        n.ixx = ix * ix;
        n.iyy = iy * iy;
        return n;
    };
    const double nu = c.nu, omn = c.one_minus_nu;
    for (int e = tid; e < (R + 2) * MC; e += TX * TY) {
        const int my = e / MC, mx = e - my * MC;
        const int gi = i0 - 1 + mx, gj = j0 - 1 + my;
        if (gi < 0 || gi >= nx || gj < 0 || gj >= ny) continue;
        const Nb n = nb(gi, gj);
        const int ly = my + 1, lx = mx + 1, cx = lx + n.cx, cy = ly + n.cy;
        const double Dl = __ldg(D + (size_t)gj * nx + gi);
        const double wxx = ((ys[ly][cx + 1] - ys[ly][cx]) - (ys[ly][cx] - ys[ly][cx - 1])) * n.ixx;
        const double wyy = ((ys[cy + 1][lx] - ys[cy][lx]) - (ys[cy][lx] - ys[cy - 1][lx])) * n.iyy;
        const double wxy = ((ys[ly + n.yr][lx + n.xr] - ys[ly + n.yr][lx + n.xl]) * n.sr -
                            (ys[ly + n.yl][lx + n.xr] - ys[ly + n.yl][lx + n.xl]) * n.sl) * n.sy;
        Mxx[my][mx] = -Dl * (wxx + nu * wyy);
        Myy[my][mx] = -Dl * (wyy + nu * wxx);
        Mxy[my][mx] = (-Dl * omn) * wxy;
    }
    __syncthreads();
    for (int e = tid; e < TX * R; e += TX * TY) {
        const int ly = e / TX, lx = e - ly * TX;
        const int gi = i0 + lx, gj = j0 + ly;
        if (gi >= nx || gj >= ny) continue;
        const size_t g = (size_t)gj * nx + gi;
        const Nb n = nb(gi, gj);
        const int my = ly + 1, mx = lx + 1, cx = mx + n.cx, cy = my + n.cy;
        const double mxx = ((Mxx[my][cx + 1] - Mxx[my][cx]) - (Mxx[my][cx] - Mxx[my][cx - 1])) * n.ixx;
        const double myy = ((Myy[cy + 1][mx] - Myy[cy][mx]) - (Myy[cy][mx] - Myy[cy - 1][mx])) * n.iyy;
        const double mxy = ((Mxy[my + n.yr][mx + n.xr] - Mxy[my + n.yr][mx + n.xl]) * n.sr -
                            (Mxy[my + n.yl][mx + n.xr] - Mxy[my + n.yl][mx + n.xl]) * n.sl) * n.sy;
        double p = __ldg(q0 + g);
        if (wref) p += c.coef_mantle * (ys[ly + 2][lx + 2] - __ldg(wref + g));
        if (__ldg(mask + g) == 0) p = 0.0;
        f[g] = (((p + mxx) + 2.0 * mxy) + myy) * __ldg(inv2eta + g);
    }
}

template <int R>
__global__ void __launch_bounds__(TX* TY)
k_flexure64k(const double* __restrict__ y, const double* __restrict__ wref, const double* __restrict__ q0,
             const uint8_t* __restrict__ mask, const double* __restrict__ D, const double* __restrict__ inv2eta,
             double* __restrict__ f, int nx, int ny, FlexCoef c, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    flexure_tile64k<R>(y, wref, q0, mask, D, inv2eta, f, nx, ny, c, blockIdx.x, blockIdx.y);
}

template <int R>
__global__ void __launch_bounds__(TX* TY)
k_flexure64(const double* __restrict__ y, const double* __restrict__ wref, const double* __restrict__ q0,
            const uint8_t* __restrict__ mask, const double* __restrict__ D, const double* __restrict__ inv2eta,
            double* __restrict__ f, int nx, int ny, FlexCoef64 c, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    flexure_tile64<false, R>(y, nullptr, wref, q0, mask, D, inv2eta, f, nx, ny, c, blockIdx.x, blockIdx.y);
}

template <int R>
__global__ void __launch_bounds__(TX* TY)
k_flexure64_stage(const double* __restrict__ x, const double* __restrict__ rprev, const double* __restrict__ wref,
                  const double* __restrict__ q0, const uint8_t* __restrict__ mask, const double* __restrict__ D,
                  const double* __restrict__ inv2eta, double* __restrict__ f, int nx, int ny, FlexCoef64 c,
                  const Ctl* __restrict__ ctl, double a, double spy)
{
    __shared__ double s_sc[2];
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        s_sc[0] = (a * ctl->h) * spy;
        s_sc[1] = s_sc[0] * corner_mean_of(rprev, nx, ny);
    }
    __syncthreads();
    flexure_tile64<true, R>(x, rprev, wref, q0, mask, D, inv2eta, f, nx, ny, c, blockIdx.x, blockIdx.y, s_sc[0], s_sc[1]);
}

// fn(rows of a tile as a type, grid, block) with the rows tile64_rows takes
template <typename F> static void tile64_launch(int nx, int ny, F fn)
{
    const int r = tile64_rows(nx, ny);
    const dim3 g((nx + TX - 1) / TX, (ny + r - 1) / r), b(TX, TY);
    if (r == 4) fn(std::integral_constant<int, 4>{}, g, b);
    else if (r == 8) fn(std::integral_constant<int, 8>{}, g, b);
    else fn(std::integral_constant<int, 16>{}, g, b);
}

void launch_flexure_stage64(const double* x, const double* rprev, const double* wref, const double* q0,
                            const uint8_t* mask, const double* D, const double* inv2eta, double* f, int nx, int ny,
                            const FlexCoef& c, const Ctl* ctl, double a, double spy, cudaStream_t s)
{
    const FlexCoef64 cf = flex_coef_f64(c);
    tile64_launch(nx, ny, [&](auto r, dim3 g, dim3 b) {
        constexpr int R = decltype(r)::value;
        if (rprev)
            k_flexure64_stage<R><<<g, b, 0, s>>>(x, rprev, wref, q0, mask, D, inv2eta, f, nx, ny, cf, ctl, a, spy);
        else
            k_flexure64<R><<<g, b, 0, s>>>(x, wref, q0, mask, D, inv2eta, f, nx, ny, cf, nullptr);
    });
}

__global__ void __launch_bounds__(TX* TY)
k_flexure_f32(const double* __restrict__ y, const double* __restrict__ wref, const float* __restrict__ q0,
              const uint8_t* __restrict__ mask, const float* __restrict__ D, const float* __restrict__ inv2eta,
              float* __restrict__ f, int nx, int ny, FlexCoefF c, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    flexure_f32_body(y, wref, q0, mask, D, inv2eta, f, nx, ny, c, blockIdx.x, blockIdx.y);
}

// ---------------------------------------------------------------------------
// Mixed stencil by tiles (uniform spacing), the state as a float pair x =
// whi + wlo.  With rprev (the previous stage's raw RHS) the RK stage state
// x + sdf (rprev - cm) is formed on the way into the tile, sdf = (a h) spy
// with h the step size in the control block and cm the corner mean of rprev
// (thread 0 has the only FP64 instructions).  With dxw = x - w_ref the load
// takes the mantle term coef_mantle (dxw + sdf (rprev - cm)) at masked cells.
// Moments come from the tile, f from the moments.  64 x 16 outputs, 256 threads as four groups of
// 64 columns: a thread keeps its column in every pass, walks down it with the
// vertical window in registers, and has some fifteen independent loads in
// flight where column strips (a warp per 28 columns, shuffles for the
// x-neighbours) had one row's and waited on them: 2048^2 54.1 -> 43.9 us, 512 x
// 1024 16.8 -> 10.6 us an RK4 stage.  It issues 224 instructions a cell and
// keeps the issue slots 65 % busy; with cell indices divided out per element
// it issued 304 and took 50.9 us at 2048^2.
// The grid is even in both directions, so the last tile has two columns and
// two rows at least, which the one-sided forms at the far edges need.
// ---------------------------------------------------------------------------
constexpr int TXF = 64, TYF = 16, NGF = 4, YRF = TYF + 4, YCF = TXF + 4, MRF = TYF + 2, MCF = TXF + 2;

__device__ __forceinline__ void flexure_tile(const float* __restrict__ whi, const float* __restrict__ wlo,
                                             const float* __restrict__ rprev, const float* __restrict__ dxw,
                                             const float* __restrict__ q0, const uint8_t* __restrict__ mask,
                                             const float* __restrict__ D, const float* __restrict__ inv2eta,
                                             float* __restrict__ f, int nx, int ny, const FlexCoefF& c, int bx, int by,
                                             const Ctl* __restrict__ ctl = nullptr, double a = 0.0, double spy = 0.0)
{
    __shared__ float2 ys[YRF][YCF];
    __shared__ float Mxx[MRF][MCF], Myy[MRF][MCF], Mxy[MRF][MCF];
    __shared__ float s_sc[2];
    const int tid = threadIdx.x + threadIdx.y * blockDim.x, tx = tid % TXF, grp = tid / TXF;
    const int i0 = bx * TXF, j0 = by * TYF;
    const int gi = i0 + tx;                            // this thread's column
    const bool col = gi < nx;
    if (tid == 0) {
        s_sc[0] = rprev ? (float)(a * ctl->h * spy) : 0.f;
        s_sc[1] = rprev ? (float)corner_mean_of(rprev, nx, ny) : 0.f;
    }
    // the state: this column's rows grp, grp + 4, ..; the four halo columns by
    // the first 80 threads
    constexpr int NL = YRF / NGF;
    float2 xv[NL + 1];
    float rv[NL + 1];
    const int hr = tid / 4, hc = tid % 4, hx = hc < 2 ? hc : TXF + hc;   // halo element: row, tile column
    {
        const int ha = i0 - 2 + hx;
#pragma unroll
        for (int q = 0; q <= NL; ++q) {
            const int r = q < NL ? grp + NGF * q : hr, i = q < NL ? gi : ha, j = j0 - 2 + r;
            const bool in = (q < NL || tid < 4 * YRF) && i >= 0 && i < nx && j >= 0 && j < ny;
            const int g = in ? j * nx + i : 0;
            xv[q] = in ? make_float2(__ldg(whi + g), __ldg(wlo + g)) : make_float2(0.f, 0.f);
            rv[q] = in && rprev ? __ldg(rprev + g) : 0.f;
        }
    }
    __syncthreads();
    const float sdf = s_sc[0], cm = s_sc[1];
#pragma unroll
    for (int q = 0; q <= NL; ++q) {
        float2 v = xv[q];
        if (rprev) {   // two-sum of the pair and the increment (its corner mean drops out of every difference)
            const float inc = sdf * rv[q];
            const float sm = v.x + inc, bb = sm - v.x;
            const float er = (v.x - (sm - bb)) + (inc - bb);
            const float l2 = v.y + er;
            v.x = sm + l2;
            v.y = l2 - (v.x - sm);
        }
        if (q < NL) ys[grp + NGF * q][tx + 2] = v;
        else if (tid < 4 * YRF) ys[hr][hx] = v;
    }
    __syncthreads();
    auto dif = [](float2 p, float2 q) { return (q.x - p.x) + (q.y - p.y); };
    // moments of grid rows j0 - 1 .. j0 + 16, a run per group, walking down
    // three rows of this column
    const bool left = gi == 0, right = gi == nx - 1;
    const int lc = tx + 2 + (left ? 1 : right ? -1 : 0);   // centre of the second x-differences (tile column)
    const float sx = left || right ? c.inv_dx : c.inv_2dx;
    if (col) {
        constexpr int RUN = (MRF + NGF - 1) / NGF;
        int m0 = grp * RUN, m1 = min(m0 + RUN, MRF);
        if (j0 == 0 && m0 == 0) m0 = 1;
        m1 = min(m1, ny + 1 - j0);
        float w0 = 0.f, w1 = 0.f, w2, x1 = 0.f, x2;
        float2 y0, y1, y2;
        auto row = [&](int r, float& w, float& x, float2& y) {   // tile row r
            const float2 p = ys[r][lc - 1], q = ys[r][lc], s = ys[r][lc + 1];
            const float dA = dif(p, q), dB = dif(q, s);
            x = (dB - dA) * c.inv_dx2;
            w = (left ? dA : right ? dB : dA + dB) * sx;
            y = left ? p : right ? s : q;
        };
        if (m0 < m1) {
            row(m0, w0, x1, y0);
            row(m0 + 1, w1, x1, y1);
        }
        const float* Dp = D + (j0 - 1) * nx + gi;
#pragma unroll
        for (int q = 0; q < RUN; ++q) {
            const int m = m0 + q, j = j0 - 1 + m;
            if (m >= m1) break;
            const float Dl = __ldg(Dp + m * nx);
            row(m + 2, w2, x2, y2);
            float wxy, wyy;
            if (j == 0 || j == ny - 1) {
                wxy = (j == 0 ? w2 - w1 : w1 - w0) * c.inv_dy;
                const int r = (j == 0 ? 1 : ny - 2) - j0 + 2;
                wyy = (dif(ys[r][tx + 2], ys[r + 1][tx + 2]) - dif(ys[r - 1][tx + 2], ys[r][tx + 2])) * c.inv_dy2;
            } else {
                wxy = (w2 - w0) * c.inv_2dy;
                wyy = (dif(y1, y2) - dif(y0, y1)) * c.inv_dy2;
            }
            Mxx[m][tx + 1] = -Dl * (x1 + c.nu * wyy);
            Myy[m][tx + 1] = -Dl * (wyy + c.nu * x1);
            Mxy[m][tx + 1] = (-Dl * c.one_minus_nu) * wxy;
            w0 = w1; w1 = w2; x1 = x2; y0 = y1; y1 = y2;
        }
    }
    // and of the two columns beside the tile
    if (tid >= TXF * NGF - 2 * MRF) {
        const int e = tid - (TXF * NGF - 2 * MRF), m = e / 2, mx = e % 2 ? MCF - 1 : 0;
        const int i = i0 - 1 + mx, j = j0 - 1 + m;
        if (i >= 0 && i < nx && j >= 0 && j < ny) {
            const int lx = mx + 1, ly = m + 1;
            const int cx = lx + (i == 0) - (i == nx - 1), cy = ly + (j == 0) - (j == ny - 1);
            const int xl = lx - (i > 0), xr = lx + (i < nx - 1), yl = ly - (j > 0), yr = ly + (j < ny - 1);
            const float hxs = xr - xl == 2 ? c.inv_2dx : c.inv_dx, hys = yr - yl == 2 ? c.inv_2dy : c.inv_dy;
            const float Dl = __ldg(D + j * nx + i);
            const float wxx = (dif(ys[ly][cx], ys[ly][cx + 1]) - dif(ys[ly][cx - 1], ys[ly][cx])) * c.inv_dx2;
            const float wyy = (dif(ys[cy][lx], ys[cy + 1][lx]) - dif(ys[cy - 1][lx], ys[cy][lx])) * c.inv_dy2;
            const float wxy = (dif(ys[yr][xl], ys[yr][xr]) * hxs - dif(ys[yl][xl], ys[yl][xr]) * hxs) * hys;
            Mxx[m][mx] = -Dl * (wxx + c.nu * wyy);
            Myy[m][mx] = -Dl * (wyy + c.nu * wxx);
            Mxy[m][mx] = (-Dl * c.one_minus_nu) * wxy;
        }
    }
    // the output rows' operands, requested before the barrier
    constexpr int RO = TYF / NGF;
    float qv[RO], iv[RO], dv[RO], ov[RO];
    uint32_t on[RO];
    const int o0 = grp * RO, ge = (j0 + o0) * nx + gi;
#pragma unroll
    for (int q = 0; q < RO; ++q) {
        const bool in = col && j0 + o0 + q < ny;
        const int g = in ? ge + q * nx : 0;
        qv[q] = in ? __ldg(q0 + g) : 0.f;
        iv[q] = in ? __ldg(inv2eta + g) : 0.f;
        dv[q] = in && dxw ? __ldg(dxw + g) : 0.f;
        ov[q] = in && rprev ? __ldg(rprev + g) : 0.f;
        on[q] = in ? (uint32_t)__ldg(mask + g) : 0u;
    }
    __syncthreads();
    if (!col) return;
    const int mc = tx + 1, cc = mc + (left ? 1 : right ? -1 : 0), cl = mc - (left ? 0 : 1), cr = mc + (right ? 0 : 1);
    // output row o is row o + 1 of the moments
    float q0v = (Mxy[o0][cr] - Mxy[o0][cl]) * sx, q1v = (Mxy[o0 + 1][cr] - Mxy[o0 + 1][cl]) * sx;
    float y0 = Myy[o0][mc], y1 = Myy[o0 + 1][mc];
#pragma unroll
    for (int q = 0; q < RO; ++q) {
        const int o = o0 + q, j = j0 + o, m = o + 1;
        if (j >= ny) break;
        const float q2v = (Mxy[m + 1][cr] - Mxy[m + 1][cl]) * sx, y2 = Myy[m + 1][mc];
        const float mxx = ((Mxx[m][cc + 1] - 2.f * Mxx[m][cc]) + Mxx[m][cc - 1]) * c.inv_dx2;
        float mxy, myy;
        if (j == 0 || j == ny - 1) {
            mxy = (j == 0 ? q2v - q1v : q1v - q0v) * c.inv_dy;
            const int r = (j == 0 ? 1 : ny - 2) - j0 + 1;
            myy = ((Myy[r + 1][mc] - 2.f * Myy[r][mc]) + Myy[r - 1][mc]) * c.inv_dy2;
        } else {
            mxy = (q2v - q0v) * c.inv_2dy;
            myy = ((y2 - 2.f * y1) + y0) * c.inv_dy2;
        }
        float dy = dv[q];
        if (rprev) dy += sdf * (ov[q] - cm);
        const float p = on[q] ? (dxw ? qv[q] + c.coef_mantle * dy : qv[q]) : 0.f;
        f[ge + q * nx] = (((p + mxx) + 2.f * mxy) + myy) * iv[q];
        q0v = q1v; q1v = q2v; y0 = y1; y1 = y2;
    }
}

__global__ void __launch_bounds__(TXF* NGF)
k_flexure_tile(const float* __restrict__ whi, const float* __restrict__ wlo, const float* __restrict__ rprev,
               const float* __restrict__ dxw, const float* __restrict__ q0, const uint8_t* __restrict__ mask,
               const float* __restrict__ D, const float* __restrict__ inv2eta, float* __restrict__ f, int nx, int ny,
               FlexCoefF c, const Ctl* __restrict__ ctl, double a, double spy, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    flexure_tile(whi, wlo, rprev, dxw, q0, mask, D, inv2eta, f, nx, ny, c, blockIdx.x, blockIdx.y, ctl, a, spy);
}
static dim3 tile_grid(int nx, int ny) { return dim3((nx + TXF - 1) / TXF, (ny + TYF - 1) / TYF); }

template <typename T>
void launch_flexure(const double* y, const double* wref, const T* q0, const uint8_t* mask, const T* D,
                    const T* inv2eta, T* f, int nx, int ny, const FlexCoef& c, cudaStream_t s, const int* gate,
                    const float* whi, const float* wlo)
{
    dim3 b(TX, TY), g((nx + TX - 1) / TX, (ny + TY - 1) / TY);
    if (sizeof(T) == 4 && c.ixm == nullptr) {
        const FlexCoefF cf = flex_coef_f32(c);
        if (whi && !wref) {
            k_flexure_tile<<<tile_grid(nx, ny), TXF * NGF, 0, s>>>(whi, wlo, nullptr, nullptr, (const float*)q0, mask,
                                                                   (const float*)D, (const float*)inv2eta, (float*)f,
                                                                   nx, ny, cf, nullptr, 0.0, 0.0, gate);
            return;
        }
        // the FP64 state by column strips (the shared-memory tile form is
        // kept for FI_FLEXURE_TILES=1)
        static const bool tiles = [] {
            const char* e = getenv("FI_FLEXURE_TILES");
            return e && e[0] == '1';
        }();
        if (!tiles) {
            const int seg = strip_seg_single(nx, ny);
            const int tasks = ((nx + SW - 1) / SW) * ((ny + seg - 1) / seg);
            k_flexure_strip_y<<<(tasks + 7) / 8, 256, 0, s>>>(y, wref, (const float*)q0, mask, (const float*)D,
                                                              (const float*)inv2eta, (float*)f, nx, ny, cf, seg, gate);
            return;
        }
        k_flexure_f32<<<g, b, 0, s>>>(y, wref, (const float*)q0, mask, (const float*)D, (const float*)inv2eta,
                                      (float*)f, nx, ny, cf, gate);
        return;
    }
    if constexpr (sizeof(T) == 8) {
        tile64_launch(nx, ny, [&](auto r, dim3 g64, dim3 b64) {
            constexpr int R = decltype(r)::value;
            if (c.ixm == nullptr)
                k_flexure64<R><<<g64, b64, 0, s>>>(y, wref, q0, mask, D, inv2eta, f, nx, ny, flex_coef_f64(c), gate);
            else
                k_flexure64k<R><<<g64, b64, 0, s>>>(y, wref, q0, mask, D, inv2eta, f, nx, ny, c, gate);
        });
    } else {
        k_flexure<<<g, b, 0, s>>>(y, wref, q0, mask, D, inv2eta, f, nx, ny, c, gate);
    }
}

void launch_flexure_stage(const float* whi, const float* wlo, const float* rprev, const float* dxw, const float* q0,
                          const uint8_t* mask, const float* D, const float* inv2eta, float* f, int nx, int ny,
                          const FlexCoef& c, const Ctl* ctl, double a, double spy, cudaStream_t s,
                          const int* gate)
{
    k_flexure_tile<<<tile_grid(nx, ny), TXF * NGF, 0, s>>>(whi, wlo, rprev, dxw, q0, mask, D, inv2eta, f, nx, ny,
                                                           flex_coef_f32(c), ctl, a, spy, gate);
}

// ---------------------------------------------------------------------------
// Row transforms.  A block handles RB rows; nx real samples are packed as
// h = nx/2 complex samples (z[m] = x[2m] + i x[2m+1]).
// ---------------------------------------------------------------------------
static int rows_per_block(int h)
{
    int rb = 512 / (h > 0 ? h : 1);
    if (rb < 1) rb = 1;
    if (rb > 8) rb = 8;
    return rb;
}
static int threads_for(int work)
{
    int t = 32;
    while (t < work && t < 256) t *= 2;
    return t;
}

template <typename T>
__device__ __forceinline__ void rows_fwd_body(const T* __restrict__ in, int in_pitch, int in_width, int nrows_in,
                           typename vec2<T>::type* __restrict__ S, Plan2D p, int RB, int bx, int by)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ unsigned char smem_raw[];
    C2* b0 = reinterpret_cast<C2*>(smem_raw);
    C2* b1 = b0 + RB * p.h;
    const int h = p.h;
    const int j0 = bx * RB;
    const int nthr = blockDim.x;
    for (int e = threadIdx.x; e < RB * h; e += nthr) {
        const int line = e / h, m = e - line * h;
        const int j = j0 + line;
        C2 v = mk2<T>((T)0, (T)0);
        if (j < nrows_in) {
            const T* row = in + (size_t)j * in_pitch;
            const int i = 2 * m;
            if (i + 1 < in_width) {
                if ((in_pitch & 1) == 0) v = *reinterpret_cast<const C2*>(row + i);
                else v = mk2<T>(row[i], row[i + 1]);
            } else if (i < in_width) {
                v = mk2<T>(row[i], (T)0);
            }
        }
        b0[e] = v;
    }
    __syncthreads();
    C2* r = block_fft<T>(b0, b1, p.row.d, RB, h, twp<T>(p.row), -1);
    const C2* rtw = rtwp<T>(p);
    for (int e = threadIdx.x; e < RB * (h + 1); e += nthr) {
        const int line = e / (h + 1), k = e - line * (h + 1);
        const int j = j0 + line;
        if (j >= nrows_in) continue;
        const C2 Zk = r[line * h + (k == h ? 0 : k)];
        const C2 Zc = r[line * h + (k == 0 ? 0 : h - k)];
        C2 E, O;
        E.x = (T)0.5 * (Zk.x + Zc.x);
        E.y = (T)0.5 * (Zk.y - Zc.y);
        O.x = (T)0.5 * (Zk.y + Zc.y);
        O.y = (T)-0.5 * (Zk.x - Zc.x);
        S[(size_t)j * p.sp + k] = cadd(E, cmul(__ldg(rtw + k), O));
    }
}

template <typename T>
__global__ void k_rows_fwd(const T* __restrict__ in, int in_pitch, int in_width, int nrows_in,
                           typename vec2<T>::type* __restrict__ S, Plan2D p, int RB, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    rows_fwd_body<T>(in, in_pitch, in_width, nrows_in, S, p, RB, blockIdx.x, 0);
}

template <typename T>
void launch_rows_fwd(const T* in, int in_pitch, int in_width, int nrows_in, typename vec2<T>::type* S,
                     const Plan2D& p, cudaStream_t s, const int* gate)
{
    typedef typename vec2<T>::type C2;
    if (lines_rows_fwd<T>(in, in_pitch, in_width, nrows_in, S, p, s, gate)) return;
    const int RB = p.rb > 0 ? p.rb : rows_per_block(p.h);
    const size_t sm = 2 * (size_t)RB * p.h * sizeof(C2);
    set_smem(k_rows_fwd<T>, sm);
    const int nblk = (nrows_in + RB - 1) / RB;
    const int nt = p.rt > 0 ? p.rt : threads_for(RB * p.h / 4);
    k_rows_fwd<T><<<nblk, nt, sm, s>>>(in, in_pitch, in_width, nrows_in, S, p, RB, gate);
}

template <typename T>
__device__ __forceinline__ void rows_inv_body(const typename vec2<T>::type* __restrict__ S, int nrows, T* __restrict__ out,
                           int out_pitch, Plan2D p, int RB, T scale, int bx, int by)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ unsigned char smem_raw[];
    C2* b0 = reinterpret_cast<C2*>(smem_raw);
    C2* b1 = b0 + RB * p.h;
    const int h = p.h;
    const int j0 = bx * RB;
    const int nthr = blockDim.x;
    const C2* rtw = rtwp<T>(p);
    // Z[k] = (X[k] + conj X[h-k]) + i conj(w^k) (X[k] - conj X[h-k])
    for (int e = threadIdx.x; e < RB * h; e += nthr) {
        const int line = e / h, k = e - line * h;
        const int j = j0 + line;
        C2 z = mk2<T>((T)0, (T)0);
        if (j < nrows) {
            const C2 A = S[(size_t)j * p.sp + k];
            C2 B = S[(size_t)j * p.sp + (h - k)];
            B.y = -B.y;
            const C2 sum = cadd(A, B), dif = csub(A, B);
            const C2 t = cmulc(dif, __ldg(rtw + k));
            z.x = sum.x - t.y;
            z.y = sum.y + t.x;
        }
        b0[e] = z;
    }
    __syncthreads();
    C2* r = block_fft<T>(b0, b1, p.row.d, RB, h, twp<T>(p.row), +1);
    for (int e = threadIdx.x; e < RB * h; e += nthr) {
        const int line = e / h, m = e - line * h;
        const int j = j0 + line;
        if (j >= nrows) continue;
        C2 v = r[e];
        v.x *= scale;
        v.y *= scale;
        *reinterpret_cast<C2*>(out + (size_t)j * out_pitch + 2 * m) = v;
    }
}

template <typename T>
__global__ void k_rows_inv(const typename vec2<T>::type* __restrict__ S, int nrows, T* __restrict__ out,
                           int out_pitch, Plan2D p, int RB, T scale, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    rows_inv_body<T>(S, nrows, out, out_pitch, p, RB, scale, blockIdx.x, 0);
}

template <typename T>
void launch_rows_inv(const typename vec2<T>::type* S, T* out, const Plan2D& p, double scale, cudaStream_t s,
                     const int* gate)
{
    typedef typename vec2<T>::type C2;
    if (lines_rows_inv<T>(S, out, p, scale, s, gate)) return;
    const int RB = p.rb > 0 ? p.rb : rows_per_block(p.h);
    const size_t sm = 2 * (size_t)RB * p.h * sizeof(C2);
    set_smem(k_rows_inv<T>, sm);
    const int nblk = (p.ny + RB - 1) / RB;
    const int nt = p.rt > 0 ? p.rt : threads_for(RB * p.h / 4);
    k_rows_inv<T><<<nblk, nt, sm, s>>>(S, p.ny, out, p.nx, p, RB, (T)scale, gate);
}

// ---------------------------------------------------------------------------
// Column kernels.  A block loads CB spectrum columns (all ny rows) into
// shared memory, column-major, and transforms them together.
// ---------------------------------------------------------------------------
// Columns per block: two float2 or one double2 column, i.e. 16-byte row
// segments, which keeps hundreds of blocks in flight at 512^2.
// Column c of a block lives at c * col_stride(ny) in shared memory: one
// complex element of padding per column, so the CB columns of a row segment
// (loaded and stored together) fall in different banks instead of one.
__host__ __device__ __forceinline__ int col_stride(int ny) { return ny + 1; }

template <typename T> static int cols_per_block(int ny)
{
    typedef typename vec2<T>::type C2;
    int cb = (int)(16 / sizeof(C2));
    if (cb < 1) cb = 1;
    while (cb > 1 && 2 * (size_t)cb * col_stride(ny) * sizeof(C2) > 200 * 1024) cb /= 2;
    return cb;
}

template <typename T>
__device__ __forceinline__ void load_cols(typename vec2<T>::type* b0, const typename vec2<T>::type* S, int k0,
                                          int CB, int nrows_in, const Plan2D& p)
{
    typedef typename vec2<T>::type C2;
    const int ny = p.col.d.n, ls = col_stride(ny);
    for (int e = threadIdx.x; e < CB * ny; e += blockDim.x) {
        const int c = e % CB, l = e / CB;
        const int k = k0 + c;
        C2 v = mk2<T>((T)0, (T)0);
        if (k <= p.h && l < nrows_in) v = S[(size_t)l * p.sp + k];
        b0[c * ls + l] = v;
    }
}

template <typename T>
__device__ __forceinline__ void cols_hartley_body(typename vec2<T>::type* __restrict__ S, const T* __restrict__ mA,
                               const T* __restrict__ mB, int even, Plan2D p, int CB, int bx, int by)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ unsigned char smem_raw[];
    const int ny = p.col.d.n, ls = col_stride(ny);
    C2* b0 = reinterpret_cast<C2*>(smem_raw);
    C2* b1 = b0 + (size_t)CB * ls;
    const int k0 = bx * CB;
    load_cols<T>(b0, S, k0, CB, ny, p);
    __syncthreads();
    C2* r = block_fft<T>(b0, b1, p.col.d, CB, ls, twp<T>(p.col), -1);
    const int half = ny / 2 + 1;
    for (int e = threadIdx.x; e < CB * half; e += blockDim.x) {
        const int c = e % CB, l = e / CB;
        const int k = k0 + c;
        if (k > p.h) continue;
        const int lm = (ny - l) % ny;
        C2* col = r + (size_t)c * ls;
        const size_t ia = (size_t)l * p.sp + k, ib = (size_t)lm * p.sp + k;
        const C2 Fa = col[l], Fb = col[lm];
        if (even) {
            const T ma = mA[ia], mb = mA[ib];
            C2 a = Fa, b = Fb;
            a.x *= ma; a.y *= ma;
            b.x *= mb; b.y *= mb;
            col[l] = a;
            if (lm != l) col[lm] = b;
        } else {
            // Hartley values at (k,l), (-k,-l), (-k,l), (k,-l)
            const T H_kl = Fb.x - Fa.y, H_mkml = Fb.x + Fa.y;
            const T H_mkl = Fa.x + Fb.y, H_kml = Fa.x - Fb.y;
            const T G_kl = mA[ia] * H_kl, G_kml = mA[ib] * H_kml;
            const T G_mkl = mB[ia] * H_mkl, G_mkml = mB[ib] * H_mkml;
            C2 a, b;
            a.x = (T)0.5 * (G_kml + G_mkl);
            a.y = (T)0.5 * (G_mkml - G_kl);
            b.x = (T)0.5 * (G_kl + G_mkml);
            b.y = (T)0.5 * (G_mkl - G_kml);
            col[l] = a;
            if (lm != l) col[lm] = b;
        }
    }
    __syncthreads();
    C2* other = (r == b0) ? b1 : b0;
    C2* q = block_fft<T>(r, other, p.col.d, CB, ls, twp<T>(p.col), +1);
    for (int e = threadIdx.x; e < CB * ny; e += blockDim.x) {
        const int c = e % CB, l = e / CB;
        const int k = k0 + c;
        if (k <= p.h) S[(size_t)l * p.sp + k] = q[c * ls + l];
    }
}

template <typename T>
__global__ void k_cols_hartley(typename vec2<T>::type* __restrict__ S, const T* __restrict__ mA,
                               const T* __restrict__ mB, int even, Plan2D p, int CB, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    cols_hartley_body<T>(S, mA, mB, even, p, CB, blockIdx.x, 0);
}

template <typename T>
void launch_cols_hartley(typename vec2<T>::type* S, const T* mA, const T* mB, int even, const Plan2D& p,
                         cudaStream_t s, const int* gate)
{
    typedef typename vec2<T>::type C2;
    if (lines_cols_hartley<T>(S, mA, mB, even, p, s, gate)) return;
    const int CB = p.cb > 0 ? p.cb : cols_per_block<T>(p.ny);
    const size_t sm = 2 * (size_t)CB * col_stride(p.ny) * sizeof(C2);
    set_smem(k_cols_hartley<T>, sm);
    const int nblk = (p.h + 1 + CB - 1) / CB;
    const int nt = p.ct > 0 ? p.ct : threads_for(CB * p.ny / 4);
    k_cols_hartley<T><<<nblk, nt, sm, s>>>(S, mA, mB, even, p, CB, gate);
}

template <typename T>
__global__ void k_cols_conv(typename vec2<T>::type* __restrict__ S, const typename vec2<T>::type* __restrict__ K,
                            int nrows_in, const int* __restrict__ out_rows, int n_out, Plan2D p, int CB, int do_inv)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ unsigned char smem_raw[];
    const int ny = p.col.d.n, ls = col_stride(ny);
    C2* b0 = reinterpret_cast<C2*>(smem_raw);
    C2* b1 = b0 + (size_t)CB * ls;
    const int k0 = blockIdx.x * CB;
    load_cols<T>(b0, S, k0, CB, nrows_in, p);
    __syncthreads();
    C2* r = block_fft<T>(b0, b1, p.col.d, CB, ls, twp<T>(p.col), -1);
    if (!do_inv) {
        for (int e = threadIdx.x; e < CB * ny; e += blockDim.x) {
            const int c = e % CB, l = e / CB;
            const int k = k0 + c;
            if (k <= p.h) S[(size_t)l * p.sp + k] = r[c * ls + l];
        }
        return;
    }
    for (int e = threadIdx.x; e < CB * ny; e += blockDim.x) {
        const int c = e % CB, l = e / CB;
        const int k = k0 + c;
        if (k > p.h) continue;
        r[c * ls + l] = cmul(r[c * ls + l], K[(size_t)l * p.sp + k]);
    }
    __syncthreads();
    C2* other = (r == b0) ? b1 : b0;
    C2* q = block_fft<T>(r, other, p.col.d, CB, ls, twp<T>(p.col), +1);
    for (int e = threadIdx.x; e < CB * n_out; e += blockDim.x) {
        const int c = e % CB, o = e / CB;
        const int k = k0 + c;
        if (k <= p.h) S[(size_t)o * p.sp + k] = q[c * ls + out_rows[o]];
    }
}

template <typename T>
void launch_cols_conv(typename vec2<T>::type* S, const typename vec2<T>::type* K, int nrows_in, const int* out_rows,
                      int n_out, const Plan2D& p, cudaStream_t s)
{
    typedef typename vec2<T>::type C2;
    if (lines_cols_conv<T>(S, K, nrows_in, n_out, p, s)) return;
    const int CB = p.cb > 0 ? p.cb : cols_per_block<T>(p.ny);
    const size_t sm = 2 * (size_t)CB * col_stride(p.ny) * sizeof(C2);
    set_smem(k_cols_conv<T>, sm);
    const int nblk = (p.h + 1 + CB - 1) / CB;
    const int nt = p.ct > 0 ? p.ct : threads_for(CB * p.ny / 4);
    k_cols_conv<T><<<nblk, nt, sm, s>>>(S, K, nrows_in, out_rows, n_out, p, CB, 1);
}

template <typename T>
void launch_cols_fwd(typename vec2<T>::type* S, int nrows_in, const Plan2D& p, cudaStream_t s)
{
    typedef typename vec2<T>::type C2;
    const int CB = p.cb > 0 ? p.cb : cols_per_block<T>(p.ny);
    const size_t sm = 2 * (size_t)CB * col_stride(p.ny) * sizeof(C2);
    set_smem(k_cols_conv<T>, sm);
    const int nblk = (p.h + 1 + CB - 1) / CB;
    k_cols_conv<T><<<nblk, threads_for(CB * p.ny / 4), sm, s>>>(S, nullptr, nrows_in, nullptr, 0, p, CB, 0);
}

// Inverse rows of the compacted convolution spectrum.  Rows 0..ny-1 are the
// cropped output rows; rows ny and ny+1 are the linear-lag rows 0 and
// 2*ny-2 that hold the corner values of apply_zerobc_at_corners_dp.
template <typename T>
__global__ void k_conv_rows_inv(const typename vec2<T>::type* __restrict__ S, int n_out, double* __restrict__ out,
                                int nx, int ny, int i_off, double* __restrict__ corners, int col1, Plan2D p,
                                int RB, T scale)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ unsigned char smem_raw[];
    C2* b0 = reinterpret_cast<C2*>(smem_raw);
    C2* b1 = b0 + RB * p.h;
    const int h = p.h;
    const int j0 = blockIdx.x * RB;
    const int nthr = blockDim.x;
    const C2* rtw = rtwp<T>(p);
    for (int e = threadIdx.x; e < RB * h; e += nthr) {
        const int line = e / h, k = e - line * h;
        const int j = j0 + line;
        C2 z = mk2<T>((T)0, (T)0);
        if (j < n_out) {
            const C2 A = S[(size_t)j * p.sp + k];
            C2 B = S[(size_t)j * p.sp + (h - k)];
            B.y = -B.y;
            const C2 sum = cadd(A, B), dif = csub(A, B);
            const C2 t = cmulc(dif, __ldg(rtw + k));
            z.x = sum.x - t.y;
            z.y = sum.y + t.x;
        }
        b0[e] = z;
    }
    __syncthreads();
    C2* r = block_fft<T>(b0, b1, p.row.d, RB, h, twp<T>(p.row), +1);
    const T* rr = reinterpret_cast<const T*>(r);
    for (int e = threadIdx.x; e < RB * nx; e += nthr) {
        const int line = e / nx, i = e - line * nx;
        const int j = j0 + line;
        if (j < ny) out[(size_t)j * nx + i] = (double)(rr[(size_t)line * 2 * h + i_off + i] * scale);
    }
    if (threadIdx.x == 0) {
        for (int line = 0; line < RB; ++line) {
            const int j = j0 + line;
            const T* row = rr + (size_t)line * 2 * h;
            if (j == ny) {            // linear lag row 0
                corners[0] = (double)(row[0] * scale);
                corners[3] = (double)(row[col1] * scale);
            } else if (j == ny + 1) { // linear lag row 2*ny-2
                corners[2] = (double)(row[0] * scale);
                corners[1] = (double)(row[col1] * scale);
            }
        }
    }
}

template <typename T>
void launch_conv_rows_inv(const typename vec2<T>::type* S, int n_out, double* out, int nx, int ny, int i_off,
                          double* corners, int /*corner_row0*/, int /*corner_row1*/, int corner_col1,
                          const Plan2D& p, double scale, cudaStream_t s)
{
    typedef typename vec2<T>::type C2;
    if (lines_conv_rows_inv<T>(S, n_out, out, nx, ny, i_off, corners, corner_col1, p, scale, s)) return;
    const int RB = p.rb > 0 ? p.rb : rows_per_block(p.h);
    const size_t sm = 2 * (size_t)RB * p.h * sizeof(C2);
    set_smem(k_conv_rows_inv<T>, sm);
    const int nblk = (n_out + RB - 1) / RB;
    const int nt = p.rt > 0 ? p.rt : threads_for(RB * p.h / 4);
    k_conv_rows_inv<T><<<nblk, nt, sm, s>>>(S, n_out, out, nx, ny, i_off, corners, corner_col1, p, RB, (T)scale);
}

// ---------------------------------------------------------------------------
// Batched launches: the same bodies over every member of an ensemble.  A
// member whose attempt needs no new RHS (need_rhs == 0) returns at once.
// ---------------------------------------------------------------------------
int rhs_rows_per_block(int h) { return rows_per_block(h); }
int rhs_threads_for(int work) { return threads_for(work); }
template <typename T> int rhs_cols_per_block(int ny) { return cols_per_block<T>(ny); }
int rhs_line_threads(int n, const Plan2D& p, bool f32)
{
    // the batched kernels carry every line length they take; one that a
    // single domain would transform on lines has to be among them, or the
    // member would not get the bits it gets alone
    const long long points = (long long)p.h * p.ny;
    return f32 ? line_threads<float>(n, points) : line_threads<double>(n, points);
}
size_t rhs_line_bytes(int n, bool f32) { return f32 ? line_bytes<float>(n) : line_bytes<double>(n); }
template int rhs_cols_per_block<float>(int);
template int rhs_cols_per_block<double>(int);

template <typename T>
__global__ void __launch_bounds__(256) k_b_flexure(const BMember* __restrict__ M, BList L)
{
    batch_walk(L, [&](int m) { return true; }, [&](int m, int local) {   // the list holds the members with work
        const BMember& b = M[m];
        const int bx = local % b.fgx, by = local / b.fgx;
        if constexpr (sizeof(T) == 4) {
            // mixed members have uniform spacing and carry now%w as a float pair
            flexure_tile(b.d.whi, b.d.wlo, nullptr, nullptr, (const float*)b.q0, b.mask, (const float*)b.D,
                         (const float*)b.inv2eta, (float*)b.f, b.p.nx, b.p.ny, b.fcf, bx, by);
        } else if (b.fc.ixm == nullptr) {
            flexure_tile64<false, TY64>(b.y, nullptr, nullptr, (const double*)b.q0, b.mask, (const double*)b.D,
                                  (const double*)b.inv2eta, (double*)b.f, b.p.nx, b.p.ny, b.fc64, bx, by);
        } else {
            flexure_tile64k<TY64>(b.y, nullptr, (const double*)b.q0, b.mask, (const double*)b.D, (const double*)b.inv2eta,
                            (double*)b.f, b.p.nx, b.p.ny, b.fc, bx, by);
        }
        __syncthreads();   // the next virtual block reuses the shared tiles
    });
}

template <typename T>
__global__ void __launch_bounds__(512) k_b_rows_fwd(const BMember* __restrict__ M, BList L)
{
    typedef typename vec2<T>::type C2;
    batch_walk(L, [&](int m) { return true; }, [&](int m, int local) {   // the list holds the members with work
        const BMember& b = M[m];
        if (b.lines & 1) {
#define FI_GO(N) rows_fwd_lines<T, N>((const T*)b.f, b.p.nx, b.p.nx, b.p.ny, (C2*)b.S, b.p, local)
            FI_LINE_SWITCH(b.p.h, FI_GO)
#undef FI_GO
        } else {
            rows_fwd_body<T>((const T*)b.f, b.p.nx, b.p.nx, b.p.ny, (C2*)b.S, b.p, b.RB, local, 0);
        }
        __syncthreads();
    });
}

template <typename T>
__global__ void __launch_bounds__(512) k_b_cols_hartley(const BMember* __restrict__ M, BList L)
{
    typedef typename vec2<T>::type C2;
    batch_walk(L, [&](int m) { return true; }, [&](int m, int local) {   // the list holds the members with work
        const BMember& b = M[m];
        if (b.lines & 2) {
#define FI_GO(N) cols_hartley_lines<T, N>((C2*)b.S, (const T*)b.mA, (const T*)b.mB, b.even, b.p, local)
            FI_LINE_SWITCH(b.p.ny, FI_GO)
#undef FI_GO
        } else {
            cols_hartley_body<T>((C2*)b.S, (const T*)b.mA, (const T*)b.mB, b.even, b.p, b.CB, local, 0);
        }
        __syncthreads();
    });
}

template <typename T>
__global__ void __launch_bounds__(512) k_b_rows_inv(const BMember* __restrict__ M, BList L, int stage)
{
    typedef typename vec2<T>::type C2;
    batch_walk(L, [&](int m) { return true; }, [&](int m, int local) {
        const BMember& b = M[m];
        T scale;   // 1/(nx*ny*1.), converted on the host
        if constexpr (sizeof(T) == 4) scale = b.norm_scale_f;
        else scale = b.norm_scale;
        if (b.lines & 1) {
#define FI_GO(N) rows_inv_lines<T, N>((const C2*)b.S, b.p.ny, (T*)b.raw7[stage], b.p.nx, b.p, scale, local)
            FI_LINE_SWITCH(b.p.h, FI_GO)
#undef FI_GO
        } else {
            rows_inv_body<T>((const C2*)b.S, b.p.ny, (T*)b.raw7[stage], b.p.nx, b.p, b.RB, scale, local, 0);
        }
        __syncthreads();
    });
}

template <typename T> void batch_grids(size_t rows_smem, size_t cols_smem, int rows_threads, int cols_threads,
                                       int* g_flex, int* g_rows, int* g_cols, int* g_red)
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    auto resident = [&](auto kern, int threads, size_t smem) {
        int per = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem) != cudaSuccess || per < 1) per = 1;
        return per * nsm;
    };
    *g_flex = resident(k_b_flexure<T>, TX * TY, 0);
    *g_rows = resident(k_b_rows_fwd<T>, rows_threads, rows_smem);
    const int gi = resident(k_b_rows_inv<T>, rows_threads, rows_smem);
    if (gi < *g_rows) *g_rows = gi;
    *g_cols = resident(k_b_cols_hartley<T>, cols_threads, cols_smem);
    *g_red = batch_red_resident<T>() * nsm;
}

template <typename T> void batch_flexure(const BMember* M, BList L, int nblk, cudaStream_t s)
{
    // 256 threads: the FP64 tiles read them as TX x TY, the mixed one as 4 x 64
    k_b_flexure<T><<<nblk, dim3(TX, TY), 0, s>>>(M, L);
}
int batch_flexure_tiles64(int nx, int ny) { return ((nx + TX - 1) / TX) * ((ny + TY64 - 1) / TY64); }
int batch_flexure_tiles32(int nx, int ny)
{
    const dim3 g = tile_grid(nx, ny);
    return (int)(g.x * g.y);
}
template <typename T>
void batch_rows_fwd(const BMember* M, BList L, int nblk, int threads, size_t smem, cudaStream_t s)
{
    set_smem(k_b_rows_fwd<T>, smem);
    k_b_rows_fwd<T><<<nblk, threads, smem, s>>>(M, L);
}
template <typename T>
void batch_cols_hartley(const BMember* M, BList L, int nblk, int threads, size_t smem, cudaStream_t s)
{
    set_smem(k_b_cols_hartley<T>, smem);
    k_b_cols_hartley<T><<<nblk, threads, smem, s>>>(M, L);
}
template <typename T>
void batch_rows_inv(const BMember* M, BList L, int nblk, int threads, size_t smem, cudaStream_t s, int stage)
{
    set_smem(k_b_rows_inv<T>, smem);
    k_b_rows_inv<T><<<nblk, threads, smem, s>>>(M, L, stage);
}

// True stages: the RHS at stage state y (stage 0: x, 1-5: the stage buffer,
// 6: x2) with the mantle term at that state: mixed members over the float pair
// of the stage state (stage 0: of x) and its dxw, FP64 members over the FP64
// state.
template <typename T>
__global__ void __launch_bounds__(256) k_b_flexure_y(const BMember* __restrict__ M, BList L, int stage)
{
    batch_walk(L, [&](int m) { return true; }, [&](int m, int local) {
        const BMember& b = M[m];
        const int bx = local % b.fgx, by = local / b.fgx;
        const double* y = stage == 0 ? b.d.x : (stage == 6 ? b.d.ts_x2 : b.yst);
        if constexpr (sizeof(T) == 4) {
            const bool s0 = stage == 0;
            flexure_tile(s0 ? b.xhi : b.yhi, s0 ? b.xlo : b.ylo, nullptr, s0 ? b.xdw : b.ydw, (const float*)b.q0, b.mask,
                         (const float*)b.D, (const float*)b.inv2eta, (float*)b.f, b.p.nx, b.p.ny, b.fcf, bx, by);
        } else if (b.fc.ixm == nullptr) {
            flexure_tile64<false, TY64>(y, nullptr, b.wref, (const double*)b.q0, b.mask, (const double*)b.D,
                                  (const double*)b.inv2eta, (double*)b.f, b.p.nx, b.p.ny, b.fc64, bx, by);
        } else {
            flexure_tile64k<TY64>(y, b.wref, (const double*)b.q0, b.mask, (const double*)b.D, (const double*)b.inv2eta,
                            (double*)b.f, b.p.nx, b.p.ny, b.fc, bx, by);
        }
        __syncthreads();
    });
}
template <typename T> void batch_flexure_y(const BMember* M, BList L, int nblk, int stage, cudaStream_t s)
{
    k_b_flexure_y<T><<<nblk, dim3(TX, TY), 0, s>>>(M, L, stage);
}

template <typename T> void batch_prepare(size_t rows_smem, size_t cols_smem)
{
    set_smem(k_b_rows_fwd<T>, rows_smem);
    set_smem(k_b_rows_inv<T>, rows_smem);
    set_smem(k_b_cols_hartley<T>, cols_smem);
}

#define FI_BATCH_INST(T)                                                                                   \
    template void batch_prepare<T>(size_t, size_t);                                                        \
    template void batch_grids<T>(size_t, size_t, int, int, int*, int*, int*, int*);                        \
    template void batch_flexure<T>(const BMember*, BList, int, cudaStream_t);                    \
    template void batch_rows_fwd<T>(const BMember*, BList, int, int, size_t, cudaStream_t);      \
    template void batch_cols_hartley<T>(const BMember*, BList, int, int, size_t, cudaStream_t);  \
    template void batch_rows_inv<T>(const BMember*, BList, int, int, size_t, cudaStream_t, int);      \
    template void batch_flexure_y<T>(const BMember*, BList, int, int, cudaStream_t);
FI_BATCH_INST(double)
FI_BATCH_INST(float)

#define FI_INST(T)                                                                                            \
    template void launch_flexure<T>(const double*, const double*, const T*, const uint8_t*, const T*, const T*, \
                                    T*, int, int, const FlexCoef&, cudaStream_t, const int*, const float*,    \
                                    const float*);                                                            \
    template void launch_rows_fwd<T>(const T*, int, int, int, vec2<T>::type*, const Plan2D&, cudaStream_t,    \
                                     const int*);                                                             \
    template void launch_cols_hartley<T>(vec2<T>::type*, const T*, const T*, int, const Plan2D&, cudaStream_t, \
                                         const int*);                                                         \
    template void launch_rows_inv<T>(const vec2<T>::type*, T*, const Plan2D&, double, cudaStream_t, const int*); \
    template void launch_cols_conv<T>(vec2<T>::type*, const vec2<T>::type*, int, const int*, int, const Plan2D&, \
                                      cudaStream_t);                                                          \
    template void launch_cols_fwd<T>(vec2<T>::type*, int, const Plan2D&, cudaStream_t);                       \
    template void launch_conv_rows_inv<T>(const vec2<T>::type*, int, double*, int, int, int, double*, int, int,  \
                                          int, const Plan2D&, double, cudaStream_t);

FI_INST(double)
FI_INST(float)

}  // namespace fi
