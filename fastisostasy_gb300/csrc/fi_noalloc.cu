// fi_noalloc.cu — calc_lvelva for callers that cannot allocate device memory.
//
// Some callers may not allocate once they are running: a coupled ice-sheet /
// climate model that divides HBM among its components at start-up and treats
// any later cudaMalloc as a budget violation, or a host loop that must not
// pay the device-wide synchronisation that cudaFree implies.  fi_lvelva needs
// a handle, whose creation allocates, and allocates a temporary on each call.
//
// fi_lvelva_static runs the same FP64 viscous-rate kernels on device arrays
// owned by the caller and allocates nothing.  Its scratch (load term,
// 1/(2 eta), the stencil output, the half spectrum, the 1/(kappa R)
// multipliers, the twiddle tables and the raw inverse-transform output) lives
// in one file-scope __device__ array sized for grids of at most
// FI_STATIC_MAX_N x FI_STATIC_MAX_N cells (256 x 256: 3,219,472 bytes), which
// every GPU that loads the library holds until the process exits.  Larger or
// odd-sized grids are refused with FI_E_SIZE before any work is queued.
// Nothing in the scratch has to start at zero: every word a kernel reads was
// written earlier in the same call.
//
// Host code cannot use the array's name as a device address, so every call
// looks the address up on the current device with cudaGetSymbolAddress (a
// lookup that allocates nothing once the library's device code is loaded,
// and that stays valid after a cudaDeviceReset, which a cached pointer would
// not).  The first call on a device loads that code; make it before
// capturing any stream.  All calls on one device share the one array: calls
// whose work can overlap on the GPU (different streams, or different host
// threads) race on it and must be serialised by the caller.
//
// Spacing: dx, dy for a uniform grid, or the per-cell dx*K and dy*K fields
// of a distorted projection (src/fastisostasy.f90:152-155), which
// calc_lvelva's finite differences use cell by cell (src/lv_elva.f90:31).
#include <cmath>
#include <cstring>

#include "../../include/fi_gpu.h"
#include "fi_kernels.h"
#include "fi_state.h"

using namespace fi;

namespace {

constexpr int NA_N = FI_STATIC_MAX_N;                       // max cells per axis
constexpr int NA_CELLS = NA_N * NA_N;
constexpr int NA_SP = ((NA_N / 2 + 1) + 7) / 8 * 8;          // spectrum row pitch (complex)
constexpr size_t NA_SPEC = (size_t)NA_N * NA_SP;             // spectrum entries

// byte layout of the scratch array
constexpr size_t OFF_Q0 = 0;
constexpr size_t OFF_I2E = OFF_Q0 + (size_t)NA_CELLS * 8;
constexpr size_t OFF_F = OFF_I2E + (size_t)NA_CELLS * 8;
constexpr size_t OFF_RAW = OFF_F + (size_t)NA_CELLS * 8;
constexpr size_t OFF_S = OFF_RAW + (size_t)NA_CELLS * 8;
constexpr size_t OFF_MA = OFF_S + NA_SPEC * 16;
constexpr size_t OFF_MB = OFF_MA + NA_SPEC * 8;
constexpr size_t OFF_TWR = OFF_MB + NA_SPEC * 8;             // row FFT, length nx/2
constexpr size_t OFF_TWC = OFF_TWR + (size_t)(NA_N / 2) * 16; // column FFT, length ny
constexpr size_t OFF_RTW = OFF_TWC + (size_t)NA_N * 16;       // real-FFT twiddles, nx/2 + 1
constexpr size_t NA_BYTES = OFF_RTW + (size_t)(NA_N / 2 + 1) * 16;
static_assert(NA_BYTES == 3219472, "scratch size stated in the header comment");

static __device__ __align__(256) unsigned char g_fi_static_scratch[NA_BYTES];

// Everything a call derives from its arguments before the stencil, in one
// launch: the load term, 1/(2 eta) and the multipliers m(k, l), m(-k, l) in the
// half-spectrum layout, 1/(dx K) and 1/(dy K) of a distorted grid, and, in the
// blocks after those of the grid, the twiddles exp(-2 pi i t / n), one a
// thread (an FP64 sine is a chain of hundreds of FP64 instructions, three in a
// row took 9 us in a launch of their own).
__global__ void k_na_prepare(const double* __restrict__ cf, const uint8_t* __restrict__ mask,
                             const double* __restrict__ eta, const double* __restrict__ kappa,
                             const double* __restrict__ R, const double* __restrict__ dxm,
                             const double* __restrict__ dym, double g, int nx, int ny, int sp, double* q0, double* i2e,
                             double* mA, double* mB, double* ixm, double* iym, double2* twr, double2* twc,
                             double2* rtw)
{
    const int n = nx * ny, h = nx / 2;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    const int cells = (n + (int)blockDim.x - 1) / (int)blockDim.x * (int)blockDim.x;
    if (e >= cells) {
        int t = e - cells, len = h;
        double2* out = twr;
        if (t >= h) { t -= h; len = ny; out = twc; }
        if (out == twc && t >= ny) { t -= ny; len = nx; out = rtw; }
        if (out == rtw && t > h) return;
        double s, c;
        sincospi(-2.0 * t / len, &s, &c);
        out[t] = make_double2(c, s);
        return;
    }
    if (e >= n) return;
    q0[e] = mask[e] ? -g * cf[e] : 0.0;
    i2e[e] = 1.0 / (2.0 * eta[e]);
    if (dxm) {
        ixm[e] = 1.0 / dxm[e];
        iym[e] = 1.0 / dym[e];
    }
    const int i = e % nx, l = e / nx;
    if (i <= h) {
        const int a = l * nx + i, b = l * nx + (nx - i) % nx;
        mA[l * sp + i] = 1.0 / (kappa[a] * R[a]);
        mB[l * sp + i] = 1.0 / (kappa[b] * R[b]);
    }
}

FftDesc na_factorize(int n)
{
    FftDesc d;
    memset(&d, 0, sizeof(d));
    d.n = n;
    int m = n, e2 = 0;
    while (m % 2 == 0) { m /= 2; e2++; }
    int n8 = e2 / 3, r = e2 % 3, n4 = 0, n2 = 0;
    if (r == 1) { if (n8 > 0) { n8--; n4 = 2; } else n2 = 1; }
    else if (r == 2) n4 = 1;
    for (int i = 0; i < n8; ++i) d.fac[d.nf++] = 8;
    for (int i = 0; i < n4; ++i) d.fac[d.nf++] = 4;
    for (int i = 0; i < n2; ++i) d.fac[d.nf++] = 2;
    for (int f = 3; m > 1; f += 2)
        while (m % f == 0) { d.fac[d.nf++] = f; m /= f; }
    return d;
}

}  // namespace

extern "C" int fi_lvelva_static(const double* d_w, const double* d_canom_full, const uint8_t* d_maskactive,
                                const double* d_D_lith, const double* d_eta_eff, const double* d_kappa,
                                const double* d_R, const double* d_dx_matrix, const double* d_dy_matrix, int nx,
                                int ny, double dx, double dy, double g, double nu, double sec_per_year,
                                double* d_dwdt, void* stream)
{
    if (!d_w || !d_canom_full || !d_maskactive || !d_D_lith || !d_eta_eff || !d_kappa || !d_R || !d_dwdt)
        return FI_E_ARG;
    if (!(dx > 0.0) || !(dy > 0.0)) return FI_E_ARG;
    if ((d_dx_matrix == nullptr) != (d_dy_matrix == nullptr)) return FI_E_ARG;   // both or neither
    // grids the static scratch cannot hold are refused, not truncated
    if (nx < 4 || ny < 4 || nx > NA_N || ny > NA_N || (nx & 1) || (ny & 1)) return FI_E_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    void* sym = nullptr;
    if (cudaGetSymbolAddress(&sym, g_fi_static_scratch) != cudaSuccess || !sym) return FI_E_CUDA;
    unsigned char* const base = static_cast<unsigned char*>(sym);
    double* q0 = reinterpret_cast<double*>(base + OFF_Q0);
    double* i2e = reinterpret_cast<double*>(base + OFF_I2E);
    double* f = reinterpret_cast<double*>(base + OFF_F);
    double* raw = reinterpret_cast<double*>(base + OFF_RAW);
    double2* S = reinterpret_cast<double2*>(base + OFF_S);
    double* mA = reinterpret_cast<double*>(base + OFF_MA);
    double* mB = reinterpret_cast<double*>(base + OFF_MB);
    double2* twr = reinterpret_cast<double2*>(base + OFF_TWR);
    double2* twc = reinterpret_cast<double2*>(base + OFF_TWC);
    double2* rtw = reinterpret_cast<double2*>(base + OFF_RTW);

    Plan2D p;
    memset(&p, 0, sizeof(p));
    p.nx = nx;
    p.ny = ny;
    p.h = nx / 2;
    p.sp = ((p.h + 1) + 7) / 8 * 8;
    p.row.d = na_factorize(p.h);
    p.row.tw64 = twr;
    p.col.d = na_factorize(ny);
    p.col.tw64 = twc;
    p.rtw64 = rtw;

    // the inverse spacings live where the transforms write later: the raw
    // output and the half spectrum
    double* ixm = raw;
    double* iym = reinterpret_cast<double*>(S);
    const int nb = (nx * ny + 255) / 256, tb = (p.h + ny + p.h + 1 + 255) / 256;
    k_na_prepare<<<nb + tb, 256, 0, s>>>(d_canom_full, d_maskactive, d_eta_eff, d_kappa, d_R, d_dx_matrix, d_dy_matrix, g,
                                         nx, ny, p.sp, q0, i2e, mA, mB, ixm, iym, twr, twc, rtw);
    FlexCoef c;
    memset(&c, 0, sizeof(c));
    c.nu = nu;
    c.one_minus_nu = 1.0 - nu;
    c.inv_dx = 1.0 / dx;
    c.inv_2dx = 1.0 / (2 * dx);
    c.inv_dx2 = 1.0 / (dx * dx);
    c.inv_dy = 1.0 / dy;
    c.inv_2dy = 1.0 / (2 * dy);
    c.inv_dy2 = 1.0 / (dy * dy);
    if (d_dx_matrix) {   // else uniform spacing from dx, dy
        c.ixm = ixm;
        c.iym = iym;
    }
    launch_flexure<double>(d_w, nullptr, q0, d_maskactive, d_D_lith, i2e, f, nx, ny, c, s);
    launch_rows_fwd<double>(f, nx, nx, ny, S, p, s);
    launch_cols_hartley<double>(S, mA, mB, 0, p, s);
    const double norm = (double)(float)((long long)nx * ny);   // nx*ny*1. (default real)
    launch_rows_inv<double>(S, raw, p, 1.0 / norm, s);
    rhs_finish<double>(d_dwdt, raw, nx, ny, sec_per_year, s);
    return cudaGetLastError() == cudaSuccess ? FI_OK : FI_E_CUDA;
}
