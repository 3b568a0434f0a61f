// fi_lines.cu — transforms of one domain on register lines (fi_rfft.cuh):
// row and column passes of the RHS and of the convolutions for the lengths
// that have one.
#include <mutex>

#include "fi_lines.cuh"
#include "fi_shapes.h"

#ifndef FI_LINES_T   // one translation unit per precision (fi_lines64.cu)
#define FI_LINES_T float
#endif

namespace fi {

template <typename T, int H>
__global__ void __launch_bounds__(line_block_max<T, H>())
k_lines_rows_fwd(const T* __restrict__ in, int pitch, int width, int nrows, typename vec2<T>::type* __restrict__ S,
                 Plan2D p, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    rows_fwd_lines<T, H>(in, pitch, width, nrows, S, p, blockIdx.x);
}

template <typename T, int H>
__global__ void __launch_bounds__(line_block_max<T, H>())
k_lines_rows_inv(const typename vec2<T>::type* __restrict__ S, int nrows, T* __restrict__ out, int pitch, Plan2D p,
                 T scale, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    rows_inv_lines<T, H>(S, nrows, out, pitch, p, scale, blockIdx.x);
}

template <typename T, int N>
__global__ void __launch_bounds__(line_block_max<T, N>())
k_lines_cols(typename vec2<T>::type* __restrict__ S, const T* __restrict__ mA, const T* __restrict__ mB, int even,
             Plan2D p, const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;
    cols_hartley_lines<T, N>(S, mA, mB, even, p, blockIdx.x);
}

// Convolution columns: rows >= nrows_in are zero; after the multiply by the
// kernel spectrum the rows of the crop (first = nrows_in/2 - 1 on) and the
// lags 0 and 2 nrows_in - 2 are written back compacted (rows 0 .. nrows_in + 1).
template <typename T, int N>
__global__ void __launch_bounds__(line_block_max<T, N>())
k_lines_cols_conv(typename vec2<T>::type* __restrict__ S, const typename vec2<T>::type* __restrict__ K, int nrows_in,
                  Plan2D p)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int E = LineShape<T, N>::E, TH = LineShape<T, N>::threads;
    const int CB = blockDim.x / TH;
    const int c = threadIdx.x % CB, t = threadIdx.x / CB;
    const int k = blockIdx.x * CB + c;
    const bool live = k <= p.h;
    C2* sm = reinterpret_cast<C2*>(smem_raw) + (size_t)c * line_smem<T, N>();
    const C2* tw = LineTab<T>::tw(p.col);
    C2 v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
        const int l = t + TH * m;
        v[m] = (live && l < nrows_in) ? S[(size_t)l * p.sp + k] : mk2<T>((T)0, (T)0);
    }
    line_fft<T, N, -1, false>(v, sm, tw, t);
#pragma unroll
    for (int m = 0; m < E; ++m)
        if (live) v[m] = cmul(v[m], K[(size_t)(t + TH * m) * p.sp + k]);
    line_fft<T, N, +1, false>(v, sm, tw, t);
    if (!live) return;
    const int first = nrows_in / 2 - 1;
#pragma unroll
    for (int m = 0; m < E; ++m) {
        const int l = t + TH * m;
        int o = l - first;
        if (o < 0 || o >= nrows_in) o = l == 0 ? nrows_in : l == 2 * nrows_in - 2 ? nrows_in + 1 : -1;
        if (o >= 0) S[(size_t)o * p.sp + k] = v[m];
    }
}

// Inverse rows of the compacted convolution spectrum, cropped, with the
// corner values of the linear lags (rows ny and ny + 1).
template <typename T, int H>
__global__ void __launch_bounds__(line_block_max<T, H>())
k_lines_conv_rows_inv(const typename vec2<T>::type* __restrict__ S, int n_out, double* __restrict__ out, int nx,
                      int ny, int i_off, double* __restrict__ corners, int col1, Plan2D p, T scale)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int E = LineShape<T, H>::E, TH = LineShape<T, H>::threads;
    constexpr bool WARP = TH <= 32;
    const int line = threadIdx.x / TH, t = threadIdx.x % TH;
    const int j = blockIdx.x * (int)(blockDim.x / TH) + line;
    C2* sm = reinterpret_cast<C2*>(smem_raw) + (size_t)line * line_smem<T, H>();
    const bool live = j < n_out;
    const size_t jj = live ? j : 0;
    C2 v[E];
    line_rows_inv<T, H, WARP>([&](int k) { return S[jj * p.sp + k]; }, v, sm, LineTab<T>::tw(p.row), LineTab<T>::rtw(p), t, live);
    if (!live) return;
#pragma unroll
    for (int m = 0; m < E; ++m) {
        const int i2 = 2 * (t + TH * m);
        const T a[2] = {v[m].x * scale, v[m].y * scale};
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            if (j < ny) {
                const int i = i2 + b - i_off;
                if (i >= 0 && i < nx) out[jj * nx + i] = (double)a[b];
            } else {
                if (i2 + b == 0) corners[j == ny ? 0 : 2] = (double)a[b];
                if (i2 + b == col1) corners[j == ny ? 3 : 1] = (double)a[b];
            }
        }
    }
}

namespace {

// Raises a kernel's dynamic shared-memory limit once; it belongs to the
// kernel and only ever grows.
template <typename K> void line_smem_limit(K kern, size_t bytes, size_t* cur)
{
    static std::mutex mu;
    if (bytes <= 48 * 1024) return;
    std::lock_guard<std::mutex> lk(mu);
    if (bytes <= *cur) return;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess) *cur = bytes;
}

}  // namespace

// Lines per block where nothing was tuned: 128 threads for rows, 32-byte
// segments for columns; half of that in double precision, where the time of a
// small grid is the FP64 instructions of its busiest SM quarter.
template <typename T, int N, bool COL> int line_default()
{
    constexpr int th = LineShape<T, N>::threads;
    if (COL) return sizeof(T) == 4 ? 4 : 1;
    constexpr int most = sizeof(T) == 4 ? 128 : 64;
    return th >= most ? 1 : most / th;
}

#define FI_LAUNCH(kern, N, lines, count, ...)                                                          \
    do {                                                                                               \
        constexpr int th = LineShape<T, N>::threads;                                                   \
        const int nt = line_block(lines, th, line_block_max<T, N>());                                  \
        const size_t sm = (size_t)(nt / th) * line_smem<T, N>() * 2 * sizeof(T);                       \
        static size_t cur = 0;                                                                         \
        line_smem_limit(kern<T, N>, sm, &cur);                                                         \
        const int per = nt / th;                                                                       \
        kern<T, N><<<((count) + per - 1) / per, nt, sm, s>>>(__VA_ARGS__);                             \
    } while (0)

template <typename T>
bool lines_rows_fwd(const T* in, int in_pitch, int in_width, int nrows_in, typename vec2<T>::type* S, const Plan2D& p,
                    cudaStream_t s, const int* gate)
{
    if (!line_threads<T>(p.h, (long long)p.h * p.ny) || p.h > 2048) return false;
#define FI_GO(N)                                                                                     \
    FI_LAUNCH(k_lines_rows_fwd, N, (p.rb > 0 ? p.rb : line_default<T, N, false>()), nrows_in, in, in_pitch, in_width, \
              nrows_in, S, p, gate)
    FI_LINE_SWITCH(p.h, FI_GO)
#undef FI_GO
    return true;
}

template <typename T>
bool lines_rows_inv(const typename vec2<T>::type* S, T* out, const Plan2D& p, double scale, cudaStream_t s,
                    const int* gate)
{
    if (!line_threads<T>(p.h, (long long)p.h * p.ny) || p.h > 2048) return false;
#define FI_GO(N)                                                                                            \
    FI_LAUNCH(k_lines_rows_inv, N, (p.rb > 0 ? p.rb : line_default<T, N, false>()), p.ny, S, p.ny, out, p.nx, p, \
              (T)scale, gate)
    FI_LINE_SWITCH(p.h, FI_GO)
#undef FI_GO
    return true;
}

template <typename T>
bool lines_cols_hartley(typename vec2<T>::type* S, const T* mA, const T* mB, int even, const Plan2D& p, cudaStream_t s,
                        const int* gate)
{
    if (!line_threads<T>(p.ny, (long long)p.h * p.ny) || p.ny > 2048) return false;
#define FI_GO(N) \
    FI_LAUNCH(k_lines_cols, N, (p.cb > 0 ? p.cb : line_default<T, N, true>()), p.h + 1, S, mA, mB, even, p, gate)
    FI_LINE_SWITCH(p.ny, FI_GO)
#undef FI_GO
    return true;
}

template <typename T>
bool lines_cols_conv(typename vec2<T>::type* S, const typename vec2<T>::type* K, int nrows_in, int n_out,
                     const Plan2D& p, cudaStream_t s)
{
    if (!line_threads<T>(p.ny, (long long)p.h * p.ny) || n_out != nrows_in + 2) return false;
#define FI_GO(N) \
    FI_LAUNCH(k_lines_cols_conv, N, (p.cb > 0 ? p.cb : line_default<T, N, true>()), p.h + 1, S, K, nrows_in, p)
    FI_LINE_SWITCH(p.ny, FI_GO)
    if (p.ny == 4096) FI_GO(4096);
    if (p.ny == 3072) FI_GO(3072);
#undef FI_GO
    return true;
}

template <typename T>
bool lines_conv_rows_inv(const typename vec2<T>::type* S, int n_out, double* out, int nx, int ny, int i_off,
                         double* corners, int corner_col1, const Plan2D& p, double scale, cudaStream_t s)
{
    if (!line_threads<T>(p.h, (long long)p.h * p.ny) || p.h > 2048) return false;
#define FI_GO(N)                                                                                              \
    FI_LAUNCH(k_lines_conv_rows_inv, N, (p.rb > 0 ? p.rb : line_default<T, N, false>()), n_out, S, n_out, out, nx, ny, \
              i_off, corners, corner_col1, p, (T)scale)
    FI_LINE_SWITCH(p.h, FI_GO)
#undef FI_GO
    return true;
}

#define FI_LINES_INST(T)                                                                                          \
    template bool lines_rows_fwd<T>(const T*, int, int, int, vec2<T>::type*, const Plan2D&, cudaStream_t,         \
                                    const int*);                                                                  \
    template bool lines_rows_inv<T>(const vec2<T>::type*, T*, const Plan2D&, double, cudaStream_t, const int*);   \
    template bool lines_cols_hartley<T>(vec2<T>::type*, const T*, const T*, int, const Plan2D&, cudaStream_t,     \
                                        const int*);                                                              \
    template bool lines_cols_conv<T>(vec2<T>::type*, const vec2<T>::type*, int, int, const Plan2D&, cudaStream_t); \
    template bool lines_conv_rows_inv<T>(const vec2<T>::type*, int, double*, int, int, int, double*, int,         \
                                         const Plan2D&, double, cudaStream_t);
FI_LINES_INST(FI_LINES_T)

}  // namespace fi
