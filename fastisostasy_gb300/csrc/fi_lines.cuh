// fi_lines.cuh — row and column passes over register lines, shared by the
// single-domain kernels (fi_lines.cu) and the batched ones (fi_rhs.cu).
//
// A block holds blockDim.x / T lines of T threads each (LineShape).  Rows lie
// one after the other (thread = line T + t); columns side by side (thread =
// t CB + c), so the CB columns of a spectrum row are read and written in one
// segment.
#pragma once

#include "fi_kernels.h"
#include "fi_rfft.cuh"

namespace fi {

template <typename T> struct LineTab;
template <> struct LineTab<float> {
    static __device__ __forceinline__ const float2* tw(const FftLen& L) { return L.tw32; }
    static __device__ __forceinline__ const float2* rtw(const Plan2D& p) { return p.rtw32; }
};
template <> struct LineTab<double> {
    static __device__ __forceinline__ const double2* tw(const FftLen& L) { return L.tw64; }
    static __device__ __forceinline__ const double2* rtw(const Plan2D& p) { return p.rtw64; }
};

// Threads of a line of n points, 0 where there is no such line kernel (the
// shared-memory transforms of fi_fft.cuh take every other length).
inline bool has_line(int n)
{
    const int m = n % 3 == 0 ? n / 3 : n;
    return (m & (m - 1)) == 0 && n >= (n % 3 == 0 ? 24 : 16) && n <= 4096;
}
// `points` (the transform's h x ny): double lines of 3 2^k points hold twelve
// a thread, so 152 SMs have a warp in every quarter from 233,000 points on,
// and each warp a serial chain of FP64 instructions three times as long as
// the shared-memory stages'.  Rows forward / columns / rows inverse, lines
// against stages: 96^2 16.7 / 24.9 / 16.7 against 10.7 / 18.6 / 10.5 us, 384^2
// (74,000 points) 19.9 / 31.2 / 20.8 against 18.3 / 27.0 / 16.7, 768^2 (295,000)
// 30.9 / 51.7 / 31.1 against 37.6 / 57.8 / 35.2, 768 x 384 (147,000) 21.4 /
// 32.6 / 21.7 against 24.8 / 33.9 / 23.3.
template <typename T> inline int line_threads(int n, long long points)
{
    if (sizeof(T) == 8 && n % 3 == 0 && points < 1 << 17) return 0;
    return has_line(n) ? n / line_points(n, sizeof(T) == 4) : 0;
}
// points of shared memory of one line (line_smem)
__host__ __device__ constexpr int line_room(int n, bool f32)
{
    const int e = line_points(n, f32), pad = (e & (e - 1)) == 0 ? e : 16;
    return ((n + n / pad + 15) / 16) * 16 + 2;
}
static_assert(line_room(192, true) == line_smem<float, 192>() && line_room(2048, true) == line_smem<float, 2048>() &&
                  line_room(96, false) == line_smem<double, 96>(), "one layout");
template <typename T> inline size_t line_bytes(int n)
{
    return has_line(n) ? line_room(n, sizeof(T) == 4) * 2 * sizeof(T) : 0;
}
// largest block of the line kernels: 16 points a thread or double points
// need up to 128 registers
template <typename T, int N> constexpr int line_block_max()
{
    return sizeof(T) == 8 || LineShape<T, N>::E > 8 ? 512 : 1024;
}

template <typename T, int H>
__device__ __forceinline__ void rows_fwd_lines(const T* __restrict__ in, int pitch, int width, int nrows,
                                               typename vec2<T>::type* __restrict__ S, const Plan2D& p, int bx)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int TH = LineShape<T, H>::threads;
    constexpr bool WARP = TH <= 32;
    const int line = threadIdx.x / TH, t = threadIdx.x % TH;
    const int j = bx * (int)(blockDim.x / TH) + line;
    C2* sm = reinterpret_cast<C2*>(smem_raw) + (size_t)line * line_smem<T, H>();
    const bool live = j < nrows;
    const size_t jj = live ? j : 0;
    const T* row = in + jj * pitch;
    C2* out = S + jj * p.sp;
    const bool pairs = (pitch & 1) == 0;
    line_rows_fwd<T, H, WARP>(
        [&](int i) {
            if (i + 1 < width) return pairs ? *reinterpret_cast<const C2*>(row + i) : mk2<T>(row[i], row[i + 1]);
            return mk2<T>(i < width ? row[i] : (T)0, (T)0);
        },
        [&](int k, C2 v) { out[k] = v; }, sm, LineTab<T>::tw(p.row), LineTab<T>::rtw(p), t, live);
}

template <typename T, int H>
__device__ __forceinline__ void rows_inv_lines(const typename vec2<T>::type* __restrict__ S, int nrows,
                                               T* __restrict__ out, int pitch, const Plan2D& p, T scale, int bx)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int E = LineShape<T, H>::E, TH = LineShape<T, H>::threads;
    constexpr bool WARP = TH <= 32;
    const int line = threadIdx.x / TH, t = threadIdx.x % TH;
    const int j = bx * (int)(blockDim.x / TH) + line;
    C2* sm = reinterpret_cast<C2*>(smem_raw) + (size_t)line * line_smem<T, H>();
    const bool live = j < nrows;
    const size_t jj = live ? j : 0;
    C2 v[E];
    line_rows_inv<T, H, WARP>([&](int k) { return S[jj * p.sp + k]; }, v, sm, LineTab<T>::tw(p.row), LineTab<T>::rtw(p), t, live);
    if (!live) return;
#pragma unroll
    for (int m = 0; m < E; ++m)
        *reinterpret_cast<C2*>(out + jj * pitch + 2 * (t + TH * m)) = cscale(v[m], scale);
}

template <typename T, int N>
__device__ __forceinline__ void cols_hartley_lines(typename vec2<T>::type* __restrict__ S, const T* __restrict__ mA,
                                                   const T* __restrict__ mB, int even, const Plan2D& p, int bx)
{
    typedef typename vec2<T>::type C2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int E = LineShape<T, N>::E, TH = LineShape<T, N>::threads;
    const int CB = blockDim.x / TH;
    const int c = threadIdx.x % CB, t = threadIdx.x / CB;
    const int k = bx * CB + c;
    const bool live = k <= p.h;
    C2* sm = reinterpret_cast<C2*>(smem_raw) + (size_t)c * line_smem<T, N>();
    const C2* tw = LineTab<T>::tw(p.col);
    C2 v[E];
    constexpr bool AHEAD = E <= 16;   // request the even factors with the column, registers allowing
    T fa[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
        const size_t e = (size_t)(t + TH * m) * p.sp + k;
        v[m] = live ? S[e] : mk2<T>((T)0, (T)0);
        if (AHEAD) fa[m] = (live && even) ? __ldg(mA + e) : (T)0;
    }
    line_fft<T, N, -1, false>(v, sm, tw, t);
    if (even) {
#pragma unroll
        for (int m = 0; m < E; ++m) {
            if (!AHEAD) fa[m] = live ? __ldg(mA + (size_t)(t + TH * m) * p.sp + k) : (T)0;
            v[m] = cscale(v[m], fa[m]);
        }
    } else {
        // Hartley values at (k,l), (-k,-l), (-k,l), (k,-l)
        __syncthreads();
#pragma unroll
        for (int m = 0; m < E; ++m) sm[line_pad<E>(t + TH * m)] = v[m];
        __syncthreads();
#pragma unroll
        for (int m = 0; m < E; ++m) {
            const int l = t + TH * m, lm = l == 0 ? 0 : N - l;
            const size_t ia = (size_t)l * p.sp + k, ib = (size_t)lm * p.sp + k;
            const C2 Fa = v[m], Fb = sm[line_pad<E>(lm)];
            const T H_kl = Fb.x - Fa.y, H_mkml = Fb.x + Fa.y;
            const T H_mkl = Fa.x + Fb.y, H_kml = Fa.x - Fb.y;
            const T G_kl = (live ? __ldg(mA + ia) : (T)0) * H_kl, G_kml = (live ? __ldg(mA + ib) : (T)0) * H_kml;
            const T G_mkl = (live ? __ldg(mB + ia) : (T)0) * H_mkl, G_mkml = (live ? __ldg(mB + ib) : (T)0) * H_mkml;
            v[m].x = (T)0.5 * (G_kml + G_mkl);
            v[m].y = (T)0.5 * (G_mkml - G_kl);
        }
    }
    line_fft<T, N, +1, false>(v, sm, tw, t);
    if (!live) return;
#pragma unroll
    for (int m = 0; m < E; ++m) S[(size_t)(t + TH * m) * p.sp + k] = v[m];
}

// Switch over the line lengths: FN is a macro taking the length.
#define FI_LINE_SWITCH(n, FN) \
    switch (n) {              \
    case 16: FN(16); break;   \
    case 24: if constexpr (sizeof(T) == 4) { FN(24); } break;   /* no double plan of 131,072 points has it */ \
    case 48: FN(48); break;   \
    case 96: FN(96); break;   \
    case 192: FN(192); break; \
    case 384: FN(384); break; \
    case 768: FN(768); break; \
    case 1536: FN(1536); break; \
    case 32: FN(32); break;   \
    case 64: FN(64); break;   \
    case 128: FN(128); break; \
    case 256: FN(256); break; \
    case 512: FN(512); break; \
    case 1024: FN(1024); break; \
    case 2048: FN(2048); break; \
    }

// single-domain launches (fi_lines.cu); false where the length has no line kernel
template <typename T>
bool lines_rows_fwd(const T* in, int in_pitch, int in_width, int nrows_in, typename vec2<T>::type* S, const Plan2D& p,
                    cudaStream_t s, const int* gate);
template <typename T>
bool lines_rows_inv(const typename vec2<T>::type* S, T* out, const Plan2D& p, double scale, cudaStream_t s,
                    const int* gate);
template <typename T>
bool lines_cols_hartley(typename vec2<T>::type* S, const T* mA, const T* mB, int even, const Plan2D& p, cudaStream_t s,
                        const int* gate);
template <typename T>
bool lines_cols_conv(typename vec2<T>::type* S, const typename vec2<T>::type* K, int nrows_in, int n_out,
                     const Plan2D& p, cudaStream_t s);
template <typename T>
bool lines_conv_rows_inv(const typename vec2<T>::type* S, int n_out, double* out, int nx, int ny, int i_off,
                         double* corners, int corner_col1, const Plan2D& p, double scale, cudaStream_t s);

}  // namespace fi
