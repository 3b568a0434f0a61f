// fi_rfft.cuh — FFT lines of 2^k and 3 2^k points, the points in registers.
//
// T = N/E threads share one line of N complex points; thread t holds the E
// points x[t + T m], m < E, before every stage, and after the last one again
// (the self-sorting Stockham order), so a caller loads from and stores to
// global memory straight from registers.  A stage of radix R (E first, the
// remainder last) does E/R butterflies per thread; between stages the line
// goes through shared memory once.
//
// Why this form: the shared-memory Stockham stages of fi_fft.cuh
// (one butterfly per thread, two shared-memory passes and a block barrier per
// stage, runtime sizes) spend most of their time on addresses, barriers and
// staging: a 2048-point column pair took three barriers and six passes
// through shared memory each way.  Here all strides are compile-time, a
// 512-point line needs two exchanges, and lines of at most 32 threads
// exchange under a warp barrier.  Measured per launch (CUDA events, their
// overhead of about 4 us included): mixed 2048^2 rows forward 31.1 -> 16.4,
// columns 60.1 -> 25.1, rows inverse 27.0 -> 14.3 us; its 4096-point
// convolution columns 225 -> 116 us; mixed 512 x 1024 10.2 -> 8.3, 16.6 ->
// 10.3, 8.8 -> 7.9 us.  FP64, bound by the FP64 pipe (2 instructions a clock
// and SM), gains the smaller operation count: 1024^2 52 -> 43, 94 -> 80,
// 50 -> 43 us, 512^2 20.9 -> 16.1, 30.9 -> 24.2, 19.1 -> 15.3 us.
// Lengths 2^k from 16 and 3 2^k from 24 on take this form (faster at each one
// measured; in the step engine shorter ones too); the others keep the
// shared-memory stages.
#pragma once

#include "fi_fft.cuh"

namespace fi {

// points per thread: 8 keeps a double-precision line at 32 data registers;
// 16 saves an exchange where a float line is long (1024 = 16 16 4 against
// 8 8 8 2).  Double lines up to 256 points have 4: a small FP64 grid has fewer
// warps than the GPU has SM quarters, and an FP64 instruction takes a quarter
// 64 clocks however little it has to do (256^2: rows 12.1 -> 8.2 us, columns
// 23 -> 14.7; 512^2 rows unchanged).  Lengths 3 2^k: 12 (radices 4, 2 and a last 3), or 24 (8, 4, 2, 3)
// where a float line is long.
__host__ __device__ constexpr int line_points(int n, bool f32)
{
    const int e = n % 3 == 0 ? (f32 && n >= 768 ? 24 : 12) : f32 ? (n >= 1024 ? 16 : 8) : n <= 256 ? 4 : 8;
    return n < e ? n : e;   // (the step engine's shortest lines: one thread)
}
template <typename T, int N> struct LineShape {
    static constexpr int E = line_points(N, sizeof(T) == 4);
    static constexpr int threads = N / E;
};
// radix of the stage that has `rem` = N / Ns left: the powers of two first
constexpr int line_radix(int E, int rem)
{
    const int most = E == 24 ? 8 : E == 12 ? 4 : E;
    const int p2 = rem % 3 == 0 ? rem / 3 : rem;
    return p2 > 1 ? (p2 < most ? p2 : most) : rem;
}

// index of point i in shared memory: one point of padding per E (or 16)
// points, so the strided stores of a stage fall in different banks
template <int E> __host__ __device__ constexpr int line_pad(int i) { return i + i / ((E & (E - 1)) == 0 ? E : 16); }
template <typename T, int N> __host__ __device__ constexpr int line_smem()
{
    // an odd multiple of two points: lines side by side start two banks apart
    return ((line_pad<LineShape<T, N>::E>(N) + 15) / 16) * 16 + 2;
}

template <typename C2> __device__ __forceinline__ C2 cscale(C2 a, decltype(C2::x) s)
{
    a.x *= s;
    a.y *= s;
    return a;
}

template <typename C2, int SIGN> __device__ __forceinline__ C2 rot_w8(C2 o)   // o exp(SIGN i pi/4) sqrt(2)
{
    C2 r;
    if (SIGN < 0) { r.x = o.x + o.y; r.y = o.y - o.x; }
    else { r.x = o.x - o.y; r.y = o.y + o.x; }
    return r;
}

template <typename T, typename C2, int SIGN> __device__ __forceinline__ void rdft4(C2& v0, C2& v1, C2& v2, C2& v3)
{
    const C2 s0 = cadd(v0, v2), d0 = csub(v0, v2);
    const C2 s1 = cadd(v1, v3), d1 = csub(v1, v3);
    v0 = cadd(s0, s1);
    v2 = csub(s0, s1);
    if (SIGN < 0) {
        v1.x = d0.x + d1.y; v1.y = d0.y - d1.x;
        v3.x = d0.x - d1.y; v3.y = d0.y + d1.x;
    } else {
        v1.x = d0.x - d1.y; v1.y = d0.y + d1.x;
        v3.x = d0.x + d1.y; v3.y = d0.y - d1.x;
    }
}

// a + s b and a - s b
template <typename T, typename C2> __device__ __forceinline__ void addsub_scaled(C2 a, C2 b, T s, C2& p, C2& m)
{
    p.x = a.x + s * b.x; p.y = a.y + s * b.y;
    m.x = a.x - s * b.x; m.y = a.y - s * b.y;
}

template <typename T, typename C2, int SIGN> __device__ __forceinline__ void rdft8(C2* v)
{
    C2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    C2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    rdft4<T, C2, SIGN>(e0, e1, e2, e3);
    rdft4<T, C2, SIGN>(o0, o1, o2, o3);
    const T h = (T)0.70710678118654752440084436210484903928;
    const C2 t1 = rot_w8<C2, SIGN>(o1);                // w8 o1 / h
    const C2 u3 = rot_w8<C2, SIGN>(o3);
    C2 t3;                                                   // w8^3 o3 / h = (SIGN i) w8 o3 / h
    if (SIGN < 0) { t3.x = u3.y; t3.y = -u3.x; }
    else { t3.x = -u3.y; t3.y = u3.x; }
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    addsub_scaled<T>(e1, t1, h, v[1], v[5]);
    if (SIGN < 0) {
        v[2].x = e2.x + o2.y; v[2].y = e2.y - o2.x;
        v[6].x = e2.x - o2.y; v[6].y = e2.y + o2.x;
    } else {
        v[2].x = e2.x - o2.y; v[2].y = e2.y + o2.x;
        v[6].x = e2.x + o2.y; v[6].y = e2.y - o2.x;
    }
    addsub_scaled<T>(e3, t3, h, v[3], v[7]);
}

template <typename T, typename C2, int SIGN> __device__ __forceinline__ void rdft16(C2* v)
{
    // 4 x 4: columns i = 0..3 (points i + 4 a), twiddle w16^(i q), rows
#pragma unroll
    for (int i = 0; i < 4; ++i) rdft4<T, C2, SIGN>(v[i], v[i + 4], v[i + 8], v[i + 12]);
    const T c1 = (T)0.92387953251128675612818318939678829, s1 = (T)0.38268343236508977172845998403039887;
    const T h = (T)0.70710678118654752440084436210484903928;
    const T sg = (T)(SIGN < 0 ? -1 : 1);
    const C2 w1 = mk2<T>(c1, sg * s1), w3 = mk2<T>(s1, sg * c1), w9 = mk2<T>(-c1, -sg * s1);
    v[5] = cmul(v[5], w1);
    v[9] = cscale(rot_w8<C2, SIGN>(v[9]), h);
    v[13] = cmul(v[13], w3);
    v[6] = cscale(rot_w8<C2, SIGN>(v[6]), h);
    v[10] = mul_mi(v[10], SIGN);
    v[14] = cscale(mul_mi(rot_w8<C2, SIGN>(v[14]), SIGN), h);
    v[7] = cmul(v[7], w3);
    v[11] = cscale(mul_mi(rot_w8<C2, SIGN>(v[11]), SIGN), h);
    v[15] = cmul(v[15], w9);
#pragma unroll
    for (int q = 0; q < 4; ++q) rdft4<T, C2, SIGN>(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    // output q + 4 p sits at v[4 q + p]
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = q + 1; p < 4; ++p) {
            const C2 t = v[4 * q + p];
            v[4 * q + p] = v[4 * p + q];
            v[4 * p + q] = t;
        }
}

template <typename T, typename C2, int SIGN> __device__ __forceinline__ void rdft3(C2& a, C2& b, C2& c)
{
    const T s1 = (T)(SIGN < 0 ? -0.86602540378443864676372317075293618 : 0.86602540378443864676372317075293618);
    const C2 s = cadd(b, c), d = csub(b, c);
    const C2 m = mk2<T>(a.x - (T)0.5 * s.x, a.y - (T)0.5 * s.y);
    a = cadd(a, s);
    b = mk2<T>(m.x - s1 * d.y, m.y + s1 * d.x);
    c = mk2<T>(m.x + s1 * d.y, m.y - s1 * d.x);
}

// Barrier among the threads of a line: 1 a warp barrier where a line never
// leaves a warp, 0 the block's, n > 1 named barrier 1 of n threads (lines that
// only those threads of a block work on).
template <int SYNC> __device__ __forceinline__ void line_sync()
{
    if (SYNC == 1) __syncwarp();
    else if (SYNC == 0) __syncthreads();
    else asm volatile("bar.sync 1, %0;" ::"n"(SYNC) : "memory");
}

// Stages from sub-transform size Ns on.  v: this thread's points t + T m;
// sm: the line's shared memory; tw: exp(-2 pi i k / N).  Every thread of the
// block calls it (threads without a line pass live = false: they only keep
// the barriers).
template <typename T, int N, int SIGN, int WARP, bool TWSH, int Ns>
__device__ __forceinline__ void line_stages(typename vec2<T>::type* v, typename vec2<T>::type* sm,
                                            const typename vec2<T>::type* __restrict__ tw, int t)
{
    typedef typename vec2<T>::type C2;
    constexpr int E = LineShape<T, N>::E, TH = LineShape<T, N>::threads;
    constexpr int R = line_radix(E, N / Ns);
    constexpr int NB = E / R;                      // butterflies per thread
    C2 u[NB][R];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int jm = (t + TH * b) & (Ns - 1);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            C2 a = v[b + NB * r];
            if (Ns > 1 && r > 0) {
                a = cmul(a, tw_load<T, C2, TWSH>(tw, jm * r * (N / (Ns * R)), SIGN));
            }
            u[b][r] = a;
        }
        if (R == 2) {
            const C2 a = u[b][0], c = u[b][1 % R];
            u[b][0] = cadd(a, c);
            u[b][1 % R] = csub(a, c);
        } else if (R == 3) {
            rdft3<T, C2, SIGN>(u[b][0], u[b][1 % R], u[b][2 % R]);
        } else if (R == 4) {
            rdft4<T, C2, SIGN>(u[b][0], u[b][1 % R], u[b][2 % R], u[b][3 % R]);
        } else if (R == 8) {
            rdft8<T, C2, SIGN>(u[b]);
        } else if (R == 16) {
            rdft16<T, C2, SIGN>(u[b]);
        }
    }
    if constexpr (Ns * R < N) {
        line_sync<WARP>();                         // the previous exchange has been read
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const int j = t + TH * b, jm = j & (Ns - 1);
#pragma unroll
            for (int r = 0; r < R; ++r) sm[line_pad<E>((j - jm) * R + jm + r * Ns)] = u[b][r];
        }
        line_sync<WARP>();
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = sm[line_pad<E>(t + TH * m)];
        line_stages<T, N, SIGN, WARP, TWSH, Ns * R>(v, sm, tw, t);
    } else {
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int r = 0; r < R; ++r) v[b + NB * r] = u[b][r];
    }
}

// TWSH: the twiddles are in shared memory
template <typename T, int N, int SIGN, int WARP, bool TWSH = false>
__device__ __forceinline__ void line_fft(typename vec2<T>::type* v, typename vec2<T>::type* sm,
                                         const typename vec2<T>::type* __restrict__ tw, int t)
{
    line_stages<T, N, SIGN, WARP, TWSH, 1>(v, sm, tw, t);
}

// ---------------------------------------------------------------------------
// Row and column passes on such lines.  `live` is false for the threads of a
// line beyond the last one.
// ---------------------------------------------------------------------------
// Real row of 2H samples -> half spectrum: z[m] = x[2m] + i x[2m+1], one
// H-point transform, then X[k] and X[H-k] from Z[k] and Z[H-k] together:
// with E = (Z[k] + conj Z[H-k])/2 and W = w^k (Z[k] - conj Z[H-k])/(2i),
// X[k] = E + W and X[H-k] = conj(E - W).
// load(i): samples i and i + 1 of the row (i even); store(k, X[k]).
template <typename T, int H, int WARP, bool TWSH = false, typename Load, typename Store>
__device__ __forceinline__ void line_rows_fwd(Load load, Store store, typename vec2<T>::type* sm,
                                              const typename vec2<T>::type* __restrict__ tw,
                                              const typename vec2<T>::type* __restrict__ rtw, int t, bool live)
{
    typedef typename vec2<T>::type C2;
    constexpr int E = LineShape<T, H>::E, TH = LineShape<T, H>::threads;
    C2 v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = live ? load(2 * (t + TH * m)) : mk2<T>((T)0, (T)0);
    line_fft<T, H, -1, WARP, TWSH>(v, sm, tw, t);
    line_sync<WARP>();
#pragma unroll
    for (int m = 0; m < E; ++m) sm[line_pad<E>(t + TH * m)] = v[m];
    line_sync<WARP>();
    if (!live) return;
    const T half = (T)0.5;
#pragma unroll
    for (int q = 0; q < E / 2; ++q) {
        const int k = t + TH * q;
        const C2 Zk = v[q];                        // point t + TH q
        if (k == 0) {
            store(0, mk2<T>(Zk.x + Zk.y, (T)0));
            store(H, mk2<T>(Zk.x - Zk.y, (T)0));
            const C2 Zm = sm[line_pad<E>(H / 2)];
            store(H / 2, mk2<T>(Zm.x, -Zm.y));
        } else {
            const C2 Zc = sm[line_pad<E>(H - k)];
            C2 Ev, O;
            Ev.x = half * (Zk.x + Zc.x);
            Ev.y = half * (Zk.y - Zc.y);
            O.x = half * (Zk.y + Zc.y);
            O.y = half * (Zc.x - Zk.x);
            const C2 W = cmul(tw_load<T, C2, TWSH>(rtw, k, -1), O);
            store(k, cadd(Ev, W));
            store(H - k, mk2<T>(Ev.x - W.x, W.y - Ev.y));
        }
    }
}

// Half spectrum of a row -> the H-point line whose inverse transform is the
// packed real row: with s = X[k] + conj X[H-k] and u = conj(w^k) (X[k] -
// conj X[H-k]), z[k] = s + i u and z[H-k] = conj(s) + i conj(u).
// X(k): the spectrum value k.
template <typename T, int H, int WARP, bool TWSH = false, typename Load>
__device__ __forceinline__ void line_rows_inv(Load X,
                                              typename vec2<T>::type* v, typename vec2<T>::type* sm,
                                              const typename vec2<T>::type* __restrict__ tw,
                                              const typename vec2<T>::type* __restrict__ rtw, int t, bool live)
{
    typedef typename vec2<T>::type C2;
    constexpr int E = LineShape<T, H>::E, TH = LineShape<T, H>::threads;
    if (live) {
#pragma unroll
        for (int q = 0; q < E / 2; ++q) {
            const int k = t + TH * q;
            const C2 A = X(k), B = X(H - k);
            if (k == 0) {
                // the imaginary parts of X[0] and X[H] do not enter a real row's transform
                const C2 M = X(H / 2);
                sm[0] = mk2<T>(A.x + B.x, A.x - B.x);
                sm[line_pad<E>(H / 2)] = mk2<T>((T)2 * M.x, (T)-2 * M.y);
            } else {
                const C2 s = mk2<T>(A.x + B.x, A.y - B.y), d = mk2<T>(A.x - B.x, A.y + B.y);
                const C2 u = cmulc(d, tw_load<T, C2, TWSH>(rtw, k, -1));
                sm[line_pad<E>(k)] = mk2<T>(s.x - u.y, s.y + u.x);
                sm[line_pad<E>(H - k)] = mk2<T>(s.x + u.y, u.x - s.y);
            }
        }
    }
    line_sync<WARP>();
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = sm[line_pad<E>(t + TH * m)];
    line_fft<T, H, +1, WARP, TWSH>(v, sm, tw, t);
}

}  // namespace fi
