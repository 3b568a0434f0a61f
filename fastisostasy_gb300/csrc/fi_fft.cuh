// fi_fft.cuh — block-cooperative shared-memory Stockham FFT (any length).
//
// Self-sorting Stockham formulation: a stage of radix R over sub-transform
// size Ns takes butterfly j from x[j + r*n/R] (r < R), multiplies by the
// twiddle w^((j mod Ns) * r * n/(Ns*R)) with w = exp(-2 pi i / n), does a
// radix-R DFT and writes y[(j/Ns)*Ns*R + j mod Ns + r*Ns].  After all stages
// the result is in natural order.  All threads of the block walk over the
// butterflies of `nl` lines (line l at offset l*ls), so a block can work on
// several rows or columns at once; every stage ends in __syncthreads().
//
// Twiddles come from a per-length table tw[t] = exp(-2 pi i t / n) built on
// the host in long double; sign = -1 is the forward transform, +1 the
// unnormalised inverse.  SH = true reads the table from a shared-memory copy
// (a persistent kernel keeps it resident instead of refetching it from L2
// after the data it streams has pushed it out of L1).
#pragma once

#include "fi_common.cuh"

namespace fi {

template <typename T, typename C2, bool SH = false>
__device__ __forceinline__ C2 tw_load(const C2* __restrict__ tw, int t, int sign)
{
    C2 w = SH ? tw[t] : __ldg(tw + t);
    if (sign > 0) w.y = -w.y;
    return w;
}

// radix-2/4/8 DFTs in registers
template <typename T, typename C2>
__device__ __forceinline__ void dft2(C2& a, C2& b)
{
    C2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

// multiply by -i (forward) or +i (inverse)
template <typename C2>
__device__ __forceinline__ C2 mul_mi(C2 a, int sign)
{
    C2 r;
    if (sign < 0) { r.x = a.y; r.y = -a.x; }
    else { r.x = -a.y; r.y = a.x; }
    return r;
}

template <typename T, typename C2>
__device__ __forceinline__ void dft4(C2& v0, C2& v1, C2& v2, C2& v3, int sign)
{
    C2 s0 = cadd(v0, v2), d0 = csub(v0, v2);
    C2 s1 = cadd(v1, v3), d1 = mul_mi(csub(v1, v3), sign);
    v0 = cadd(s0, s1);
    v2 = csub(s0, s1);
    v1 = cadd(d0, d1);
    v3 = csub(d0, d1);
}

template <typename T, typename C2>
__device__ __forceinline__ void dft8(C2* v, int sign)
{
    // even / odd radix-4, then combine with w8^q
    C2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    C2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4<T, C2>(e0, e1, e2, e3, sign);
    dft4<T, C2>(o0, o1, o2, o3, sign);
    const T h = (T)0.70710678118654752440084436210484903928;
    // o1 *= w8^1, o2 *= w8^2, o3 *= w8^3 ; w8 = exp(sign * i pi / 4)
    C2 t1, t3;
    if (sign < 0) {
        t1.x = h * (o1.x + o1.y); t1.y = h * (o1.y - o1.x);     // (1 - i)/sqrt2
        t3.x = h * (o3.y - o3.x); t3.y = -h * (o3.x + o3.y);    // (-1 - i)/sqrt2
    } else {
        t1.x = h * (o1.x - o1.y); t1.y = h * (o1.y + o1.x);     // (1 + i)/sqrt2
        t3.x = -h * (o3.x + o3.y); t3.y = h * (o3.x - o3.y);    // (-1 + i)/sqrt2
    }
    C2 t2 = mul_mi(o2, sign);
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, t1); v[5] = csub(e1, t1);
    v[2] = cadd(e2, t2); v[6] = csub(e2, t2);
    v[3] = cadd(e3, t3); v[7] = csub(e3, t3);
}

template <typename T, typename C2>
__device__ __forceinline__ void dft3(C2& a, C2& b, C2& c, int sign)
{
    const T c1 = (T)-0.5;
    const T s1 = (T)(sign < 0 ? -0.86602540378443864676372317075293618 : 0.86602540378443864676372317075293618);
    C2 s = cadd(b, c), d = csub(b, c);
    C2 m;
    m.x = a.x + c1 * s.x;
    m.y = a.y + c1 * s.y;
    a = cadd(a, s);
    // +/- i*s1*d
    C2 r;
    r.x = -s1 * d.y;
    r.y = s1 * d.x;
    b = cadd(m, r);
    c = csub(m, r);
}

// cos and sin of 2 pi k / R, k = 1 .. R/2 (R = 5, 7)
template <int R> __host__ __device__ constexpr double odd_cos(int k)
{
    return R == 5 ? (k == 1 ? 0.30901699437494742410229341718281906 : -0.80901699437494742410229341718281906)
                  : (k == 1   ? 0.62348980185873353052500488400423981
                     : k == 2 ? -0.22252093395631440428890256449679476
                              : -0.90096886790241912623610231950744505);
}
template <int R> __host__ __device__ constexpr double odd_sin(int k)
{
    return R == 5 ? (k == 1 ? 0.95105651629515357211643933337938214 : 0.58778525229247312916870595463907277)
                  : (k == 1   ? 0.78183148246802980870844452667405775
                     : k == 2 ? 0.97492791218182360701813168299393122
                              : 0.43388373911755812047576833284835875);
}

// radix 5 or 7 in registers by the symmetry of the roots: with a_r = v_r +
// v_{R-r}, b_r = v_r - v_{R-r}, outputs q and R - q are (v_0 + sum a_r cos) -+
// i (sum b_r sin)
template <typename T, int R, typename C2> __device__ __forceinline__ void dft_odd(C2* v, int sign)
{
    constexpr int H = R / 2;
    C2 a[H], b[H];
    C2 sum = v[0];
#pragma unroll
    for (int r = 1; r <= H; ++r) {
        a[r - 1] = cadd(v[r], v[R - r]);
        b[r - 1] = csub(v[r], v[R - r]);
        sum = cadd(sum, a[r - 1]);
    }
    C2 out[R];
    out[0] = sum;
#pragma unroll
    for (int q = 1; q <= H; ++q) {
        C2 P = v[0], Q = mk2<T>((T)0, (T)0);
#pragma unroll
        for (int r = 1; r <= H; ++r) {
            const int e = (r * q) % R, k = e <= H ? e : R - e;
            const T c = (T)odd_cos<R>(k), w = (T)(e <= H ? odd_sin<R>(k) : -odd_sin<R>(k));
            P.x += a[r - 1].x * c;
            P.y += a[r - 1].y * c;
            Q.x += b[r - 1].x * w;
            Q.y += b[r - 1].y * w;
        }
        if (sign > 0) { Q.x = -Q.x; Q.y = -Q.y; }
        out[q] = mk2<T>(P.x + Q.y, P.y - Q.x);
        out[R - q] = mk2<T>(P.x - Q.y, P.y + Q.x);
    }
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = out[q];
}

// One line-parallel Stockham stage.  Specialised radices keep the R values
// in registers; other primes go through stage_odd.
template <typename T, int R, bool SH = false>
__device__ __forceinline__ void stage_fixed(const typename vec2<T>::type* __restrict__ src,
                                            typename vec2<T>::type* __restrict__ dst, int n, int nl,
                                            int ls, int Ns, const typename vec2<T>::type* __restrict__ tw,
                                            int sign, int tid, int nthr)
{
    typedef typename vec2<T>::type C2;
    const int NR = n / R;
    const int tstep = n / (Ns * R);
    const int items = nl * NR;
    auto butterfly = [&](int line, int j, int jm, int out0) {
        const C2* x = src + (size_t)line * ls;
        C2* y = dst + (size_t)line * ls;
        C2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            C2 a = x[j + r * NR];
            if (r > 0 && jm > 0) a = cmul(a, tw_load<T, C2, SH>(tw, jm * r * tstep, sign));
            v[r] = a;
        }
        if (R == 2) dft2<T, C2>(v[0], v[1]);
        else if (R == 4) dft4<T, C2>(v[0], v[1], v[2], v[3], sign);
        else if (R == 8) dft8<T, C2>(v, sign);
        else if (R == 3) dft3<T, C2>(v[0], v[1], v[2], sign);
        else if constexpr (R == 5 || R == 7) dft_odd<T, R>(v, sign);
#pragma unroll
        for (int r = 0; r < R; ++r) y[out0 + r * Ns] = v[r];
    };
    for (int it = tid; it < items; it += nthr) {
        const int line = it / NR;
        const int j = it - line * NR;
        const int jm = j % Ns;
        butterfly(line, j, jm, (j / Ns) * Ns * R + jm);
    }
}

// A stage of prime radix R > 7 by the symmetry of its roots: with a_r = x_r + x_{R-r}
// and b_r = x_r - x_{R-r} (twiddles applied), outputs q and R - q are
// (x_0 + sum a_r cos) -+ i (sum b_r sin), r < R/2: two real multiply-adds per
// term and output where the direct sum takes a complex multiply and an add for
// each of R terms.  (122 = 2 61 cells in FP64, where the instruction count is
// the time: rows 29.6 -> 15.7 us, columns 56 -> 25; an RK4 update of the mixed
// step engine there 890 -> 740 us.)  The sums and differences are formed once,
// in place in src, which the stage consumes.  Radix 5 and 7 keep their points
// in registers (dft_odd): through this pass with its extra barrier a 100^2
// update took 799 us against 711 of the direct sums, in registers 597.  In FP32
// radices up to 23 form the sums and differences again for each output pair,
// without that pass and barrier: an update of 66^2 (11) 899 -> 820 us, 190^2
// (19) 1232 -> 1175, 92^2 (23) 895 -> 887; 116^2 (29) would take 966 against
// 942, 122^2 (61) 1028 against 954.
constexpr int ODD_ONE_PASS = 23;
template <typename T, bool SH = false>
__device__ void stage_odd(typename vec2<T>::type* __restrict__ src, typename vec2<T>::type* __restrict__ dst, int n,
                          int nl, int ls, int R, int Ns, const typename vec2<T>::type* __restrict__ tw, int sign,
                          int tid, int nthr)
{
    typedef typename vec2<T>::type C2;
    const int NR = n / R;
    const int tstep = n / (Ns * R);
    const int step = n / R;   // table stride of the R-th roots of unity
    const int hR = R / 2, nj = nl * NR;
    if (sizeof(T) == 4 && R <= ODD_ONE_PASS) {
        // sums and differences formed by each output pair for itself
        for (int it = tid; it < nj * (hR + 1); it += nthr) {
            const int q = it / nj, jl = it - q * nj;
            const int line = jl / NR, j = jl - line * NR;
            const C2* x = src + (size_t)line * ls + j;
            const int jm = j % Ns;
            C2* y = dst + (size_t)line * ls + (j - jm) * R + jm;
            C2 P = x[0], Q = mk2<T>((T)0, (T)0);
            int e = 0;   // r q mod R
            for (int r = 1; r <= hR; ++r) {
                e += q;
                if (e >= R) e -= R;
                const C2 w = tw_load<T, C2, SH>(tw, e * step, -1);   // (cos, -sin)
                C2 a = x[r * NR], b = x[(R - r) * NR];
                if (jm > 0) {
                    a = cmul(a, tw_load<T, C2, SH>(tw, jm * r * tstep, sign));
                    b = cmul(b, tw_load<T, C2, SH>(tw, jm * (R - r) * tstep, sign));
                }
                P.x += (a.x + b.x) * w.x;
                P.y += (a.y + b.y) * w.x;
                Q.x -= (a.x - b.x) * w.y;
                Q.y -= (a.y - b.y) * w.y;
            }
            const C2 lo = mk2<T>(P.x + Q.y, P.y - Q.x), hi = mk2<T>(P.x - Q.y, P.y + Q.x);
            y[q * Ns] = sign < 0 ? lo : hi;
            if (q > 0) y[(R - q) * Ns] = sign < 0 ? hi : lo;
        }
        return;
    }
    for (int it = tid; it < nj * hR; it += nthr) {
        const int r = it / nj + 1, jl = it - (r - 1) * nj;
        const int line = jl / NR, j = jl - line * NR;
        C2* x = src + (size_t)line * ls + j;
        const int jm = j % Ns;
        C2 a = x[r * NR], b = x[(R - r) * NR];
        if (jm > 0) {
            a = cmul(a, tw_load<T, C2, SH>(tw, jm * r * tstep, sign));
            b = cmul(b, tw_load<T, C2, SH>(tw, jm * (R - r) * tstep, sign));
        }
        x[r * NR] = cadd(a, b);
        x[(R - r) * NR] = csub(a, b);
    }
    __syncthreads();
    for (int it = tid; it < nj * (hR + 1); it += nthr) {
        const int q = it / nj, jl = it - q * nj;
        const int line = jl / NR, j = jl - line * NR;
        const C2* x = src + (size_t)line * ls + j;
        C2* y = dst + (size_t)line * ls + (j / Ns) * Ns * R + j % Ns;
        C2 P = x[0], Q = mk2<T>((T)0, (T)0);
        if (q == 0) {
            for (int r = 1; r <= hR; ++r) P = cadd(P, x[r * NR]);
            y[0] = P;
            continue;
        }
        int e = 0;   // r q mod R
        for (int r = 1; r <= hR; ++r) {
            e += q;
            if (e >= R) e -= R;
            const C2 w = tw_load<T, C2, SH>(tw, e * step, -1);   // (cos, -sin)
            const C2 a = x[r * NR], b = x[(R - r) * NR];
            P.x += a.x * w.x;
            P.y += a.y * w.x;
            Q.x -= b.x * w.y;
            Q.y -= b.y * w.y;
        }
        const C2 lo = mk2<T>(P.x + Q.y, P.y - Q.x), hi = mk2<T>(P.x - Q.y, P.y + Q.x);
        y[q * Ns] = sign < 0 ? lo : hi;
        y[(R - q) * Ns] = sign < 0 ? hi : lo;
    }
}

// Runs all stages on nl lines held in buf0 (scratch buf1, same shape).
// Returns the buffer holding the result.  Must be called by every thread of
// the block (it synchronises internally); the caller synchronises before.
// ODD: with the radices other than 2, 3, 4 and 8 (a persistent kernel that
// inlines four transforms is up to 2 % faster without them).
template <typename T, bool SH = false, bool ODD = true>
__device__ typename vec2<T>::type* block_fft(typename vec2<T>::type* buf0, typename vec2<T>::type* buf1,
                                             const FftDesc& d, int nl, int ls,
                                             const typename vec2<T>::type* __restrict__ tw, int sign)
{
    typedef typename vec2<T>::type C2;
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nthr = blockDim.x * blockDim.y * blockDim.z;
    C2* src = buf0;
    C2* dst = buf1;
    int Ns = 1;
    for (int s = 0; s < d.nf; ++s) {
        const int R = d.fac[s];
        switch (R) {
        case 8: stage_fixed<T, 8, SH>(src, dst, d.n, nl, ls, Ns, tw, sign, tid, nthr); break;
        case 4: stage_fixed<T, 4, SH>(src, dst, d.n, nl, ls, Ns, tw, sign, tid, nthr); break;
        case 2: stage_fixed<T, 2, SH>(src, dst, d.n, nl, ls, Ns, tw, sign, tid, nthr); break;
        case 3: stage_fixed<T, 3, SH>(src, dst, d.n, nl, ls, Ns, tw, sign, tid, nthr); break;
        case 5:
            if constexpr (ODD) stage_fixed<T, 5, SH>(src, dst, d.n, nl, ls, Ns, tw, sign, tid, nthr);
            break;
        case 7:
            if constexpr (ODD) stage_fixed<T, 7, SH>(src, dst, d.n, nl, ls, Ns, tw, sign, tid, nthr);
            break;
        default:
            if constexpr (ODD) stage_odd<T, SH>(src, dst, d.n, nl, ls, R, Ns, tw, sign, tid, nthr);
            break;
        }
        __syncthreads();
        C2* t = src;
        src = dst;
        dst = t;
        Ns *= R;
    }
    return src;
}

}  // namespace fi
