// fi_cluster.cuh — every step of a small mixed domain's update in one launch
// of one thread-block cluster.
//
// What bounds it: latency.  A 64^2 right-hand side is 20 kflop a block, but it
// is a chain of stencil, row transform, column transform and inverse, each of
// which needs all of the domain.  The step engine (fi_engine.cu) passes the
// fields through L2 and waits at three grid barriers and some twenty block
// barriers per right-hand side; the adaptive integrators launch five kernels
// per stage.  Here the domain lives in the shared memory of 8 or 16 blocks for
// the whole update: rows are split over the blocks, the spectrum's columns
// likewise, and what another block needs travels through distributed shared
// memory between three cluster barriers per right-hand side:
//
//   1  stage state formed (its two edge rows pushed to the neighbours)
//   2  moments, f, row transforms written (column owners pull their columns)
//   3  columns transformed, multiplied, transformed back (pushed to the row
//      owners); inverse rows, the corner values pushed to every block
//
// Stage states are float pairs; an RK4 increment enters them without its
// corner mean, a constant that every difference drops and that the mantle term
// and the sum of the stages take off once the corners have arrived.  The
// arithmetic per cell is that of the step engine (RK4), of ts_fused /
// ts_commit_pair (reference stages) and of dp_stage_pair / dp_err /
// ts_commit_tpair (true stages).
//
// Measured (one RK4 update of ten steps, CUDA events, the engine's time
// first): 32^2 389 -> 186 us, 64^2 399 -> 225, 96^2 457 -> 309, 128^2 436 ->
// 281, 192^2 508 -> 452, 256^2 475 -> 540.  A 64^2 right-hand side takes 8600
// clocks, of which the three barriers 1750, the column pass 2000, the row
// passes 2500 (32 threads a block have a line to work on) and the stencil
// 2000; at 256^2 the stencil's 7300 and the column pass's 5800 of 20700 lead.
// Adaptive updates, which launched eight kernels an attempt (forty with true
// stages) inside a graph loop: coupling step with true stages at 192^2, 20
// attempts of 7 right-hand sides, 4.98 -> 2.22 ms.
//
// Every block decides alike: step control is replicated from the same
// numbers in the same order, so all threads of the cluster meet the same
// barriers.  There is no other wait.
#pragma once

#include <cooperative_groups.h>

#include <cstring>
#include <mutex>

#include "fi_cluster.h"
#include "fi_lines.cuh"
#include "fi_tableau.cuh"

namespace cg = cooperative_groups;

namespace fi {

namespace {

// rows of one block: an even number, so that no block holds a single row
__host__ __device__ inline int clu_rpc(int ny, int nc) { return 2 * ((ny + 2 * nc - 1) / (2 * nc)); }
// rows of one thread
__host__ __device__ inline int clu_run(int nx, int rpc, int nt) { return (rpc + nt / nx - 1) / (nt / nx); }
__host__ __device__ inline int clu_cpc(int h, int nc) { return (h + 1 + nc - 1) / nc; }

// Shared-memory layout (floats).  The moments, and after them the spectrum
// slices and transform scratch, share one region: the moments are dead once f
// is formed, the rest once the next stage state is.
// Everything a right-hand side reads again and again is copied in once: a
// cluster barrier's acquire drops the L1 lines, so a global operand costs an L2
// trip in every phase (64^2: 324 us an update with D, the load, 1/(2 eta) and
// the twiddles in global memory, 227 with them here).
struct CluLay {
    int xh, xl, dxw, fr, yh, yl, u, rspec, rrecv, line, twr, twc, rtw, fac, map, D, q0, ie, kk, total;
    // stages: stage outputs kept here (the adaptive pair with true stages, where they fit)
    __host__ __device__ CluLay(int nx, int h, int ny, int rpc, int cpc, int stages)
    {
        const int n = rpc * nx, halo = (rpc + 4) * nx;
        int o = 0;
        auto take = [&](int k) { const int at = o; o += (k + 3) / 4 * 4; return at; };
        xh = take(n); xl = take(n); dxw = take(n); fr = take(n);
        yh = take(halo); yl = take(halo);
        u = o;
        const int moments = 3 * ((rpc + 2) * nx);
        rspec = take(2 * (h + 1) * (rpc + 1));
        rrecv = take(2 * (h + 1) * (rpc + 1));
        line = o;
        // scratch of the transforms: register lines, or two shared-memory
        // buffers of all rows (columns) where a length has none
        const int lr = line_scratch(h, rpc), lc = line_scratch(ny, cpc);
        take(lr > lc ? lr : lc);
        if (o - u < moments) take(moments - (o - u));
        twr = take(2 * h);
        twc = take(2 * ny);
        rtw = take(2 * (h + 1));
        fac = take(cpc * ny);
        map = take(ny);
        D = take((rpc + 2) * nx);
        q0 = take(n);
        ie = take(n);
        kk = take(stages * n);
        total = o;
    }
    // lengths whose line is at most a warp wide
    __host__ __device__ static bool line_ok(int n)
    {
        const int m = n % 3 == 0 ? n / 3 : n;
        return (m & (m - 1)) == 0 && n >= (n % 3 == 0 ? 24 : 16) && n <= (n % 3 == 0 ? 384 : 256);
    }
    __host__ __device__ static int line_scratch(int n, int lines)
    {
        if (!line_ok(n)) return 2 * 2 * lines * n;
        // a whole warp works, so the lines are rounded up to its number
        const int lpw = 32 / (n / line_points(n, true));
        return 2 * line_room(n, true) * ((lines + lpw - 1) / lpw * lpw);
    }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// address of the same shared-memory location in block `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t a, int rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ float2 ld_dsm2(uint32_t a)
{
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ void st_dsm2(uint32_t a, float2 v)
{
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void st_dsm(uint32_t a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_dsm(uint32_t a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// (row, column) walk of the block's threads over a strip of width w
struct CluWalk {
    int r0, i0, dr, di, w;
    __device__ __forceinline__ CluWalk(int width, int tid, int nt)
    {
        w = width;
        r0 = tid / width;
        i0 = tid - r0 * width;
        dr = nt / width;
        di = nt - dr * width;
    }
    __device__ __forceinline__ void next(int& r, int& i) const
    {
        i += di;
        r += dr;
        if (i >= w) {
            i -= w;
            ++r;
        }
    }
};

// hi + lo = (xh + xl) + inc by an FP32 two-sum
__device__ __forceinline__ void pair_add(float xh, float xl, float inc, float& hi, float& lo)
{
    const float sm = xh + inc, bb = sm - xh;
    const float er = (xh - (sm - bb)) + (inc - bb);
    const float l2 = xl + er;
    hi = sm + l2;
    lo = l2 - (hi - sm);
}

// Shared state of a block outside the dynamic arrays.
struct CluShared {
    alignas(16) float corner[4];        // raw(1,1), raw(nx,ny), raw(1,ny), raw(nx,1) of the last right-hand side
    // the blocks' partial reductions, of this attempt and of the one before,
    // and the warps' (threads / 32 of them): two maxima and a sum, which takes
    // the place of two floats where it is in FP64 (sum64)
    float part[2][16][4];
    float red[16][4];
    double t, dt, tf, h;
    double tol, err;
    long long n_acc, n_rej, n_att;
    int go, accepted, status, iter, have;
    double cx;
    float cm[8];            // corner means of the stage outputs
    float f[24];            // float scalars of the current stage or attempt
};

__device__ __forceinline__ double* sum64(float* slot) { return reinterpret_cast<double*>(slot + 2); }

// What the transform phases need, the same for all threads of a block.
struct CluCtx {
    CluLay L;
    int nx, ny, h, rpc, cpc, even, rank, nr;
    const float *mAT, *mBT;
    float scale;
    FftDesc row, col;
};
__shared__ __align__(16) unsigned char s_ctx[sizeof(CluCtx)];
extern __shared__ __align__(16) float smf[];

// The transform phases.  (As functions called by every kernel they compiled
// faster and ran slower, 256^2 530 -> 747 us an update: the call spills what the
// stencil keeps.)
struct CluFft {
    const CluCtx& c;
    const uint32_t* map;    // grid row -> cluster address of its row-spectrum slot, k = 0
    const float2 *twr, *twc, *rtw;
    __device__ CluFft() : c(*reinterpret_cast<const CluCtx*>(s_ctx))
    {
        map = reinterpret_cast<const uint32_t*>(smf + c.L.map);
        twr = reinterpret_cast<const float2*>(smf + c.L.twr);
        twc = reinterpret_cast<const float2*>(smf + c.L.twc);
        rtw = reinterpret_cast<const float2*>(smf + c.L.rtw);
    }

    template <int H> __device__ __forceinline__ void rows_fwd_line() const
    {
        constexpr int TH = LineShape<float, H>::threads, LPW = 32 / TH;
        const int wl = (threadIdx.x >> 5) * LPW + (threadIdx.x & 31) / TH, t = threadIdx.x % TH;
        float2* rs = reinterpret_cast<float2*>(smf + c.L.rspec);
        const int rp = c.rpc + 1, nx = c.nx;
        const float* fr = smf + c.L.fr;
        for (int line = wl; line - wl % LPW < c.nr; line += ((int)blockDim.x / 32) * LPW) {
            const bool live = line < c.nr;
            float2* b = reinterpret_cast<float2*>(smf + c.L.line) + (size_t)line * line_smem<float, H>();
            line_rows_fwd<float, H, true, true>(
                [&](int i) { return *reinterpret_cast<const float2*>(fr + line * nx + i); },
                [&](int k, float2 v) { rs[k * rp + line] = v; }, b, twr, rtw, t, live);
        }
    }

    __device__ __forceinline__ void rows_fwd_any() const
    {
        const int h = c.h, rp = c.rpc + 1;
        float2* b0 = reinterpret_cast<float2*>(smf + c.L.line);
        float2* b1 = b0 + c.rpc * h;
        const float2* f2 = reinterpret_cast<const float2*>(smf + c.L.fr);   // rows packed as complex pairs
        for (int e = threadIdx.x; e < c.nr * h; e += (int)blockDim.x) b0[e] = f2[e];
        __syncthreads();
        const float2* Z = block_fft<float, true>(b0, b1, c.row, c.nr, h, twr, -1);
        float2* rs = reinterpret_cast<float2*>(smf + c.L.rspec);
        const CluWalk wk(h + 1, threadIdx.x, (int)blockDim.x);
        for (int r = wk.r0, k = wk.i0; r < c.nr; wk.next(r, k)) {
            const float2 Zk = Z[r * h + (k == h ? 0 : k)], Zc = Z[r * h + (k == 0 ? 0 : h - k)];
            const float2 E = make_float2(0.5f * (Zk.x + Zc.x), 0.5f * (Zk.y - Zc.y));
            const float2 O = make_float2(0.5f * (Zk.y + Zc.y), -0.5f * (Zk.x - Zc.x));
            rs[k * rp + r] = cadd(E, cmul(rtw[k], O));
        }
    }

    // spectrum value (k, l): read from, and returned to, the owner of row l
    __device__ __forceinline__ float2 pull(int k, int l) const { return ld_dsm2(map[l] + 8u * k * (c.rpc + 1)); }
    __device__ __forceinline__ void push(int k, int l, float2 v) const
    {
        st_dsm2(map[l] + 8u * k * (c.rpc + 1) + 4u * (c.L.rrecv - c.L.rspec), v);
    }

    template <int N> __device__ __forceinline__ void cols_line(int k0, int nk) const
    {
        constexpr int E = LineShape<float, N>::E, TH = LineShape<float, N>::threads, LPW = 32 / TH;
        const int wl = (threadIdx.x >> 5) * LPW + (threadIdx.x & 31) / TH, t = threadIdx.x % TH;
        for (int cl = wl; cl - wl % LPW < nk; cl += ((int)blockDim.x / 32) * LPW) {
            const bool live = cl < nk;
            const int k = k0 + cl;
            float2* b = reinterpret_cast<float2*>(smf + c.L.line) + (size_t)cl * line_smem<float, N>();
            float2 v[E];
            const float* fa = smf + c.L.fac + (live ? cl : 0) * N;
#pragma unroll
            for (int m = 0; m < E; ++m) v[m] = live ? pull(k, t + TH * m) : make_float2(0.f, 0.f);
            line_fft<float, N, -1, true, true>(v, b, twc, t);
            if (c.even) {
#pragma unroll
                for (int m = 0; m < E; ++m) v[m] = cscale(v[m], fa[t + TH * m]);
            } else {
                __syncwarp();
#pragma unroll
                for (int m = 0; m < E; ++m) b[line_pad<E>(t + TH * m)] = v[m];
                __syncwarp();
#pragma unroll
                for (int m = 0; m < E; ++m) {
                    const int l = t + TH * m, lm = l == 0 ? 0 : N - l;
                    v[m] = live ? hartley(v[m], b[line_pad<E>(lm)], k, l, lm) : v[m];
                }
            }
            line_fft<float, N, +1, true, true>(v, b, twc, t);
            if (live) {
#pragma unroll
                for (int m = 0; m < E; ++m) push(k, t + TH * m, v[m]);
            }
        }
    }

    // DFT value at (k, l) of DHT^-1 (m H) from those of the DFT at l and -l
    __device__ __forceinline__ float2 hartley(float2 Fa, float2 Fb, int k, int l, int lm) const
    {
        const int ny = c.ny;
        const size_t ia = (size_t)k * ny + l, ib = (size_t)k * ny + lm;
        const float H_kl = Fb.x - Fa.y, H_mkml = Fb.x + Fa.y, H_mkl = Fa.x + Fb.y, H_kml = Fa.x - Fb.y;
        const float G_kl = __ldg(c.mAT + ia) * H_kl, G_kml = __ldg(c.mAT + ib) * H_kml;
        const float G_mkl = __ldg(c.mBT + ia) * H_mkl, G_mkml = __ldg(c.mBT + ib) * H_mkml;
        return make_float2(0.5f * (G_kml + G_mkl), 0.5f * (G_mkml - G_kl));
    }

    __device__ __forceinline__ void cols_any(int k0, int nk) const
    {
        const int ny = c.ny;
        float2* b0 = reinterpret_cast<float2*>(smf + c.L.line);
        float2* b1 = b0 + c.cpc * ny;
        const CluWalk wk(ny, threadIdx.x, (int)blockDim.x);
        for (int cl = wk.r0, l = wk.i0; cl < nk; wk.next(cl, l)) b0[cl * ny + l] = pull(k0 + cl, l);
        __syncthreads();
        float2* F = block_fft<float, true>(b0, b1, c.col, nk, ny, twc, -1);
        float2* o = F == b0 ? b1 : b0;
        for (int cl = wk.r0, l = wk.i0; cl < nk; wk.next(cl, l)) {
            const int lm = l == 0 ? 0 : ny - l;
            const float2 Fa = F[cl * ny + l];
            o[cl * ny + l] = c.even ? cscale(Fa, smf[c.L.fac + cl * ny + l])
                                   : hartley(Fa, F[cl * ny + lm], k0 + cl, l, lm);
        }
        __syncthreads();
        const float2* q = block_fft<float, true>(o, F, c.col, nk, ny, twc, +1);
        for (int cl = wk.r0, l = wk.i0; cl < nk; wk.next(cl, l)) push(k0 + cl, l, q[cl * ny + l]);
    }

    template <int H> __device__ __forceinline__ void rows_inv_line() const
    {
        constexpr int E = LineShape<float, H>::E, TH = LineShape<float, H>::threads, LPW = 32 / TH;
        const int wl = (threadIdx.x >> 5) * LPW + (threadIdx.x & 31) / TH, t = threadIdx.x % TH;
        const float2* rr = reinterpret_cast<const float2*>(smf + c.L.rrecv);
        const int rp = c.rpc + 1, nx = c.nx;
        float* fr = smf + c.L.fr;
        for (int line = wl; line - wl % LPW < c.nr; line += ((int)blockDim.x / 32) * LPW) {
            const bool live = line < c.nr;
            float2* b = reinterpret_cast<float2*>(smf + c.L.line) + (size_t)line * line_smem<float, H>();
            float2 v[E];
            __syncwarp();
            line_rows_inv<float, H, true, true>([&](int k) { return rr[k * rp + line]; }, v, b, twr, rtw, t, live);
            if (live) {
#pragma unroll
                for (int m = 0; m < E; ++m)
                    *reinterpret_cast<float2*>(fr + line * nx + 2 * (t + TH * m)) = cscale(v[m], c.scale);
            }
        }
    }

    __device__ __forceinline__ void rows_inv_any() const
    {
        const int h = c.h, rp = c.rpc + 1;
        float2* b0 = reinterpret_cast<float2*>(smf + c.L.line);
        float2* b1 = b0 + c.rpc * h;
        const float2* rr = reinterpret_cast<const float2*>(smf + c.L.rrecv);
        const CluWalk wk(h, threadIdx.x, (int)blockDim.x);
        for (int r = wk.r0, k = wk.i0; r < c.nr; wk.next(r, k)) {
            const float2 A = rr[k * rp + r], Bv = rr[(h - k) * rp + r];
            const float2 s = make_float2(A.x + Bv.x, A.y - Bv.y), d = make_float2(A.x - Bv.x, A.y + Bv.y);
            const float2 u = cmulc(d, rtw[k]);
            b0[r * h + k] = make_float2(s.x - u.y, s.y + u.x);
        }
        __syncthreads();
        const float2* z = block_fft<float, true>(b0, b1, c.row, c.nr, h, twr, +1);
        float2* f2 = reinterpret_cast<float2*>(smf + c.L.fr);
        for (int e = threadIdx.x; e < c.nr * h; e += (int)blockDim.x) f2[e] = cscale(z[e], c.scale);
    }
};

__device__ __forceinline__ void clu_rows_fwd()
{
    const CluFft f;
    switch (f.c.h) {
    case 16: f.rows_fwd_line<16>(); break;
    case 24: f.rows_fwd_line<24>(); break;
    case 32: f.rows_fwd_line<32>(); break;
    case 48: f.rows_fwd_line<48>(); break;
    case 64: f.rows_fwd_line<64>(); break;
    case 96: f.rows_fwd_line<96>(); break;
    case 128: f.rows_fwd_line<128>(); break;
    case 192: f.rows_fwd_line<192>(); break;
    case 256: f.rows_fwd_line<256>(); break;
    default: f.rows_fwd_any(); break;
    }
}
__device__ __forceinline__ void clu_cols()
{
    const CluFft f;
    const int k0 = f.c.rank * f.c.cpc;
    int nk = f.c.h + 1 - k0;
    nk = nk < 0 ? 0 : nk < f.c.cpc ? nk : f.c.cpc;
    switch (f.c.ny) {
    case 16: f.cols_line<16>(k0, nk); break;
    case 24: f.cols_line<24>(k0, nk); break;
    case 32: f.cols_line<32>(k0, nk); break;
    case 48: f.cols_line<48>(k0, nk); break;
    case 64: f.cols_line<64>(k0, nk); break;
    case 96: f.cols_line<96>(k0, nk); break;
    case 128: f.cols_line<128>(k0, nk); break;
    case 192: f.cols_line<192>(k0, nk); break;
    case 256: f.cols_line<256>(k0, nk); break;
    case 384: f.cols_line<384>(k0, nk); break;
    default: f.cols_any(k0, nk); break;
    }
}
__device__ __forceinline__ void clu_rows_inv()
{
    const CluFft f;
    switch (f.c.h) {
    case 16: f.rows_inv_line<16>(); break;
    case 24: f.rows_inv_line<24>(); break;
    case 32: f.rows_inv_line<32>(); break;
    case 48: f.rows_inv_line<48>(); break;
    case 64: f.rows_inv_line<64>(); break;
    case 96: f.rows_inv_line<96>(); break;
    case 128: f.rows_inv_line<128>(); break;
    case 192: f.rows_inv_line<192>(); break;
    case 256: f.rows_inv_line<256>(); break;
    default: f.rows_inv_any(); break;
    }
}

// NT threads; thread (i, group) owns column i of a run of at most CH rows, the
// same cells in every phase.
template <int NT, int CH> struct Clu {
    const ClusterArgs& g;
    float* sm;
    const CluLay& L;
    CluShared& S;
    int rank, nc, nr, r0;
    int i, grp, ngrp;       // column, row group, number of groups (grp >= ngrp: no cells)
    int ra, rb;             // own rows in the block
    uint32_t active;        // mask bits of the own cells

    __device__ Clu(const ClusterArgs& a, float* s, const CluLay& l, CluShared& sh, int rk, int n)
        : g(a), sm(s), L(l), S(sh), rank(rk), nc(n)
    {

        r0 = rank * g.rpc;
        nr = g.p.ny - r0 < g.rpc ? g.p.ny - r0 : g.rpc;
        if (nr < 0) nr = 0;
        ngrp = NT / a.p.nx;
        grp = (int)threadIdx.x / a.p.nx;
        i = (int)threadIdx.x - grp * a.p.nx;
        const int run = (a.rpc + ngrp - 1) / ngrp;
        ra = grp < ngrp ? grp * run : 0;
        rb = grp < ngrp ? (ra + run < nr ? ra + run : nr) : 0;
        active = 0;
#pragma unroll
        for (int q = 0; q < CH; ++q)
            if (ra + q < rb && a.mask[(size_t)(r0 + ra + q) * a.p.nx + i]) active |= 1u << q;
    }

    // tables and fixed fields into shared memory
    __device__ __forceinline__ void copy_fixed() const
    {
        const int h = g.p.h, nx = g.p.nx, ny = g.p.ny;
        if (threadIdx.x == 0) {
            CluCtx& c = *reinterpret_cast<CluCtx*>(s_ctx);
            c.L = L;
            c.nx = nx; c.ny = ny; c.h = h;
            c.rpc = g.rpc; c.cpc = g.cpc; c.even = g.even;
            c.rank = rank; c.nr = nr;
            c.mAT = g.mAT; c.mBT = g.mBT;
            c.scale = g.norm_scale_f;
            c.row = g.p.row.d; c.col = g.p.col.d;
        }
        uint32_t* mm = reinterpret_cast<uint32_t*>(sm + L.map);
        for (int l = threadIdx.x; l < ny; l += NT) mm[l] = map_rank(smem_u32(sm + L.rspec) + 8u * (l % g.rpc), l / g.rpc);
        auto table = [&](int at, const float2* src, int n) {
            for (int e = threadIdx.x; e < n; e += NT) reinterpret_cast<float2*>(sm + at)[e] = src[e];
        };
        table(L.twr, g.p.row.tw32, h);
        table(L.twc, g.p.col.tw32, ny);
        table(L.rtw, g.p.rtw32, h + 1);
        const int k0 = rank * g.cpc;
        for (int e = threadIdx.x; e < g.cpc * ny && g.even; e += NT)
            sm[L.fac + e] = k0 + e / ny <= h ? g.mAT[(size_t)k0 * ny + e] : 0.f;
        for (int e = threadIdx.x; e < (nr + 2) * nx && nr > 0; e += NT) {
            const ptrdiff_t c = (ptrdiff_t)(r0 - 1) * nx + e;
            sm[L.D + e] = c >= 0 && c < (ptrdiff_t)nx * ny ? g.D[c] : 0.f;
        }
        for (int e = threadIdx.x; e < nr * nx; e += NT) {
            const size_t c = (size_t)r0 * nx + e;
            sm[L.q0 + e] = g.q0[c];
            sm[L.ie + e] = g.inv2eta[c];
        }
    }

    // own cells: fn(row in block, cell index in block, number among the own cells)
    template <typename F> __device__ __forceinline__ void cells(F fn) const
    {
#pragma unroll
        for (int q = 0; q < CH; ++q)
            if (ra + q < rb) fn(ra + q, (ra + q) * g.p.nx + i, q);
    }

    // the stage state of a cell, into the block's rows and the neighbours' halo
    __device__ __forceinline__ void put_y(int r, float hi, float lo) const
    {
        const int nx = g.p.nx;
        float* yh = sm + L.yh;
        float* yl = sm + L.yl;
        const int o = (r + 2) * nx + i;
        yh[o] = hi;
        yl[o] = lo;
        if (r < 2 && rank > 0) {
            const int q = (g.rpc + 2 + r) * nx + i;
            st_dsm(map_rank(smem_u32(yh + q), rank - 1), hi);
            st_dsm(map_rank(smem_u32(yl + q), rank - 1), lo);
        }
        if (r >= nr - 2 && r0 + nr < g.p.ny) {
            const int q = (r - (nr - 2)) * nx + i;
            st_dsm(map_rank(smem_u32(yh + q), rank + 1), hi);
            st_dsm(map_rank(smem_u32(yl + q), rank + 1), lo);
        }
    }

    // corner mean of the last right-hand side (every block after a barrier)
    __device__ __forceinline__ double corner() const
    {
        return corner_mean((double)S.corner[0], (double)S.corner[1], (double)S.corner[2], (double)S.corner[3]);
    }

    // One right-hand side at the stage state in yh/yl, its edge rows already
    // pushed.  mantle(e, q): the state part of the mantle term at a cell
    // (true stages), read before fr is overwritten.  one_thread: run by the
    // last thread when the corners of the previous right-hand side have
    // arrived, before any mantle() (its FP64 latency stays off the warps that
    // have cells everywhere).  Leaves raw in fr and its corners on their way to every
    // block (valid after the next barrier).
    template <bool MANTLE, typename One, typename Mantle>
    __device__ __forceinline__ void rhs(One one_thread, Mantle mantle) const
    {
        const int nx = g.p.nx, ny = g.p.ny;
        cluster_barrier();                                  // 1: halo rows and corners have arrived
        if (threadIdx.x == NT - 1) one_thread();
        const float* yh = sm + L.yh;
        const float* yl = sm + L.yl;
        const float* Dp = sm + L.D;
        const int mrows = (g.rpc + 2) * nx;
        float* Mxx = sm + L.u;
        float* Myy = Mxx + mrows;
        float* Mxy = Myy + mrows;
        const float nu = g.fcf.nu, omn = g.fcf.one_minus_nu;
        const bool left = i == 0, right = i == nx - 1;
        const int ic = left ? 1 : right ? nx - 2 : i;       // centre of the second differences in x
        const int il = left ? 0 : i - 1, ir = right ? nx - 1 : i + 1;
        const float cx = left || right ? g.fcf.inv_dx : g.fcf.inv_2dx;
        // moments of rows r0 - 1 .. r0 + nr (row m of the buffers is grid row
        // r0 - 1 + m), walking down the column with three rows of it in
        // registers; the one-sided second differences are the central ones
        // one cell inside
        if (grp < ngrp && nr > 0) {
            const int run = (nr + 2 + ngrp - 1) / ngrp;
            int m0 = grp * run, m1 = m0 + run < nr + 2 ? m0 + run : nr + 2;
            if (r0 == 0 && m0 == 0) m0 = 1;
            if (r0 + nr == ny && m1 == nr + 2) m1 = nr + 1;
            float w0, w1, w2, x1, x2, h0, h1, h2, l0, l1, l2;
            // column differences and value of grid row j (rows beyond the grid are not used)
            auto row = [&](int j, float& w, float& x, float& h, float& l) {
                const int o = ((j < 0 ? 0 : j < ny ? j : ny - 1) - r0 + 2) * nx + ic;
                const float ha = yh[o - 1], hb = yh[o], hc = yh[o + 1], la = yl[o - 1], lb = yl[o], lc = yl[o + 1];
                const float dA = (hb - ha) + (lb - la), dB = (hc - hb) + (lc - lb);
                x = (dB - dA) * g.fcf.inv_dx2;
                w = (left ? dA : right ? dB : dA + dB) * cx;
                h = left ? ha : right ? hc : hb;
                l = left ? la : right ? lc : lb;
            };
            if (m0 < m1) {
                row(r0 + m0 - 2, w0, x1, h0, l0);
                row(r0 + m0 - 1, w1, x1, h1, l1);
            }
            for (int m = m0; m < m1; ++m) {
                const int j = r0 - 1 + m, o = m * nx + i;
                row(j + 1, w2, x2, h2, l2);
                float wxy, wyy;
                if (j == 0 || j == ny - 1) {
                    wxy = (j == 0 ? w2 - w1 : w1 - w0) * g.fcf.inv_dy;
                    const int c = ((j == 0 ? 1 : ny - 2) - r0 + 2) * nx + i;
                    wyy = (((yh[c + nx] - yh[c]) + (yl[c + nx] - yl[c])) -
                           ((yh[c] - yh[c - nx]) + (yl[c] - yl[c - nx]))) * g.fcf.inv_dy2;
                } else {
                    wxy = (w2 - w0) * g.fcf.inv_2dy;
                    wyy = (((h2 - h1) + (l2 - l1)) - ((h1 - h0) + (l1 - l0))) * g.fcf.inv_dy2;
                }
                const float Dl = Dp[o];
                Mxx[o] = -Dl * (x1 + nu * wyy);
                Myy[o] = -Dl * (wyy + nu * x1);
                Mxy[o] = (-Dl * omn) * wxy;
                w0 = w1; w1 = w2; x1 = x2;
                h0 = h1; h1 = h2; l0 = l1; l1 = l2;
            }
        }
        __syncthreads();
        float* fr = sm + L.fr;
        {
            const float* q0p = sm + L.q0;
            const float* iep = sm + L.ie;
            // row r of the block is row r + 1 of the moment buffers
            float q0 = 0.f, q1 = 0.f, y0 = 0.f, y1 = 0.f;
            if (ra < rb) {
                const int o = ra * nx;
                q0 = (Mxy[o + ir] - Mxy[o + il]) * cx;
                q1 = (Mxy[o + nx + ir] - Mxy[o + nx + il]) * cx;
                y0 = Myy[o + i];
                y1 = Myy[o + nx + i];
            }
            cells([&](int r, int e, int q) {
                const int j = r0 + r, o = (r + 1) * nx;
                const float q2 = (Mxy[o + nx + ir] - Mxy[o + nx + il]) * cx, y2 = Myy[o + nx + i];
                const float mx_xx = ((Mxx[o + ic + 1] - 2.f * Mxx[o + ic]) + Mxx[o + ic - 1]) * g.fcf.inv_dx2;
                const float load = q0p[e], ie = iep[e];
                const float man = MANTLE ? mantle(e, q) : 0.f;
                float mxy, my_yy;
                if (j == 0 || j == ny - 1) {
                    mxy = (j == 0 ? q2 - q1 : q1 - q0) * g.fcf.inv_dy;
                    const int c = ((j == 0 ? 1 : ny - 2) - r0 + 1) * nx + i;
                    my_yy = ((Myy[c + nx] - 2.f * Myy[c]) + Myy[c - nx]) * g.fcf.inv_dy2;
                } else {
                    mxy = (q2 - q0) * g.fcf.inv_2dy;
                    my_yy = ((y2 - 2.f * y1) + y0) * g.fcf.inv_dy2;
                }
                const float p = (active >> q & 1u) ? load + g.fcf.coef_mantle * man : 0.f;
                fr[e] = (((p + mx_xx) + 2.f * mxy) + my_yy) * ie;
                q0 = q1; q1 = q2; y0 = y1; y1 = y2;
            });
        }
        __syncthreads();
        clu_rows_fwd();
        cluster_barrier();                                  // 2: every row's spectrum is in place
        clu_cols();
        cluster_barrier();                                  // 3: this block's rows have all their columns
        clu_rows_inv();
        __syncthreads();
        // corner values to every block
        if ((int)threadIdx.x < nc && nr > 0) {
            const int b = threadIdx.x;
            if (r0 == 0) {
                st_dsm(map_rank(smem_u32(&S.corner[0]), b), fr[0]);
                st_dsm(map_rank(smem_u32(&S.corner[3]), b), fr[nx - 1]);
            }
            if (r0 + nr == ny) {
                st_dsm(map_rank(smem_u32(&S.corner[1]), b), fr[nr * nx - 1]);
                st_dsm(map_rank(smem_u32(&S.corner[2]), b), fr[(nr - 1) * nx]);
            }
        }
    }

    // max, max, sum of per-thread values over the cluster; every block gets
    // the same totals (one barrier).  A rejected attempt has no other barrier,
    // so consecutive reductions use the two halves of S.part in turn.  The sum
    // is of floats within a block, as ts_fused_body takes it, or with SUM64 of
    // the threads' values in FP64, as ts_err_body does.  Maxima stay floats to
    // the end: one FP64 instruction after another on thread 0 (64 clocks each)
    // they took 3 us of an attempt (an update of 20 attempts: true stages at
    // 192^2 1763 -> 1710 us with the FP64 sum, 1786 without this; reference
    // stages at 128^2 309 -> 254).
    template <bool SUM64>
    __device__ __forceinline__ void reduce(float m1, float m2, float s2, int parity, double* tot) const
    {
        const unsigned FULL = 0xffffffffu;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            m1 = fmaxf(m1, __shfl_xor_sync(FULL, m1, o));
            m2 = fmaxf(m2, __shfl_xor_sync(FULL, m2, o));
        }
        const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if constexpr (SUM64) {
            double d2 = (double)s2;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d2 += __shfl_xor_sync(FULL, d2, o);
            if (lane == 0) *sum64(S.red[wid]) = d2;
        } else {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(FULL, s2, o);
            if (lane == 0) S.red[wid][2] = s2;
        }
        if (lane == 0) {
            S.red[wid][0] = m1;
            S.red[wid][1] = m2;
        }
        __syncthreads();
        if constexpr (SUM64) {
            if (wid == 0) {
                double d2 = lane < NT / 32 ? *sum64(S.red[lane]) : 0.0;
#pragma unroll
                for (int o = NT / 64; o > 0; o >>= 1) d2 += __shfl_down_sync(FULL, d2, o);
                d2 = __shfl_sync(FULL, d2, 0);
                if (lane < nc) st_dsm(map_rank(smem_u32(sum64(S.part[parity][rank])), lane), d2);
            }
        }
        if ((int)threadIdx.x < nc) {
            float a = 0.f, b = 0.f, c = 0.f;
            for (int q = 0; q < NT / 32; ++q) {
                a = fmaxf(a, S.red[q][0]);
                b = fmaxf(b, S.red[q][1]);
                if (!SUM64) c += S.red[q][2];
            }
            const int to = threadIdx.x;
            st_dsm(map_rank(smem_u32(&S.part[parity][rank][0]), to), a);
            st_dsm(map_rank(smem_u32(&S.part[parity][rank][1]), to), b);
            if (!SUM64) st_dsm(map_rank(smem_u32(&S.part[parity][rank][2]), to), c);
        }
        cluster_barrier();
        if (threadIdx.x == 0) {
            float a = 0.f, b = 0.f;
            double c = 0.0;
            for (int q = 0; q < nc; ++q) {
                a = fmaxf(a, S.part[parity][q][0]);
                b = fmaxf(b, S.part[parity][q][1]);
                c += SUM64 ? *sum64(S.part[parity][q]) : (double)S.part[parity][q][2];
            }
            tot[0] = (double)a;
            tot[1] = (double)b;
            tot[2] = c;
        }
    }
};

// The next attempt of an adaptive update (attempt_begin_one): thread 0.
__device__ __forceinline__ void clu_attempt_begin(CluShared& S, int max_iter)
{
    if (S.status != ST_OK || !(S.t < S.tf)) {
        S.go = 0;
        return;
    }
    if (++S.iter > max_iter) {
        S.status = ST_STEP;
        S.go = 0;
        return;
    }
    S.go = 1;
    S.dt = fmin(S.dt, S.tf - S.t);
    S.h = S.dt;
}

// ts_decide: thread 0
__device__ __forceinline__ void clu_decide(CluShared& S, const ClusterArgs& g, double dt_min, long long max_reject,
                                           long long rej0)
{
    S.n_att++;
    if (S.err < 1) {
        S.accepted = 1;
        S.t = S.t + S.h;
        // (pow(x, 1) is x: the controller the reference uses skips a long FP64 chain)
        S.dt = fmin(S.h * (g.q == 1.0 ? 1 / S.err : pow(1 / S.err, 1 / g.q)), g.dt_max);
        S.n_acc++;
    } else {
        S.accepted = 0;
        S.dt = S.h * 0.5;
        S.n_rej++;
        if (S.n_rej - rej0 > max_reject || S.dt < dt_min) S.status = ST_STEP;
    }
}

}  // namespace

template <int MODE, int NT, int CH>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1) k_cluster(ClusterArgs one)
{
    __shared__ CluShared S;
    __shared__ __align__(16) unsigned char s_args_raw[sizeof(ClusterArgs)];
    ClusterArgs& s_args = *reinterpret_cast<ClusterArgs*>(s_args_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), nc = (int)cl.num_blocks();
    const int tid = threadIdx.x;
    for (int e = tid; e < (int)(sizeof(ClusterArgs) / 4); e += NT)
        reinterpret_cast<int*>(&s_args)[e] = reinterpret_cast<const int*>(&one)[e];
    __syncthreads();
    const ClusterArgs& g = s_args;
    const int nx = g.p.nx, ny = g.p.ny;
    const CluLay L(nx, g.p.h, ny, g.rpc, g.cpc, g.stages);
    Ctl* ctl = g.ctl;
    if (tid == 0) {
        S.t = ctl->t;
        S.dt = ctl->dt;
        S.tf = ctl->tf;
        S.h = ctl->h;
        S.tol = ctl->tol;
        S.err = ctl->err;
        S.n_acc = S.n_rej = S.n_att = 0;
        S.status = ctl->status;
        S.accepted = ctl->accepted;
        S.iter = 0;
        S.have = 0;
        S.n_rej = ctl->n_reject;
        for (int c = 0; c < 4; ++c) S.corner[c] = 0.f;
    }
    const double dt_min = ctl->dt_min;
    const long long max_reject = ctl->max_reject, rej0 = ctl->rej0;
    (void)dt_min; (void)max_reject; (void)rej0;
    Clu<NT, CH> C(g, smf, L, S, rank, nc);
    C.copy_fixed();
    const bool lead = rank == 0 && tid == 0;
    float* xh = smf + L.xh;
    float* xl = smf + L.xl;
    float* dxw = smf + L.dxw;
    float* fr = smf + L.fr;
    // the state as a float pair (k_split, k_split_dxw)
    const double* src = MODE == CLU_TSIT ? g.w : g.x;
    // the FP64 state of the own cells in registers for the whole update (not
    // where RK4 owns eight rows: one access a step is cheaper than the spills)
    constexpr bool XREG = !(MODE == CLU_RK4 && CH == 8);
    double xr[XREG ? CH : 1];
#pragma unroll
    for (int q = 0; q < (XREG ? CH : 1); ++q) xr[q] = 0.0;
    C.cells([&](int r, int e, int q) {
        const size_t c = (size_t)(C.r0 + r) * nx + C.i;
        const double v = src[c];
        if constexpr (XREG) xr[q] = MODE == CLU_TSIT ? g.x[c] : v;
        const float a = (float)v, b = (float)(v - (double)a);
        xh[e] = a;
        xl[e] = b;
        if (MODE != CLU_TSIT) dxw[e] = (a - g.wrhi[c]) + (b - g.wrlo[c]);
    });
    cluster_barrier();   // every block has read the control block and runs

    bool steps = false;   // the state moved
    const size_t n = (size_t)nx * ny;
    (void)n;
    if constexpr (MODE == CLU_RK4) {
        // k_1 + 2 k_2 + 2 k_3 of the own cells, each raw less its corner mean
        // before it is added (the mean can be most of it)
        float acc[CH];
#pragma unroll
        for (int q = 0; q < CH; ++q) acc[q] = 0.f;
        for (int step = 0; step < g.nsteps; ++step) {
            if (tid == 0) {
                S.go = S.status == ST_OK && S.t < S.tf;
                S.h = fmin(S.dt, S.tf - S.t);   // src/integrators.f90:62-63
                for (int st = 1; st < 4; ++st) S.f[st] = (float)(c_rk4_a[st] * S.h * g.spy);
                S.f[4] = (float)((S.h / 6) * g.spy);
            }
            __syncthreads();
            if (!S.go) break;   // alike in every block
            for (int stage = 0; stage < 4; ++stage) {
                const float sdf = stage > 0 ? S.f[stage] : 0.f;
                C.cells([&](int r, int e, int q) {
                    float hi = xh[e], lo = xl[e];
                    if (stage > 0) pair_add(hi, lo, sdf * fr[e], hi, lo);
                    C.put_y(r, hi, lo);
                });
                C.template rhs<true>(
                    [&]() {
                        if (stage > 0) S.f[6] = (float)C.corner();   // of the previous stage
                    },
                    [&](int e, int q) {
                        float dy = dxw[e];
                        if (stage > 0) {
                            const float k = fr[e] - S.f[6];
                            dy += sdf * k;
                            acc[q] = stage == 1 ? k : acc[q] + 2.f * k;
                        }
                        return dy;
                    });
            }
            cluster_barrier();   // the corners of the last stage
            if (tid == NT - 1) S.f[5] = (float)C.corner();
            if (tid == 0) {
                S.t = S.t + S.h;
                S.n_acc++;
            }
            __syncthreads();
            const float cm = S.f[5], sc = S.f[4];
            C.cells([&](int r, int e, int q) {
                const size_t c = (size_t)(C.r0 + r) * nx + C.i;
                const float inc = (acc[q] + (fr[e] - cm)) * sc;
                if constexpr (XREG) xr[q] += (double)inc;   // the FP64 state update
                else g.x[c] += (double)inc;
                float hi, lo;
                pair_add(xh[e], xl[e], inc, hi, lo);
                xh[e] = hi;
                xl[e] = lo;
                dxw[e] = (hi - g.wrhi[c]) + (lo - g.wrlo[c]);
            });
            __syncthreads();
        }
        steps = S.n_acc > 0;
    }

    // ---- Tsitouras 5(4), reference-compatible: the right-hand side sees
    // now%w only, so an attempt is one right-hand side (none after a
    // rejection), the error term 0.2 dt k and its norm (ts_fused), and x += dt k
    // where it is accepted (ts_commit_pair)
    if constexpr (MODE == CLU_TSIT) {
        bool valid = false;
        for (int par = 0;; par ^= 1) {
            if (tid == 0) {
                clu_attempt_begin(S, g.max_iter);
                const double dt = S.h;
                S.cx = ((dt * c_ts_b[0] + dt * c_ts_b[3]) + dt * c_ts_b[4]) + dt * c_ts_b[5];
                S.f[0] = (float)S.cx;
                S.f[1] = (float)(dt * c_ts_b[5] - dt * c_ts_bh[5]);
                S.f[2] = (float)g.spy;
                if (S.go) S.have = 1;
            }
            __syncthreads();
            if (!S.go) break;   // alike in every block
            if (!valid) {
                C.cells([&](int r, int e, int) { C.put_y(r, xh[e], xl[e]); });
                C.template rhs<false>([]() {}, [](int, int) { return 0.f; });
                cluster_barrier();   // the corners
                if (tid == NT - 1) S.cm[0] = (float)C.corner();
                valid = true;
                __syncthreads();
            }
            const float cxf = S.f[0], ce = S.f[1], spyf = S.f[2], cm = S.cm[0];
            const double cx = S.cx;
            float m1 = 0.f, m2 = 0.f, s2 = 0.f;
            C.cells([&](int, int e, int) {
                const float k = (fr[e] - cm) * spyf;
                const float dx = ce * k;
                const float x2f = xh[e] + (xl[e] + cxf * k);
                m1 = fmaxf(m1, fabsf(x2f - dx));
                m2 = fmaxf(m2, fabsf(x2f));
                s2 += dx * dx;
            });
            double tot[3];
            C.template reduce<false>(m1, m2, s2, par, tot);
            if (tid == 0) {
                S.tol = g.atol + g.rtol * fmax(tot[0], tot[1]);
                S.err = sqrt(tot[2] / (double)n) / S.tol;
                clu_decide(S, g, dt_min, max_reject, rej0);
            }
            __syncthreads();
            if (S.accepted) {
                C.cells([&](int, int e, int q) {
                    const float k = (fr[e] - cm) * spyf;
                    xr[q] += cx * (double)k;
                    pair_add(xh[e], xl[e], cxf * k, xh[e], xl[e]);
                });
                valid = false;
                steps = true;
            }
        }
    }

    // ---- Tsitouras 5(4) with true stages (the Dormand-Prince pair, FSAL):
    // dp_stage_pair, dp_err / ts_err, ts_commit_tpair
    if constexpr (MODE == CLU_TSIT_TRUE) {
        bool valid = false;
        // stage output q of the own cells (cell index e): shared memory where
        // they fit, else the domain's stage buffers
        auto kq = [&](int q) -> float* {
            return g.stages ? smf + L.kk + q * (g.rpc * nx) : g.raw[q] + (size_t)C.r0 * nx;
        };
        for (int par = 0;; par ^= 1) {
            if (tid == 0) {
                clu_attempt_begin(S, g.max_iter);
                if (S.go) S.have = 1;
            }
            __syncthreads();
            if (!S.go) break;   // alike in every block
            float a[CH];   // the increment of the current stage state
#pragma unroll
            for (int q = 0; q < CH; ++q) a[q] = 0.f;
            // stage 0 only where no accepted attempt left its right-hand side
            for (int i = valid ? 1 : 0; i <= 6; ++i) {
                if (tid < i) S.f[tid] = (float)(c_dp_a[i][tid] * S.h * g.spy);
                __syncthreads();
                C.cells([&](int r, int e, int q) {
                    float v = 0.f;
                    for (int s = 0; s < i; ++s) v += S.f[s] * (kq(s)[e] - S.cm[s]);
                    a[q] = v;
                    float hi, lo;
                    pair_add(xh[e], xl[e], v, hi, lo);
                    C.put_y(r, hi, lo);
                });
                C.template rhs<true>([]() {}, [&](int e, int q) { return dxw[e] + a[q]; });
                cluster_barrier();   // the corners
                if (tid == NT - 1) S.cm[i] = (float)C.corner();
                float* ki = kq(i);
                C.cells([&](int, int e, int) { ki[e] = fr[e]; });
                __syncthreads();
            }
            valid = true;
            if (tid < 7) S.f[tid] = (float)(((tid < 6 ? c_dp_a[6][tid] : 0.0) - c_dp_bs[tid]) * S.h * g.spy);
            __syncthreads();
            float m1 = 0.f, m2 = 0.f, s2 = 0.f;
            C.cells([&](int, int e, int q) {
                float dx = 0.f;
                for (int s = 0; s < 7; ++s) dx += S.f[s] * (kq(s)[e] - S.cm[s]);
                const float x2f = (float)(xr[q] + (double)a[q]);
                m1 = fmaxf(m1, fabsf(x2f - dx));
                m2 = fmaxf(m2, fabsf(x2f));
                s2 += dx * dx;
            });
            double tot[3];
            C.template reduce<true>(m1, m2, s2, par, tot);
            if (tid == 0) {
                S.tol = g.atol + g.rtol * fmax(tot[0], tot[1]);
                S.err = sqrt(tot[2] / (double)n) / S.tol;
                clu_decide(S, g, dt_min, max_reject, rej0);
            }
            __syncthreads();
            if (S.accepted) {
                float* k0 = kq(0);
                const float* k6 = kq(6);
                const float* yh = smf + L.yh;
                const float* yl = smf + L.yl;
                C.cells([&](int r, int e, int q) {
                    const size_t c = (size_t)(C.r0 + r) * nx + C.i;
                    xr[q] += (double)a[q];
                    const float hi = yh[(r + 2) * nx + C.i], lo = yl[(r + 2) * nx + C.i];   // the stage-6 pair
                    xh[e] = hi;
                    xl[e] = lo;
                    dxw[e] = (hi - g.wrhi[c]) + (lo - g.wrlo[c]);
                    k0[e] = k6[e];
                });
                if (tid == 0) S.cm[0] = S.cm[6];
                steps = true;
                __syncthreads();
            }
        }
    }

    // state, now%w and the last right-hand side back to the domain
    float* last = g.raw[MODE == CLU_RK4 ? 3 : 0];
    C.cells([&](int r, int e, int q) {
        const size_t c = (size_t)(C.r0 + r) * nx + C.i;
        if (steps) {
            if constexpr (XREG) {
                g.x[c] = xr[q];
                g.w[c] = xr[q];
            } else {
                g.w[c] = g.x[c];
            }
        }
        if (MODE == CLU_RK4 ? steps : S.have != 0) last[c] = fr[e];
    });
    cluster_barrier();   // no block leaves while another may still reach into it
    if (lead) {
        ctl->t = S.t;
        ctl->h = S.h;
        ctl->n_accept += S.n_acc;
        ctl->done = S.status == ST_OK ? 0 : 1;
        if (MODE != CLU_RK4) {
            ctl->dt = S.dt;
            ctl->tol = S.tol;
            ctl->err = S.err;
            ctl->accepted = S.accepted;
            ctl->n_reject = S.n_rej;
            ctl->n_attempt += S.n_att;
            ctl->status = S.status;
            ctl->have_rhs = S.have;
            ctl->loop_iter = S.iter;
            ctl->rhs_valid = 0;
            ctl->need_rhs = 0;
            ctl->active = 0;
        }
    }
}

template <int MODE, int NT, int CH>
cudaError_t cluster_go(const ClusterArgs& a, int nc, size_t smem, cudaStream_t s, bool probe)
{
    static std::mutex mu;
    static size_t cur = 0;
    auto kern = k_cluster<MODE, NT, CH>;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (cur == 0) {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e != cudaSuccess) return e;
        }
        if (smem > cur) {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            cur = smem;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nc;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (probe) {
        // configuration only: can such a cluster be resident at all?
        int k = 0;
        const cudaError_t e = cudaOccupancyMaxActiveClusters(&k, kern, &cfg);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return e;
        }
        return k > 0 ? cudaSuccess : cudaErrorInvalidConfiguration;
    }
    return cudaLaunchKernelEx(&cfg, kern, a);
}

}  // namespace fi
