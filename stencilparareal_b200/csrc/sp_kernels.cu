// sp_kernels.cu -- sm_100a kernels of the advection-diffusion propagator.
//
// Stage kernels.  One launch evaluates the right-hand side on every cell of
// one or more fields and fuses the Runge-Kutta (or Euler, or adjoint)
// pointwise update and the periodic halo into the same pass:
//
//   reference (Convection.cpp:318-370), per RK4 step:
//     4 x [Periodicity I/J/K kernels + RHS4 stencil] + 3 x Euler + 1 x RK
//   here, per RK4 step (q = step start, y = stage values, a = accumulator):
//     S1: k=R(q);  y1=q+dt/2 k
//     S2: k=R(y1); y2=q+dt/2 k;  a=q+(y1-q)/3+dt/3 k
//     S3: k=R(y2); y3=q+dt k
//     S4: k=R(y3); q'=a+(y3-q)/3+dt/6 k   (13 field accesses per cell-update)
//   ((y1-q)/3 = dt/6 k1 and (y3-q)/3 = dt/3 k3 recover two accumulator terms
//   from stage values, so that only S2 writes the accumulator)
//
// R is RHS4Stage (Convection.cpp:57-82): Advection4 (ConvectionFunctions.h:66-104)
// plus nu * Laplace4 (ConvectionFunctions.h:135-167), written as
//   R = sum_d c_d/(12dx) * (8(q[-1]-q[+1]) - (q[-2]-q[+2]))_d
//     + nu/(12dx^2) * (16 S1 - S2 - 90 q),  S1/S2 = sums of the +-1/+-2 neighbours,
// the same coefficients regrouped into differences (the adjoint); the RK
// stages of both implementations use them combined into 13 per-offset weights (rhs_w13, sp_stencil.cuh), as the fused stage pairs do.  R2 is RHS2Stage
// (Convection.cpp:30-55) with the upwind Advection2 (ConvectionFunctions.h:18-42).
//
// Fields carry a 2-cell halo (layout in include/sp_abi.h).  Every kernel that
// writes a stencil input also writes the periodic images of the cells within
// two of a face, which replaces Periodicity::Apply (Periodicity.cu:146-214).
//
// Two implementations of every stage:
//  * k_stage_tma: a CTA owns a (32*VX) x TY tile of one field and marches a
//    chunk of z-planes.  One elected thread streams each plane's tile plus its
//    x/y halo with a single 3-D TMA box (cp.async.bulk.tensor) into a ring of
//    shared-memory slots completed on mbarriers; pointwise operands arrive the
//    same way.  The z-neighbours live in registers.  16-byte shared and global
//    accesses, VX = 2 (FP64) or 4 (FP32) cells per thread.
//  * k_stage_direct: one 16-byte chunk of a row per thread, loads straight from
//    global memory through L1: the faster one for small launches.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "sp_column.cuh"
#include "sp_device.cuh"
#include "sp_internal.h"
#include "sp_stencil.cuh"

namespace sp {

namespace {
std::atomic<long long> g_launches{0};
}
long long launches() { return g_launches.load(); }
void add_launches(long long n) { g_launches += n; }

Geo make_geo(int ni, int nj, int nk, int es, int halo) {
    Geo g;
    g.ni = ni; g.nj = nj; g.nk = nk; g.es = es; g.halo = halo;
    g.lx = (halo * es + 15) / 16 * 16 / es;
    const long long need = (long long)ni + 2 * g.lx;
    g.px = (need + 31) / 32 * 32;
    g.py = nj + 2 * halo;
    g.pz = nk + 2 * halo;
    g.plane = g.px * g.py;
    g.origin = halo * g.plane + halo * g.px + g.lx;
    g.total = g.plane * g.pz;
    return g;
}

Coef make_coef(double dx, double cx, double cy, double cz, int upwind) {
    Coef c;
    const double cs[3] = {cx, cy, cz};
    for (int d = 0; d < 3; ++d) {
        c.ca[d] = cs[d] / (12. * dx);
        if (upwind) {
            // Advection2, UPWINDADVECTION: -(c*dq)/dx, dq one-sided by the sign of c
            c.mode[d] = cs[d] > 0. ? 0 : 1;
            c.u[d] = -cs[d] / dx;
        } else {
            c.mode[d] = 2;
            c.u[d] = cs[d] / (2. * dx);
        }
    }
    c.s4 = 1. / (12. * dx * dx);
    c.s2 = 1. / (dx * dx);
    c.dx = dx;
    return c;
}

// Kernel arguments.
template <typename T>
struct KArgs {
    T* yout;          // stencil output (with images)
    T* aout;          // pointwise output (accumulator / adjoint accumulator)
    const T* yin;     // stencil input
    const T* pw0;     // pointwise operands (meaning per op)
    const T* pw1;
    const T* pw2;
    long long item_stride, origin, px, plane;
    int ni, nj, nk, pz;
    int tiles_x, zchunk, nzc;
    int zrev;         // TMA kernel: CTAs take items and z-chunks in descending order
    StoreBounds sb_y, sb_a;  // output allocations of yout and aout (bounds-checked builds)
    const int* item_lo;
    int item_base;
    T ca0, ca1, ca2;          // c_d/(12dx)
    T u0, u1, u2;             // RHS2 advection coefficients
    int m0, m1, m2;           // RHS2 difference modes
    T nl;                     // nu/(12dx^2) (adjoint) or nu/dx^2 (Euler)
    T c_y, c_acc;             // stage coefficients
    T sigma;                  // adjoint: mu_s = sigma * (stencil input)
    double* par_acc;          // adjoint: 4 parameter-gradient sums
    double gs_nu, gs_c;       // adjoint: scales of the nu and c sums
    int* err;
};

template <int OP>
struct OpTraits {
    static constexpr int npw = (OP == OP_RK_S2 || OP == OP_RK_S3) ? 1   // q
                             : (OP == OP_RK_S4) ? 2                        // acc, q
                             : (OP == OP_ADJ + 0) ? 1      // ADJ4: y4
                             : (OP == OP_ADJ + 1 || OP == OP_ADJ + 2) ? 3   // ADJ3/ADJ2: y, lam, lam_acc
                             : (OP == OP_ADJ + 3) ? 2      // ADJ1: y1, lam_acc
                             : 0;
    static constexpr bool writes_a = (OP == OP_RK_S2 || OP == OP_ADJ + 0 ||
                                      OP == OP_ADJ + 1 || OP == OP_ADJ + 2);
    static constexpr bool adjoint = OP >= OP_ADJ;
};

template <typename T>
__device__ __forceinline__ T diff_mode(int m, T c, T lo, T hi) {
    return m == 0 ? c - lo : (m == 1 ? hi - c : lo - hi);
}

// The RK update of one cell from k = R(stencil input): c the stencil input's
// centre, q0, q1 the pointwise operands.
template <typename T, int OP>
__device__ __forceinline__ void rk_update(const KArgs<T>& a, T k, T c, T q0, T q1, T& oy, T& oa) {
    if constexpr (OP == OP_RK_S1) {
        oy = fmaT(a.c_y, k, c);
    } else if constexpr (OP == OP_RK_S2) {
        oy = fmaT(a.c_y, k, q0);
        oa = fmaT(a.c_acc, k, add_third(c, q0, q0));
    } else if constexpr (OP == OP_RK_S3) {
        oy = fmaT(a.c_y, k, q0);
    } else {
        oy = fmaT(a.c_acc, k, add_third(c, q1, q0));
    }
    (void)q0; (void)q1; (void)oa;
}

// One cell of an Euler or adjoint stage.  p0..p2: pointwise operands; oy/oa: outputs;
// g[4]: adjoint parameter partial sums (unscaled).
template <typename T, int OP>
__device__ __forceinline__ void cell_op(const KArgs<T>& a, const Nb<T>& s, T p0, T p1, T p2, T& oy, T& oa,
                                        double* g, bool live) {
    if constexpr (OP == OP_EULER) {
        const T dqx = diff_mode(a.m0, s.c, s.xm1, s.xp1);
        const T dqy = diff_mode(a.m1, s.c, s.ym1, s.yp1);
        const T dqz = diff_mode(a.m2, s.c, s.zm1, s.zp1);
        const T adv = fmaT(a.u0, dqx, fmaT(a.u1, dqy, a.u2 * dqz));
        T lap;
        if constexpr (sizeof(T) == 4) {
            // FP32: the sum of the neighbours' differences from the centre (exact
            // and small), not the cancelling S1 - 6q (see rhs_w13)
            const T c = s.c;
            lap = ((s.xm1 - c) + (s.xp1 - c)) + ((s.ym1 - c) + (s.yp1 - c)) + ((s.zm1 - c) + (s.zp1 - c));
        } else {
            lap = ((s.xm1 + s.xp1) + (s.ym1 + s.yp1) + (s.zm1 + s.zp1)) - T(6) * s.c;
        }
        const T k = fmaT(a.nl, lap, adv);
        oy = fmaT(a.c_y, k, s.c);
        (void)p0; (void)p1; (void)p2; (void)oa; (void)g; (void)live;
    } else {
        const T ax = fmaT(T(8), s.xm1 - s.xp1, s.xp2 - s.xm2);
        const T ay = fmaT(T(8), s.ym1 - s.yp1, s.yp2 - s.ym2);
        const T az = fmaT(T(8), s.zm1 - s.zp1, s.zp2 - s.zm2);
        T lap;
        if constexpr (sizeof(T) == 4) {
            // FP32: 16 D1 - D2 with D1, D2 the neighbours' differences from the
            // centre (equal to -90 q + 16 S1 - S2; see rhs_w13)
            const T c = s.c;
            const T D1 = ((s.xm1 - c) + (s.xp1 - c)) + ((s.ym1 - c) + (s.yp1 - c)) + ((s.zm1 - c) + (s.zp1 - c));
            const T D2 = ((s.xm2 - c) + (s.xp2 - c)) + ((s.ym2 - c) + (s.yp2 - c)) + ((s.zm2 - c) + (s.zp2 - c));
            lap = fmaT(T(16), D1, -D2);
        } else {
            const T S1 = (s.xm1 + s.xp1) + (s.ym1 + s.yp1) + (s.zm1 + s.zp1);
            const T S2 = (s.xm2 + s.xp2) + (s.ym2 + s.yp2) + (s.zm2 + s.zp2);
            lap = fmaT(T(-90), s.c, fmaT(T(16), S1, -S2));
        }
        const T adv = fmaT(a.ca0, ax, fmaT(a.ca1, ay, a.ca2 * az));
        {
            // R^T m = -sum_d c_d D_d m + nu L m (D_d antisymmetric, L symmetric on the periodic grid)
            const T ybar = a.sigma * fmaT(a.nl, lap, -adv);
            if (live) {
                g[0] += (double)p0 * (double)lap;
                g[1] += (double)p0 * (double)ax;
                g[2] += (double)p0 * (double)ay;
                g[3] += (double)p0 * (double)az;
            }
            if constexpr (OP == OP_ADJ + 0) {         // stencil input is lam
                oy = fmaT(a.c_y, ybar, a.c_acc * s.c);  // mu3 = h ybar4 + h/3 lam
                oa = s.c + ybar;                       // lam_acc = lam + ybar4
            } else if constexpr (OP == OP_ADJ + 1 || OP == OP_ADJ + 2) {
                oy = fmaT(a.c_y, ybar, a.c_acc * p1);  // mu_{s-1} = c_y ybar_s + c_acc lam
                oa = p2 + ybar;
            } else {                                   // ADJ1: final lam_n
                oy = p1 + ybar;
            }
        }
    }
}

template <typename T, int N>
__device__ __forceinline__ void put_vec(const StoreBounds& b, T* p, int x, int ni, const Vec<T, N>& v) {
    if (x + N <= ni) {
        gst16<T>(b, p, v);
    } else {
#pragma unroll
        for (int e = 0; e < N; ++e)
            if (x + e < ni) gst1(b, p + e, v.v[e]);
    }
}

// Vector store of cells x..x+N-1 of row (y,z) plus periodic images.
template <typename T, int N>
__device__ __forceinline__ void store_images_vec(T* base, int x, int y, int z, const Vec<T, N>& v,
                                                 const KArgs<T>& a) {
    T* row = base + (long long)z * a.plane + (long long)y * a.px + x;
    const StoreBounds& b = a.sb_y;
    put_vec<T, N>(b, row, x, a.ni, v);
#pragma unroll
    for (int e = 0; e < N; ++e) {
        const int xe = x + e;
        if (xe < a.ni) {
            if (xe < 2) gst1(b, row + e + a.ni, v.v[e]);
            if (xe >= a.ni - 2) gst1(b, row + e - a.ni, v.v[e]);
        }
    }
    if (y < 2) put_vec<T, N>(b, row + (long long)a.nj * a.px, x, a.ni, v);
    if (y >= a.nj - 2) put_vec<T, N>(b, row - (long long)a.nj * a.px, x, a.ni, v);
    if (z < 2) put_vec<T, N>(b, row + (long long)a.nk * a.plane, x, a.ni, v);
    if (z >= a.nk - 2) put_vec<T, N>(b, row - (long long)a.nk * a.plane, x, a.ni, v);
}

// Reduces the four adjoint parameter sums over the CTA (warp shuffles, then
// shared memory) and adds them to par_acc with one atomic per CTA and sum.
// Every thread of the CTA must call it.
__device__ __forceinline__ void reduce_par(double* g, double* par_acc, double gs_nu, double gs_c) {
    __shared__ double red[32][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        for (int o = 16; o > 0; o >>= 1) g[i] += __shfl_xor_sync(0xffffffffu, g[i], o);
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const int nwarp = (blockDim.x * blockDim.y + 31) / 32;
    if ((tid & 31) == 0)
#pragma unroll
        for (int i = 0; i < 4; ++i) red[tid >> 5][i] = g[i];
    __syncthreads();
    if (tid < 4) {
        double v = 0.;
        for (int w = 0; w < nwarp; ++w) v += red[w][tid];
        atomicAdd(par_acc + tid, (tid == 0 ? gs_nu : gs_c) * v);
    }
}

// ---------------------------------------------------------------------------
// Direct-load stage kernel: a thread owns one 16-byte chunk (2 FP64 or 4 FP32
// cells) of one row and marches zchunk planes, everything loaded straight from
// global memory (L1 serves the reuse between the block's rows).  The chunks of a
// plane are numbered row by row, so that a row of any width fills its warps;
// grid (ceil(chunks / threads), nzc, items).
//
// Bound by latency at the sizes it is for: below ~4M FP64 cells a stage is one
// short wave, and what counts is the time from launch to the last store.  Hence
// no barrier and no shared-memory ring to fill, few registers (50-64 for the
// FP64 RK stages: 8 to 10 blocks of 128 threads per SM), a compact plane loop
// (not unrolled: 2-3 KB of code per stage instead of 10-25 KB, which the short
// kernels spent their time fetching) and programmatic dependent launch.  us per
// RK4 step, one-thread-per-cell direct kernel / best TMA ring / this kernel:
//   FP64  64^3 16.2 / 25.6 / 12.6   96^3 29.5 / 34.5 / 23.5   128^3 57.4 / 53.2 / 51.2   192^3 196 / 156 / 175
//   FP32  64^3 17.7 / 27.2 / 13.3   96^3 30.6 / 30.8 / 18.9   128^3 56.4 / 34.9 / 32.2   192^3 167 / 112 / 102
// Unrolled by two with the next plane prefetched (70-100 registers): 64^3 FP32
// 11.0, but 128^3 FP64 62.5 and FP32 41.8.

// A chunk by a plain global load, `off` bytes from `base`.  Not volatile, so that the
// compiler may move it over the stores of other cells; the bases come from pointers
// passed through after_wait, so that it cannot move over griddepcontrol.wait.
template <typename T>
__device__ __forceinline__ Vec<T, V16<T>::N> ldg16(const char* base, uint32_t off) {
    Vec<T, V16<T>::N> r;
    const char* p = base + off;
    if constexpr (sizeof(T) == 8)
        asm("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(r.v[0]), "=d"(r.v[1]) : "l"(p));
    else
        asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
            : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3])
            : "l"(p));
    return r;
}
template <typename T>
__device__ __forceinline__ Vec<T, V16<T>::N> ldg16(const T* p) {
    return ldg16<T>(reinterpret_cast<const char*>(p), 0u);
}
template <typename T>
__device__ __forceinline__ const char* after_wait(T* p) {
    asm volatile("" : "+l"(p)::"memory");
    return reinterpret_cast<const char*>(p);
}

template <typename T, int OP, int NW>
__global__ void __launch_bounds__(512)
    k_stage_direct(const __grid_constant__ KArgs<T> a, const __grid_constant__ Weights<T, NW> wt) {
    constexpr int N = V16<T>::N, NPW = OpTraits<OP>::npw;
    constexpr bool RK = OP <= OP_RK_S4;
    using V = Vec<T, N>;
    pdl_trigger();
    pdl_wait();
    const int b = blockIdx.z;
    if (a.item_lo && b + a.item_base < *a.item_lo) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = t / a.tiles_x;  // tiles_x: chunks per row
    const int x = (t - y * a.tiles_x) * N;
    double g[4] = {0., 0., 0., 0.};
    if (y < a.nj) {
        const int z0 = (a.zrev ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y) * a.zchunk;
        const int z1 = min(z0 + a.zchunk, a.nk);
        const long long ob = (long long)b * a.item_stride + a.origin;
        const long long col = ob + (long long)y * a.px + x;
        const T* S = reinterpret_cast<const T*>(after_wait(a.yin)) + col;
        [[maybe_unused]] const T* pw[3] = {nullptr, nullptr, nullptr};
        if constexpr (NPW > 0) pw[0] = reinterpret_cast<const T*>(after_wait(a.pw0)) + col;
        if constexpr (NPW > 1) pw[1] = reinterpret_cast<const T*>(after_wait(a.pw1)) + col;
        if constexpr (NPW > 2) pw[2] = reinterpret_cast<const T*>(after_wait(a.pw2)) + col;
        const long long pl = a.plane, px = a.px;
        V win[5];  // the column's planes z-2 .. z+2
#pragma unroll
        for (int i = 0; i < 4; ++i) win[i] = ldg16<T>(S + (z0 - 2 + i) * pl);
#pragma unroll 1
        for (int z = z0; z < z1; ++z) {
            const long long zo = z * pl;
            const T* P = S + zo;
            win[4] = ldg16<T>(P + 2 * pl);
            const V xl = ldg16<T>(P - N), xr = ldg16<T>(P + N);
            const V ym1 = ldg16<T>(P - px), yp1 = ldg16<T>(P + px);
            const V ym2 = ldg16<T>(P - 2 * px), yp2 = ldg16<T>(P + 2 * px);
            [[maybe_unused]] V p[3];
#pragma unroll
            for (int k = 0; k < NPW; ++k) p[k] = ldg16<T>(pw[k] + zo);
            T row[3 * N];
#pragma unroll
            for (int e = 0; e < N; ++e) { row[e] = xl.v[e]; row[N + e] = win[2].v[e]; row[2 * N + e] = xr.v[e]; }
            V oy, oa;
#pragma unroll
            for (int e = 0; e < N; ++e) {
                Nb<T> s;
                s.c = row[N + e];
                s.xm1 = row[N + e - 1]; s.xp1 = row[N + e + 1];
                s.xm2 = row[N + e - 2]; s.xp2 = row[N + e + 2];
                s.ym1 = ym1.v[e]; s.yp1 = yp1.v[e]; s.ym2 = ym2.v[e]; s.yp2 = yp2.v[e];
                s.zm1 = win[1].v[e]; s.zp1 = win[3].v[e]; s.zm2 = win[0].v[e]; s.zp2 = win[4].v[e];
                T q0 = 0, q1 = 0, q2 = 0, vy = 0, va = 0;
                if constexpr (NPW > 0) q0 = p[0].v[e];
                if constexpr (NPW > 1) q1 = p[1].v[e];
                if constexpr (NPW > 2) q2 = p[2].v[e];
                if constexpr (RK) rk_update<T, OP>(a, rhs_w13(wt.w[NW == 1 ? 0 : b], s), s.c, q0, q1, vy, va);
                else cell_op<T, OP>(a, s, q0, q1, q2, vy, va, g, x + e < a.ni);
                oy.v[e] = vy;
                oa.v[e] = va;
            }
            const bool edge = x < 2 || x + N > a.ni - 2 || y < 2 || y >= a.nj - 2 || z < 2 || z >= a.nk - 2;
            if (!edge) gst16<T>(a.sb_y, a.yout + col + zo, oy);
            else store_images_vec<T, N>(a.yout + ob, x, y, z, oy, a);
            if constexpr (OpTraits<OP>::writes_a) put_vec<T, N>(a.sb_a, a.aout + col + zo, x, a.ni, oa);
#pragma unroll
            for (int i = 0; i < 4; ++i) win[i] = win[i + 1];
        }
    }
    if constexpr (OpTraits<OP>::adjoint) reduce_par(g, a.par_acc, a.gs_nu, a.gs_c);
}

// ---------------------------------------------------------------------------
// Wrapping direct kernel: the direct kernel for chains of direct stages on grids
// whose rows are whole chunks.  It takes its neighbours at their wrapped indices,
// so no stage needs, or writes, periodic images (the driver refreshes those of the
// field it hands out).  Every offset inside a plane is worked out once per thread,
// and ZB planes are marched without a loop.
//
// What it saves is instructions: a warp's plane of S1 takes 137 (FP64) or 273 (FP32)
// instead of 211 or 326, a third of which went to images (every warp holds a chunk
// at an x face, so every warp took that path) and to moving the z-window.  FP32,
// bound by issue, gains (us per RK4 step: 96^3 18.9 -> 17.4, 128^3 32.2 -> 27.4, 192^3
// 102 -> 92; a gradient, in FP64, 64^3 58 -> 49, 96^3 110 -> 90); FP64 from 100^3 on is bound by what it reads through L2 (100^3 30 ->
// 27.4, 128^3 51.2 -> 49.0), below by the launches (64^3 12.6 -> 12.1).
template <typename T, int OP, int NW, int ZB>
__global__ void __launch_bounds__(512)
    k_stage_wrap(const __grid_constant__ KArgs<T> a, const __grid_constant__ Weights<T, NW> wt) {
    constexpr int N = V16<T>::N, ES = (int)sizeof(T), NPW = OpTraits<OP>::npw;
    constexpr bool RK = OP <= OP_RK_S4;
    using V = Vec<T, N>;
    pdl_trigger();
    pdl_wait();
    const int b = blockIdx.z;
    if (a.item_lo && b + a.item_base < *a.item_lo) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = t / a.tiles_x;  // tiles_x: chunks per row
    const int x = (t - y * a.tiles_x) * N;
    [[maybe_unused]] double g[4] = {0., 0., 0., 0.};
    auto march = [&]() {
        const int z0 = (a.zrev ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y) * a.zchunk;
        const int z1 = min(z0 + a.zchunk, a.nk);
        // byte offsets in a plane of the chunk and its neighbours
        const uint32_t row = (uint32_t)a.px * ES;
        const uint32_t o = (uint32_t)y * row + (uint32_t)x * ES;
        const uint32_t ol = o + (x == 0 ? (uint32_t)(a.ni - N) * ES : (uint32_t)-16);
        const uint32_t orr = o + (x + N == a.ni ? (uint32_t)(N - a.ni) * ES : 16u);
        auto wrap_y = [&](int d) { return o + (uint32_t)(d + (y + d < 0 ? a.nj : (y + d >= a.nj ? -a.nj : 0))) * row; };
        const uint32_t om2 = wrap_y(-2), om1 = wrap_y(-1), op1 = wrap_y(1), op2 = wrap_y(2);
        const long long pl = a.plane * ES;
        const long long base = ((long long)b * a.item_stride + a.origin) * ES;
        const char* F = after_wait(a.yin) + base;
        auto plane = [&](int z) { return F + (z < 0 ? z + a.nk : (z >= a.nk ? z - a.nk : z)) * pl; };
        [[maybe_unused]] const char* pw[3] = {nullptr, nullptr, nullptr};
        if constexpr (NPW > 0) pw[0] = after_wait(a.pw0) + base;
        if constexpr (NPW > 1) pw[1] = after_wait(a.pw1) + base;
        if constexpr (NPW > 2) pw[2] = after_wait(a.pw2) + base;
        char* Y = reinterpret_cast<char*>(a.yout) + base;
        [[maybe_unused]] char* A = reinterpret_cast<char*>(a.aout) + base;
        V win[ZB + 4];  // the column's planes z-2 .. z+ZB+1
#pragma unroll
        for (int i = 0; i < 4; ++i) win[i] = ldg16<T>(plane(z0 - 2 + i), o);
#pragma unroll 1
        for (int z = z0; z < z1; z += ZB) {
#pragma unroll
            for (int i = 0; i < ZB; ++i) win[4 + i] = ldg16<T>(plane(min(z + 2 + i, a.nk + 1)), o);
#pragma unroll
            for (int i = 0; i < ZB; ++i) {
                if (i > 0 && z + i >= z1) break;
                const long long zo = (z + i) * pl;
                const char* S = F + zo;
                const V xl = ldg16<T>(S, ol), xr = ldg16<T>(S, orr);
                const V ym1 = ldg16<T>(S, om1), yp1 = ldg16<T>(S, op1);
                const V ym2 = ldg16<T>(S, om2), yp2 = ldg16<T>(S, op2);
                [[maybe_unused]] V p[3];
#pragma unroll
                for (int k = 0; k < NPW; ++k) p[k] = ldg16<T>(pw[k] + zo, o);
                T row3[3 * N];
#pragma unroll
                for (int e = 0; e < N; ++e) { row3[e] = xl.v[e]; row3[N + e] = win[i + 2].v[e]; row3[2 * N + e] = xr.v[e]; }
                V oy, oa;
#pragma unroll
                for (int e = 0; e < N; ++e) {
                    Nb<T> s;
                    s.c = row3[N + e];
                    s.xm1 = row3[N + e - 1]; s.xp1 = row3[N + e + 1];
                    s.xm2 = row3[N + e - 2]; s.xp2 = row3[N + e + 2];
                    s.ym1 = ym1.v[e]; s.yp1 = yp1.v[e]; s.ym2 = ym2.v[e]; s.yp2 = yp2.v[e];
                    s.zm1 = win[i + 1].v[e]; s.zp1 = win[i + 3].v[e]; s.zm2 = win[i].v[e]; s.zp2 = win[i + 4].v[e];
                    T q0 = 0, q1 = 0, q2 = 0, vy = 0, va = 0;
                    if constexpr (NPW > 0) q0 = p[0].v[e];
                    if constexpr (NPW > 1) q1 = p[1].v[e];
                    if constexpr (NPW > 2) q2 = p[2].v[e];
                    if constexpr (RK) rk_update<T, OP>(a, rhs_w13(wt.w[NW == 1 ? 0 : b], s), s.c, q0, q1, vy, va);
                    else cell_op<T, OP>(a, s, q0, q1, q2, vy, va, g, true);
                    oy.v[e] = vy;
                    oa.v[e] = va;
                }
                gst16<T>(a.sb_y, reinterpret_cast<T*>(Y + zo + o), oy);
                if constexpr (OpTraits<OP>::writes_a) gst16<T>(a.sb_a, reinterpret_cast<T*>(A + zo + o), oa);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) win[i] = win[i + ZB];
        }
    };
    if (y < a.nj) march();
    if constexpr (OpTraits<OP>::adjoint) reduce_par(g, a.par_acc, a.gs_nu, a.gs_c);
}

// ---------------------------------------------------------------------------
// TMA stage kernel.  Block = 32*TY threads (warp w owns tile row w), grid
// (tiles_x*tiles_y, nzc, items), taken in descending item / z-chunk order when
// zrev is set.  Shared memory: NS stencil-input slots of (TX+2LX) x (TY+4)
// elements and NP pointwise slots of npw x TX x TY elements, followed by NS+NP
// mbarriers.  Ring bookkeeping uses running slot indices and phase bits instead
// of divisions; lanes whose cells are two or more cells away from every y face
// store one 16-byte vector (plus the x images of cells next to an x face)
// except on the four planes next to the z faces.


template <typename T, int OP, int TY, int NS, int NP, int NW>
__global__ void __launch_bounds__(32 * TY)
    k_stage_tma(const __grid_constant__ CUtensorMap tm_s, const __grid_constant__ CUtensorMap tm_p0,
                const __grid_constant__ CUtensorMap tm_p1, const __grid_constant__ CUtensorMap tm_p2,
                const KArgs<T> a, const __grid_constant__ Weights<T, NW> wt) {
    constexpr int VX = V16<T>::N;
    constexpr int TX = 32 * VX;
    constexpr int LX = VX;
    constexpr int W = TX + 2 * LX;
    constexpr int H = TY + 4;
    constexpr int YT = W * H;
    constexpr int PT = TX * TY;
    constexpr int NPA = OpTraits<OP>::npw;
    constexpr uint32_t YBYTES = YT * sizeof(T);
    constexpr uint32_t PBYTES = NPA * PT * sizeof(T);
    constexpr bool RK = OP <= OP_RK_S4;
    static_assert((YT * sizeof(T)) % 128 == 0 && (PT * sizeof(T)) % 128 == 0, "slot alignment");
    static_assert(NS >= 4, "ring depth");
    using V = Vec<T, VX>;

    extern __shared__ unsigned char smem_raw[];
    unsigned char* sbase =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    T* ys = reinterpret_cast<T*>(sbase);
    T* ps = ys + NS * YT;
    uint64_t* bar = reinterpret_cast<uint64_t*>(ps + NP * NPA * PT);

    // zrev: items and z-chunks in descending order, so that a launch starts on
    // the planes the previous launch (ascending) touched last, still in L2
    const int b = a.zrev ? (int)(gridDim.z - 1 - blockIdx.z) : (int)blockIdx.z;
    const int x0 = (blockIdx.x % a.tiles_x) * TX;
    const int y0 = (blockIdx.x / a.tiles_x) * TY;
    const int z0 = (a.zrev ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y) * a.zchunk;
    const int z1 = min(z0 + a.zchunk, a.nk);
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const int zb = b * a.pz + 2;  // padded plane index of interior z = 0 of item b
    const int ylast = z1 + 1;     // last stencil plane needed
    const bool leader = threadIdx.x == 0;

    pdl_trigger();  // the next kernel's CTAs may start as this grid's CTAs retire
    if (leader) {
        prefetch_tensormap(&tm_s);
#pragma unroll
        for (int i = 0; i < NS + NP; ++i) mbar_init(&bar[i], 1);
        fence_mbar_init();
    }
    __syncthreads();
    pdl_wait();     // fields written by the previous kernel are read from here on
    if (a.item_lo && b + a.item_base < *a.item_lo) return;  // the same for all threads of the CTA

    // tile t (interior plane, z0-2 <= t <= z1+1) -> slot (t - z0 + 2) % NS
    auto issue_y = [&](int t) {
        const int s = (t - z0 + 2) % NS;
        mbar_arrive_expect_tx(&bar[s], YBYTES);
        tma_load_3d(ys + s * YT, &tm_s, x0, y0, zb + t, &bar[s]);
    };
    auto issue_p = [&](int t) {
        const int s = (t - z0) % NP;
        mbar_arrive_expect_tx(&bar[NS + s], PBYTES);
        T* d = ps + s * NPA * PT;
        if constexpr (NPA > 0) tma_load_3d(d, &tm_p0, x0 + LX, y0 + 2, zb + t, &bar[NS + s]);
        if constexpr (NPA > 1) tma_load_3d(d + PT, &tm_p1, x0 + LX, y0 + 2, zb + t, &bar[NS + s]);
        if constexpr (NPA > 2) tma_load_3d(d + 2 * PT, &tm_p2, x0 + LX, y0 + 2, zb + t, &bar[NS + s]);
    };
    int y_hi = z0 - 3, p_hi = z0 - 1;  // highest tiles issued (leader only)
    if (leader) {
        for (int t = z0 - 2; t < z0 - 2 + NS && t <= ylast; ++t) { issue_y(t); y_hi = t; }
        if constexpr (NPA > 0)
            for (int t = z0; t < z0 + NP && t < z1; ++t) { issue_p(t); p_hi = t; }
    }

    // running ring positions: slot and phase of stencil tile z+2 (the next
    // centre), of tile z (x/y neighbours) and of pointwise tile z.  Shared
    // memory is read by 32-bit address with constant offsets, and the z-window
    // of centres lives in five registers renamed statically (the plane loop is
    // unrolled by five), so that no plane moves values between registers.
    constexpr int ES = (int)sizeof(T);
    const uint32_t ys_base = smem_u32(ys);
    const uint32_t ps_base = smem_u32(ps);
    const uint32_t own8 = (uint32_t)(((w + 2) * W + LX + lane * VX) * ES);  // this thread's centre
    const uint32_t pw8 = (uint32_t)((w * TX + lane * VX) * ES);
    int s_c = 0;
    uint32_t ph_c = 0;
    bool bad = false;
    auto next_center = [&]() -> V {
        if (!mbar_wait_bounded(&bar[s_c], ph_c)) bad = true;
        const V v = lds16<T>(ys_base + (uint32_t)s_c * YBYTES + own8);
        if (++s_c == NS) { s_c = 0; ph_c ^= 1u; }
        return v;
    };
    auto drain = [&](int y_done, int p_done) {
        if (!leader) return;
        for (int t = y_done + 1; t <= y_hi; ++t) {
            const int u = t - z0 + 2;
            (void)mbar_wait_bounded(&bar[u % NS], (uint32_t)((u / NS) & 1));
        }
        for (int t = p_done + 1; t <= p_hi; ++t)
            (void)mbar_wait_bounded(&bar[NS + (t - z0) % NP], (uint32_t)(((t - z0) / NP) & 1));
    };

    V cw[5];  // centres of planes z-2 .. z+2 at cw[(z - z0 + 0..4) % 5]
    cw[0] = next_center();
    cw[1] = next_center();
    cw[2] = next_center();
    cw[3] = next_center();
    if (__syncthreads_or(bad)) {
        if (leader) atomicExch(a.err, DEV_WAIT_TIMEOUT);
        drain(z0 + 1, z0 - 1);
        return;
    }
    if (leader) {
        fence_proxy_async_smem();
        for (int t = z0 - 2 + NS; t <= z0 - 1 + NS && t <= ylast; ++t) { issue_y(t); y_hi = t; }
    }

    const int y = y0 + w;
    const int x = x0 + lane * VX;
    const bool live = y < a.nj && x < a.ni;
    const bool full_vec = x + VX <= a.ni;
    // rows whose cells have no y image and vectors whose cells all lie inside
    // take the plain store (plus x images where a cell is within 2 of an x face)
    const bool x_img = x < 2 || x + VX > a.ni - 2;
    const bool y_img = y < 2 || y >= a.nj - 2 || !full_vec;
    const long long ob = (long long)b * a.item_stride + a.origin;
    T* yrow_out = a.yout + ob + (long long)z0 * a.plane + (long long)y * a.px + x;
    T* arow_out = nullptr;
    if constexpr (OpTraits<OP>::writes_a) arow_out = a.aout + ob + (long long)z0 * a.plane + (long long)y * a.px + x;
    double g[4] = {0., 0., 0., 0.};
    int s_n = 2 % NS;  // slot of tile z (neighbours)
    int s_p = 0;
    uint32_t ph_p = 0;

    // one plane; K = (z - z0) % 5 names the registers of the z-window
    auto iterate = [&](auto kc, int z) -> bool {
        constexpr int K = decltype(kc)::value;
        cw[(K + 4) % 5] = next_center();
        const V& cm2 = cw[K];
        const V& cm1 = cw[(K + 1) % 5];
        const V& c0 = cw[(K + 2) % 5];
        const V& cp1 = cw[(K + 3) % 5];
        const V& cp2 = cw[(K + 4) % 5];
        [[maybe_unused]] V p0v, p1v, p2v;
        if constexpr (NPA > 0) {
            if (!mbar_wait_bounded(&bar[NS + s_p], ph_p)) bad = true;
            const uint32_t P = ps_base + (uint32_t)s_p * (uint32_t)(NPA * PT * ES) + pw8;
            p0v = lds16<T>(P);
            if constexpr (NPA > 1) p1v = lds16<T, PT * ES>(P);
            if constexpr (NPA > 2) p2v = lds16<T, 2 * PT * ES>(P);
            if (++s_p == NP) { s_p = 0; ph_p ^= 1u; }
        }
        const uint32_t C = ys_base + (uint32_t)s_n * YBYTES + own8;
        if (++s_n == NS) s_n = 0;
        T row[3 * VX];
        {
            const V r0 = lds16<T, -LX * ES>(C), r2 = lds16<T, VX * ES>(C);  // c0: this plane's centre
#pragma unroll
            for (int e = 0; e < VX; ++e) { row[e] = r0.v[e]; row[VX + e] = c0.v[e]; row[2 * VX + e] = r2.v[e]; }
        }
        const V ym2 = lds16<T, -2 * W * ES>(C), ym1 = lds16<T, -W * ES>(C);
        const V yp1 = lds16<T, W * ES>(C), yp2 = lds16<T, 2 * W * ES>(C);
        V oy, oa;
#pragma unroll
        for (int e = 0; e < VX; ++e) {
            Nb<T> s;
            s.c = row[LX + e];
            s.xm1 = row[LX + e - 1]; s.xp1 = row[LX + e + 1];
            s.xm2 = row[LX + e - 2]; s.xp2 = row[LX + e + 2];
            s.ym1 = ym1.v[e]; s.yp1 = yp1.v[e]; s.ym2 = ym2.v[e]; s.yp2 = yp2.v[e];
            s.zm1 = cm1.v[e]; s.zp1 = cp1.v[e]; s.zm2 = cm2.v[e]; s.zp2 = cp2.v[e];
            [[maybe_unused]] T q0 = 0, q1 = 0, q2 = 0;
            if constexpr (NPA > 0) q0 = p0v.v[e];
            if constexpr (NPA > 1) q1 = p1v.v[e];
            if constexpr (NPA > 2) q2 = p2v.v[e];
            T vy = 0, va = 0;
            if constexpr (RK) {
                rk_update<T, OP>(a, rhs_w13(wt.w[NW == 1 ? 0 : b], s), s.c, q0, q1, vy, va);
            } else {
                cell_op<T, OP>(a, s, q0, q1, q2, vy, va, g, live && x + e < a.ni);
            }
            oy.v[e] = vy;
            oa.v[e] = va;
        }
        if (live) {
            if (!y_img && z >= 2 && z < a.nk - 2) {
                gst16<T>(a.sb_y, yrow_out, oy);
                if (x_img) {
#pragma unroll
                    for (int e = 0; e < VX; ++e) {
                        if (x + e < 2) gst1(a.sb_y, yrow_out + e + a.ni, oy.v[e]);
                        if (x + e >= a.ni - 2) gst1(a.sb_y, yrow_out + e - a.ni, oy.v[e]);
                    }
                }
            } else {
                store_images_vec<T, VX>(a.yout + ob, x, y, z, oy, a);
            }
            if constexpr (OpTraits<OP>::writes_a) {
                if (full_vec) gst16<T>(a.sb_a, arow_out, oa);
                else put_vec<T, VX>(a.sb_a, arow_out, x, a.ni, oa);
            }
        }
        yrow_out += a.plane;
        if constexpr (OpTraits<OP>::writes_a) arow_out += a.plane;
        if (__syncthreads_or(bad)) {
            if (leader) atomicExch(a.err, DEV_WAIT_TIMEOUT);
            drain(z + 2, z);
            return false;
        }
        if (leader) {
            fence_proxy_async_smem();
            if (z + NS <= ylast) { issue_y(z + NS); y_hi = z + NS; }
            if constexpr (NPA > 0)
                if (z + NP < z1) { issue_p(z + NP); p_hi = z + NP; }
        }
        return true;
    };
    for (int zz = z0; zz < z1; zz += 5) {
        if (!iterate(std::integral_constant<int, 0>{}, zz)) return;
        if (zz + 1 < z1 && !iterate(std::integral_constant<int, 1>{}, zz + 1)) return;
        if (zz + 2 < z1 && !iterate(std::integral_constant<int, 2>{}, zz + 2)) return;
        if (zz + 3 < z1 && !iterate(std::integral_constant<int, 3>{}, zz + 3)) return;
        if (zz + 4 < z1 && !iterate(std::integral_constant<int, 4>{}, zz + 4)) return;
    }
    if constexpr (OpTraits<OP>::adjoint) reduce_par(g, a.par_acc, a.gs_nu, a.gs_c);
}

// ---------------------------------------------------------------------------
// Host side of the stage launches.

namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

}  // namespace

bool make_tmap(CUtensorMap* tm, const Geo& g, const void* base, int items, int bw, int bh) {
    auto enc = encode_fn();
    if (!enc || !base) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)g.px, (cuuint64_t)g.py, (cuuint64_t)(g.pz * items)};
    const cuuint64_t strides[2] = {(cuuint64_t)(g.px * g.es), (cuuint64_t)(g.plane * g.es)};
    const cuuint32_t box[3] = {(cuuint32_t)bw, (cuuint32_t)bh, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapDataType dt = g.es == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    CUresult r = enc(tm, dt, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

namespace {

template <typename T>
KArgs<T> make_args(const Geo& g, const StageLaunch& L, const Shape& t, int* err) {
    KArgs<T> a{};
    a.yout = (T*)L.yout;
    a.yin = (const T*)L.yin;
    a.item_stride = g.total; a.origin = g.origin; a.px = g.px; a.plane = g.plane;
    a.ni = g.ni; a.nj = g.nj; a.nk = g.nk; a.pz = (int)g.pz;
    a.zchunk = t.zchunk;
    a.nzc = (g.nk + t.zchunk - 1) / t.zchunk;
    a.item_lo = L.item_lo;
    a.item_base = L.item_base;
    const Coef& c = L.coef;
    a.ca0 = (T)c.ca[0]; a.ca1 = (T)c.ca[1]; a.ca2 = (T)c.ca[2];
    a.u0 = (T)c.u[0]; a.u1 = (T)c.u[1]; a.u2 = (T)c.u[2];
    a.m0 = c.mode[0]; a.m1 = c.mode[1]; a.m2 = c.mode[2];
    a.nl = (T)(L.nu * (L.op == OP_EULER ? c.s2 : c.s4));
    a.c_y = (T)L.c_y; a.c_acc = (T)L.c_acc;
    a.err = err;
    // RK4 stages alternate the sweep direction (S1, S3 descending; S2, S4 ascending),
    // so that each stage starts on the planes the previous one touched last
    a.zrev = (L.op == OP_RK_S1 || L.op == OP_RK_S3) ? 1 : 0;
    a.sb_y = out_bounds(L.yout, g, L.items);
    switch (L.op) {
        case OP_RK_S1: break;
        case OP_RK_S2: a.aout = (T*)L.acc; a.pw0 = (const T*)L.q; break;
        case OP_RK_S3: a.pw0 = (const T*)L.q; break;
        case OP_RK_S4: a.pw0 = (const T*)L.acc; a.pw1 = (const T*)L.q; break;
        case OP_EULER: break;
        case OP_ADJ + 0: a.aout = (T*)L.lam_acc; a.pw0 = (const T*)L.ypt; break;
        case OP_ADJ + 1:
        case OP_ADJ + 2:
            a.aout = (T*)L.lam_acc; a.pw0 = (const T*)L.ypt; a.pw1 = (const T*)L.lam; a.pw2 = (const T*)L.lam_acc;
            break;
        case OP_ADJ + 3: a.pw0 = (const T*)L.ypt; a.pw1 = (const T*)L.lam_acc; break;
        default: break;
    }
    a.sb_a = out_bounds(a.aout, g, L.items);
    if (L.op >= OP_ADJ) {
        a.c_y = (T)L.c_ybar;
        a.c_acc = (T)L.c_lam;
        a.sigma = (T)L.sigma;
        a.par_acc = L.par_acc;
        a.gs_nu = L.dnu * L.sigma * c.s4;   // nu-sum * dnu * sigma / (12 dx^2)
        a.gs_c = -L.sigma / (12. * c.dx);   // c-sums: -sigma * D_d m = -sigma (8d1-d2)/(12dx)
    }
    return a;
}

template <typename T, int OP, int NW>
cudaError_t launch_direct_T(const Geo& g, const StageLaunch& L, KArgs<T> a, const Shape& t, cudaStream_t s) {
    if (t.ty != 4 && t.ty != 8 && t.ty != 16) return cudaErrorInvalidValue;
    const unsigned threads = 32u * (unsigned)t.ty;
    a.tiles_x = (g.ni + V16<T>::N - 1) / V16<T>::N;
    const long long chunks = (long long)a.tiles_x * g.nj;
    const dim3 grid((unsigned)((chunks + threads - 1) / threads), (unsigned)a.nzc, (unsigned)L.items);
    if (chunks > 0x7fffffffLL || grid.y > 65535u || grid.z > 65535u) return cudaErrorInvalidConfiguration;
    Weights<T, NW> wt;
    fill_weights(wt, L.coef, L.nu, L.nu_items, L.items);
    auto run = [&](auto k) { return launch_in_stream(!L.drain, k, grid, dim3(threads), 0, s, a, wt); };
    if (L.wrap) {
        constexpr int ZMAX = OpTraits<OP>::adjoint ? 2 : 4;  // (adjoint stages: 80-86 registers)
        switch (std::min(t.zchunk, ZMAX)) {
            case 1: return run(k_stage_wrap<T, OP, NW, 1>);
            case 2: return run(k_stage_wrap<T, OP, NW, 2>);
            case 3: return run(k_stage_wrap<T, OP, NW, std::min(3, ZMAX)>);
            default: return run(k_stage_wrap<T, OP, NW, ZMAX>);
        }
    }
    return run(k_stage_direct<T, OP, NW>);
}

template <typename T, int OP, int TY, int NS, int NP>
size_t tma_smem_bytes() {
    constexpr int VX = V16<T>::N, TX = 32 * VX, W = TX + 2 * VX, H = TY + 4;
    constexpr int NPA = OpTraits<OP>::npw;
    return 128 + (size_t)NS * W * H * sizeof(T) + (size_t)NP * NPA * TX * TY * sizeof(T) + (NS + NP) * 8;
}

template <typename T, int OP, int NW, int TY, int NS, int NP>
cudaError_t launch_tma_T(const Geo& g, const StageLaunch& L, KArgs<T> a, const Shape& t, cudaStream_t s) {
    constexpr int VX = V16<T>::N, TX = 32 * VX, W = TX + 2 * VX, H = TY + 4;
    CUtensorMap ts{}, t0{}, t1{}, t2{};
    if (!make_tmap(&ts, g, L.yin, L.items, W, H)) return cudaErrorInvalidValue;
    const void* pw[3] = {a.pw0, a.pw1, a.pw2};
    CUtensorMap* tp[3] = {&t0, &t1, &t2};
    for (int i = 0; i < OpTraits<OP>::npw; ++i)
        if (!make_tmap(tp[i], g, pw[i], L.items, TX, TY)) return cudaErrorInvalidValue;
    a.tiles_x = (g.ni + TX - 1) / TX;
    const int tiles_y = (g.nj + TY - 1) / TY;
    dim3 grid(a.tiles_x * tiles_y, a.nzc, L.items);
    if (grid.y > 65535u || grid.z > 65535u) return cudaErrorInvalidConfiguration;
    const size_t smem = tma_smem_bytes<T, OP, TY, NS, NP>();
    Weights<T, NW> wt;
    fill_weights(wt, L.coef, L.nu, L.nu_items, L.items);
    return launch_pdl(k_stage_tma<T, OP, TY, NS, NP, NW>, grid, dim3(32 * TY), smem, s, ts, t0, t1, t2, a, wt);
}

template <typename T, int OP, int NW, int TY, int NS, int NP>
cudaError_t set_attr_T() {
    return cudaFuncSetAttribute(k_stage_tma<T, OP, TY, NS, NP, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tma_smem_bytes<T, OP, TY, NS, NP>());
}

template <typename T, int OP, int NW = 1>
cudaError_t set_attr_op() {
    cudaError_t e = set_attr_T<T, OP, NW, 4, 5, 3>();
    if (e == cudaSuccess) e = set_attr_T<T, OP, NW, 8, 5, 3>();
    if (e == cudaSuccess) e = set_attr_T<T, OP, NW, 16, 4, 2>();
    return e;
}


// Ring depths per tile height: NS stencil slots (prefetch NS-3 planes ahead),
// NP pointwise slots (prefetch NP-1 planes ahead).
template <typename T, int OP, int NW>
cudaError_t launch_op(const Geo& g, const StageLaunch& L, const Shape& t, cudaStream_t s, int* err) {
    if (L.wrap && (t.tma || !wrap_supported(g))) return cudaErrorInvalidValue;
    const KArgs<T> a = make_args<T>(g, L, t, err);
    for (const void* p : {(const void*)a.yin, (const void*)a.yout, (const void*)a.aout, (const void*)a.pw0,
                          (const void*)a.pw1, (const void*)a.pw2})
        if (!aligned16(p)) return cudaErrorInvalidValue;
    if (!t.tma) return launch_direct_T<T, OP, NW>(g, L, a, t, s);
    switch (t.ty) {
        case 4: return launch_tma_T<T, OP, NW, 4, 5, 3>(g, L, a, t, s);
        case 8: return launch_tma_T<T, OP, NW, 8, 5, 3>(g, L, a, t, s);
        case 16: return launch_tma_T<T, OP, NW, 16, 4, 2>(g, L, a, t, s);
        default: return cudaErrorInvalidValue;
    }
}

template <typename T>
cudaError_t launch_T(const Geo& g, const StageLaunch& L, const Shape& t, cudaStream_t s, int* err) {
    if constexpr (sizeof(T) == 8) {
        switch (L.nu_items ? L.op : -1) {
            case -1: break;
            case OP_RK_S1: return launch_op<T, OP_RK_S1, kItemWeights>(g, L, t, s, err);
            case OP_RK_S2: return launch_op<T, OP_RK_S2, kItemWeights>(g, L, t, s, err);
            case OP_RK_S3: return launch_op<T, OP_RK_S3, kItemWeights>(g, L, t, s, err);
            case OP_RK_S4: return launch_op<T, OP_RK_S4, kItemWeights>(g, L, t, s, err);
            default: return cudaErrorInvalidValue;
        }
    } else if (L.nu_items) {
        return cudaErrorInvalidValue;
    }
    switch (L.op) {
        case OP_RK_S1: return launch_op<T, OP_RK_S1, 1>(g, L, t, s, err);
        case OP_RK_S2: return launch_op<T, OP_RK_S2, 1>(g, L, t, s, err);
        case OP_RK_S3: return launch_op<T, OP_RK_S3, 1>(g, L, t, s, err);
        case OP_RK_S4: return launch_op<T, OP_RK_S4, 1>(g, L, t, s, err);
        case OP_EULER: return launch_op<T, OP_EULER, 1>(g, L, t, s, err);
        default: break;
    }
    if constexpr (sizeof(T) == 8) {
        switch (L.op) {
            case OP_ADJ + 0: return launch_op<T, OP_ADJ + 0, 1>(g, L, t, s, err);
            case OP_ADJ + 1: return launch_op<T, OP_ADJ + 1, 1>(g, L, t, s, err);
            case OP_ADJ + 2: return launch_op<T, OP_ADJ + 2, 1>(g, L, t, s, err);
            case OP_ADJ + 3: return launch_op<T, OP_ADJ + 3, 1>(g, L, t, s, err);
            default: break;
        }
    }
    return cudaErrorInvalidValue;
}

}  // namespace

unsigned long long take_store_violations_stages() {
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_store_violations, sizeof v) != cudaSuccess) return 0;
    const unsigned int zero = 0;
    cudaMemcpyToSymbol(g_store_violations, &zero, sizeof zero);
    return v;
}

cudaError_t prepare_kernels(bool per_item) {
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    chk(set_attr_op<double, OP_RK_S1>()); chk(set_attr_op<double, OP_RK_S2>());
    chk(set_attr_op<double, OP_RK_S3>()); chk(set_attr_op<double, OP_RK_S4>());
    chk(set_attr_op<double, OP_EULER>());
    if (per_item) {
        chk(set_attr_op<double, OP_RK_S1, kItemWeights>()); chk(set_attr_op<double, OP_RK_S2, kItemWeights>());
        chk(set_attr_op<double, OP_RK_S3, kItemWeights>()); chk(set_attr_op<double, OP_RK_S4, kItemWeights>());
    }
    chk(set_attr_op<double, OP_ADJ + 0>()); chk(set_attr_op<double, OP_ADJ + 1>());
    chk(set_attr_op<double, OP_ADJ + 2>()); chk(set_attr_op<double, OP_ADJ + 3>());
    chk(set_attr_op<float, OP_RK_S1>()); chk(set_attr_op<float, OP_RK_S2>());
    chk(set_attr_op<float, OP_RK_S3>()); chk(set_attr_op<float, OP_RK_S4>());
    chk(set_attr_op<float, OP_EULER>());
    chk(prepare_pairs(per_item));
    return e;
}

namespace {
// Self-test of the bounded waits: one CTA waits on an mbarrier that nothing
// arrives on, gives up after limit_ns like every pipeline wait, records the
// timeout in the device error word and returns.
__global__ void k_wait_selftest(int* err, unsigned long long limit_ns) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    const bool ok = mbar_wait_bounded(&bar, 0, limit_ns);
    if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicExch(err, DEV_WAIT_TIMEOUT);
}
}  // namespace

cudaError_t launch_wait_selftest(int* err, unsigned long long limit_ns, cudaStream_t s) {
    add_launches(1);
    k_wait_selftest<<<1, 64, 0, s>>>(err, limit_ns);
    return cudaGetLastError();
}

// The direct kernel up to a number of cells per launch, the TMA rings beyond.
// Where the lines lie (us per RK4 step, direct / TMA): FP64 8 fields of 64^3 (2.1M
// cells) 58 / 60, 16 of them 126 / 114, one 192^3 175 / 159; FP32 192^3 (7.1M) 102 /
// 112, 256^3 234 / 204; adjoint (a whole gradient, per step) 96^3 90 / 115, 128^3
// 193 / 177.  The direct kernel takes as
// many planes per thread as give one wave of threads (FP64 95 x 97 x 93: 3 planes
// 24.0, 2 planes 26.7; FP32 1 plane 19.9, 2 planes 22.4), at most four (longer
// chunks gained nothing at 128^3-192^3); its wrapping form two planes beyond one
// wave (FP64 100^3: 1, 2, 3, 4 planes 28.9, 27.4, 31.5, 32.5; 128^3 54.7, 49.0, 49.8,
// 52.7; FP32 128^3 29, 27.4, 28.7, 31).
bool wrap_supported(const Geo& g) { return g.ni % (16 / g.es) == 0 && g.plane * g.es <= 0xffffffffLL; }

Shape default_stage_shape(const Geo& g, int items, bool adjoint) {
    const long long direct = adjoint ? 1'500'000 : (g.es == 8 ? 3'000'000 : 12'000'000);
    const long long cells = (long long)g.ni * g.nj * g.nk * items;
    const int n = 16 / g.es;
    Shape sh;
    if (cells <= direct) {
        const long long threads = (long long)((g.ni + n - 1) / n) * g.nj * g.nk * items;
        const long long wave = 148LL * (g.es == 8 ? 1024 : 1792);
        sh.tma = 0;
        const bool wrap = wrap_supported(g);
        sh.ty = g.es == 8 && !wrap ? 8 : 4;
        // (no shorter than the launch grid's limit of 65535 chunks allows)
        sh.zchunk = (int)std::max(std::min(wrap ? 2LL : 4LL, (threads + wave - 1) / wave), (g.nk + 65534) / 65535LL);
        return sh;
    }
    // TMA rings: 4-row tiles, z-chunks that give at least ~8 CTAs per SM
    sh.ty = 4;
    const long long tiles = (long long)((g.ni + 32 * n - 1) / (32 * n)) * ((g.nj + 3) / 4) * items;
    int zc = g.nk;
    while (zc > 8 && tiles * ((g.nk + zc - 1) / zc) < 148LL * 8) zc = (zc + 1) / 2;
    sh.zchunk = zc;
    return sh;
}

cudaError_t launch_stage(const Geo& g, const StageLaunch& L, const Tune& t, cudaStream_t s, int* err) {
    if (L.op < 0 || L.op >= kNumOps) return cudaErrorInvalidValue;
    const Shape& sh = t.op[L.op];
    auto launch = [&](const StageLaunch& l) {
        add_launches(1);
        return l.prec == 0 ? launch_T<double>(g, l, sh, s, err) : launch_T<float>(g, l, sh, s, err);
    };
    if (!L.nu_items || L.items <= kItemWeights) return launch(L);
    for (int b = 0; b < L.items; b += kItemWeights) {
        StageLaunch l = L;
        auto at = [&](auto* p) { return p ? (decltype(p))((const char*)p + (size_t)b * g.total * g.es) : p; };
        l.items = std::min(kItemWeights, L.items - b);
        l.nu_items = L.nu_items + b;
        l.item_base = L.item_base + b;
        l.yin = at(L.yin); l.q = at(L.q); l.acc = at(L.acc); l.yout = at(L.yout);
        const cudaError_t e = launch(l);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Pointwise kernels.

// Periodicity: what the three passes of Periodicity.cu:12-144 (I, then J over all
// I, then K over all I and J) leave in the halo, here in one launch: every halo
// cell is the interior cell at its wrapped indices, so nothing written is read.
// A warp takes one row of the padded box, all of it outside the interior's rows,
// the four x-halo cells inside.  The launches are what it costs (a call on 24^3
// had three of ~2 us each in its chain).
template <typename T>
__global__ void __launch_bounds__(256) k_periodicity(T* f, Geo g) {
    pdl_trigger();
    pdl_wait();
    const int rows_j = g.nj + 4;
    const long long rows = (long long)rows_j * (g.nk + 4);
    T* base = f + (long long)blockIdx.y * g.total + g.origin;
    const int lane = threadIdx.x & 31;
    for (long long r = blockIdx.x * 8LL + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8LL) {
        const int k = (int)(r / rows_j) - 2, j = (int)(r % rows_j) - 2;
        const int ks = k < 0 ? k + g.nk : (k >= g.nk ? k - g.nk : k);
        const int js = j < 0 ? j + g.nj : (j >= g.nj ? j - g.nj : j);
        T* dst = base + k * g.plane + j * g.px;
        const T* src = base + ks * g.plane + js * g.px;
        if (k == ks && j == js) {
            if (lane < 4) {
                const int x = lane < 2 ? lane - 2 : g.ni + lane - 2;
                dst[x] = src[x < 0 ? x + g.ni : x - g.ni];
            }
        } else {
            for (int x = lane - 2; x < g.ni + 2; x += 32)
                dst[x] = src[x < 0 ? x + g.ni : (x >= g.ni ? x - g.ni : x)];
        }
    }
}

static unsigned grid_for(long long n, int block) {
    long long b = (n + block - 1) / block;
    if (b > 148LL * 64) b = 148LL * 64;
    if (b < 1) b = 1;
    return (unsigned)b;
}

cudaError_t launch_periodicity(const Geo& g, void* field, int items, cudaStream_t s) {
    add_launches(1);
    if (items < 1 || items > 65535) return cudaErrorInvalidValue;
    const dim3 grid(grid_for((long long)(g.nj + 4) * (g.nk + 4), 8), (unsigned)items);
    if (g.es == 8) return launch_pdl(k_periodicity<double>, grid, dim3(256), 0, s, static_cast<double*>(field), g);
    return launch_pdl(k_periodicity<float>, grid, dim3(256), 0, s, static_cast<float*>(field), g);
}

// Adds the block's sums to acc[0 .. N-1] (and, for the maxima, takes the larger)
// with one atomic per block and value.  One atomic per warp and value put 65 536
// updates on the same address for a 128^3 field and held the correction at
// 212 us, whose memory traffic takes 10.  Every thread of the block must call it.
__device__ __forceinline__ void atomic_max_nonneg(double* p, double v) {
    // non-negative doubles order like their bit patterns
    atomicMax(reinterpret_cast<unsigned long long*>(p), (unsigned long long)__double_as_longlong(v));
}

template <int NSUM, int NMAX>
__device__ __forceinline__ void block_accumulate(double (&v)[NSUM + NMAX], double* acc) {
    constexpr int N = NSUM + NMAX;
    __shared__ double red[kColY][N];
#pragma unroll
    for (int i = 0; i < N; ++i)
        for (int o = 16; o > 0; o >>= 1) {
            const double w = __shfl_xor_sync(0xffffffffu, v[i], o);
            v[i] = i < NSUM ? v[i] + w : fmax(v[i], w);
        }
    if (threadIdx.x == 0)
#pragma unroll
        for (int i = 0; i < N; ++i) red[threadIdx.y][i] = v[i];
    __syncthreads();
    if (threadIdx.y == 0 && threadIdx.x < N) {
        const int i = threadIdx.x;
        double t = red[0][i];
#pragma unroll
        for (int w = 1; w < kColY; ++w) t = i < NSUM ? t + red[w][i] : fmax(t, red[w][i]);
        if (i < NSUM) atomicAdd(acc + i, t);
        else atomic_max_nonneg(acc + i, t);
    }
}

// Writes v at interior (x,y,z) of a field (origin-relative base) plus images.
template <typename T>
__device__ __forceinline__ void put_img(T* base, const Geo& g, int x, int y, int z, T v) {
    T* row = base + (long long)z * g.plane + (long long)y * g.px;
    row[x] = v;
    if (x < 2) row[x + g.ni] = v;
    if (x >= g.ni - 2) row[x - g.ni] = v;
    if (y < 2) row[(long long)g.nj * g.px + x] = v;
    if (y >= g.nj - 2) row[-(long long)g.nj * g.px + x] = v;
    if (z < 2) row[(long long)g.nk * g.plane + x] = v;
    if (z >= g.nk - 2) row[-(long long)g.nk * g.plane + x] = v;
}

template <typename TD, typename TF>
__global__ void __launch_bounds__(kColX * kColY) k_dense_to_field(const TD* d, TF* f, Geo g) {
    for_column(g, [&](int x, int y, int z) {
        put_img<TF>(f + g.origin, g, x, y, z, (TF)d[((long long)z * g.nj + y) * g.ni + x]);
    });
}

template <typename TF, typename TD>
__global__ void __launch_bounds__(kColX * kColY) k_field_to_dense(const TF* f, TD* d, Geo g) {
    for_column(g, [&](int x, int y, int z) { d[((long long)z * g.nj + y) * g.ni + x] = (TD)f[cell_at(g, x, y, z)]; });
}

cudaError_t launch_dense_to_field(const Geo& g, const void* dense, int dense_prec, void* field, cudaStream_t s) {
    add_launches(1);
    const dim3 gr = column_grid(g), bl(kColX, kColY);
    if (g.es == 8) {
        if (dense_prec == 0) k_dense_to_field<double, double><<<gr, bl, 0, s>>>((const double*)dense, (double*)field, g);
        else k_dense_to_field<float, double><<<gr, bl, 0, s>>>((const float*)dense, (double*)field, g);
    } else {
        if (dense_prec == 0) k_dense_to_field<double, float><<<gr, bl, 0, s>>>((const double*)dense, (float*)field, g);
        else k_dense_to_field<float, float><<<gr, bl, 0, s>>>((const float*)dense, (float*)field, g);
    }
    return cudaGetLastError();
}

cudaError_t launch_field_to_dense(const Geo& g, const void* field, void* dense, int dense_prec, cudaStream_t s) {
    add_launches(1);
    const dim3 gr = column_grid(g), bl(kColX, kColY);
    if (g.es == 8) {
        if (dense_prec == 0) k_field_to_dense<double, double><<<gr, bl, 0, s>>>((const double*)field, (double*)dense, g);
        else k_field_to_dense<double, float><<<gr, bl, 0, s>>>((const double*)field, (float*)dense, g);
    } else {
        if (dense_prec == 0) k_field_to_dense<float, double><<<gr, bl, 0, s>>>((const float*)field, (double*)dense, g);
        else k_field_to_dense<float, float><<<gr, bl, 0, s>>>((const float*)field, (float*)dense, g);
    }
    return cudaGetLastError();
}

template <typename TD, typename TS>
__global__ void __launch_bounds__(kColX * kColY)
    k_convert(TD* dst, Geo gd, const TS* src, Geo gs, const int* item_lo, int item) {
    if (item_lo && item < *item_lo) return;
    for_column(gd, [&](int x, int y, int z) {
        put_img<TD>(dst + gd.origin, gd, x, y, z, (TD)src[cell_at(gs, x, y, z)]);
    });
}

cudaError_t launch_convert(const Geo& gd, void* dst, const Geo& gs, const void* src, cudaStream_t s,
                           const int* item_lo, int item) {
    add_launches(1);
    const dim3 gr = column_grid(gd), bl(kColX, kColY);
    if (gd.es == 8 && gs.es == 8)
        k_convert<double, double><<<gr, bl, 0, s>>>((double*)dst, gd, (const double*)src, gs, item_lo, item);
    else if (gd.es == 8)
        k_convert<double, float><<<gr, bl, 0, s>>>((double*)dst, gd, (const float*)src, gs, item_lo, item);
    else if (gs.es == 8)
        k_convert<float, double><<<gr, bl, 0, s>>>((float*)dst, gd, (const double*)src, gs, item_lo, item);
    else
        k_convert<float, float><<<gr, bl, 0, s>>>((float*)dst, gd, (const float*)src, gs, item_lo, item);
    return cudaGetLastError();
}

// Parareal correction (UpdateStage, Parareal.h:19-35) fused with the swap of
// the coarse states (Parareal.h:164) and the defect norms.  Bound by memory:
// 128^3 with an FP32 G in the increment form (below) moves 67 MB and took
// 212 us, now 20; the FP64 form at 64^3 31 us, now 6.5.
template <typename TC>
__global__ void __launch_bounds__(kColX * kColY)
    k_update(const TC* gnew, const double* f, TC* gold, double* u, double* def, Geo g, Geo gc, const int* item_lo,
             int item) {
    if (item_lo && item < *item_lo) return;
    double s[2] = {0., 0.};  // sum (U+ - U)^2, sum U+^2
    for_column(g, [&](int x, int y, int z) {
        const long long o = cell_at(g, x, y, z), oc = cell_at(gc, x, y, z);
        const TC gn = gnew[oc];
        const double q = ((double)gn + f[o]) - (double)gold[oc];
        const double d = q - u[o];
        s[0] += d * d;
        s[1] += q * q;
        gold[oc] = gn;
        put_img<double>(u + g.origin, g, x, y, z, q);
    });
    block_accumulate<2, 0>(s, def);
}

cudaError_t launch_update(const Geo& g64, const Geo& gc, const void* gnew, const double* f, void* gold,
                          double* u_next, double* def, const int* item_lo, int item, cudaStream_t s) {
    add_launches(1);
    const dim3 gr = column_grid(g64), bl(kColX, kColY);
    if (gc.es == 8)
        k_update<double><<<gr, bl, 0, s>>>((const double*)gnew, f, (double*)gold, u_next, def, g64, gc, item_lo, item);
    else
        k_update<float><<<gr, bl, 0, s>>>((const float*)gnew, f, (float*)gold, u_next, def, g64, gc, item_lo, item);
    return cudaGetLastError();
}

// Increment form of the correction (linear G): U_{r+1} = F_r + G(delta_r),
// delta_{r+1} = U_{r+1}^new - U_{r+1}^old written, in coarse precision and with
// its periodic images, as the next slice's coarse input; defect sums as k_update.
template <typename TC>
__global__ void __launch_bounds__(kColX * kColY)
    k_update_delta(const TC* gd, const double* f, double* u, TC* dnext, double* def, Geo g, Geo gc, const int* item_lo,
                   int item) {
    if (item_lo && item < *item_lo) return;
    double s[2] = {0., 0.};
    for_column(g, [&](int x, int y, int z) {
        const long long o = cell_at(g, x, y, z);
        const double q = f[o] + (double)gd[cell_at(gc, x, y, z)];
        const double d = q - u[o];
        s[0] += d * d;
        s[1] += q * q;
        put_img<double>(u + g.origin, g, x, y, z, q);
        put_img<TC>(dnext + gc.origin, gc, x, y, z, (TC)d);
    });
    block_accumulate<2, 0>(s, def);
}

cudaError_t launch_update_delta(const Geo& g64, const Geo& gc, const void* gd, const double* f, double* u_next,
                                void* d_next, double* def, const int* item_lo, int item, cudaStream_t s) {
    add_launches(1);
    const dim3 gr = column_grid(g64), bl(kColX, kColY);
    if (gc.es == 8)
        k_update_delta<double><<<gr, bl, 0, s>>>((const double*)gd, f, u_next, (double*)d_next, def, g64, gc, item_lo,
                                                 item);
    else
        k_update_delta<float><<<gr, bl, 0, s>>>((const float*)gd, f, u_next, (float*)d_next, def, g64, gc, item_lo,
                                                item);
    return cudaGetLastError();
}

// Zeroes field number *item_lo (if in [min_item, nitems)) of an array of fields of `bytes` each.
__global__ void k_zero_item(unsigned char* base, long long bytes, int nitems, const int* item_lo, int min_item) {
    const int it = *item_lo;
    if (it < min_item || it >= nitems) return;
    ulonglong2* p = reinterpret_cast<ulonglong2*>(base + (long long)it * bytes);
    const long long n = bytes / 16;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        p[t] = make_ulonglong2(0ull, 0ull);
}

cudaError_t launch_zero_item(void* base, long long bytes, int nitems, const int* item_lo, cudaStream_t s,
                             int min_item) {
    add_launches(1);
    k_zero_item<<<grid_for(bytes / 16, 256), 256, 0, s>>>(static_cast<unsigned char*>(base), bytes, nitems, item_lo,
                                                         min_item);
    return cudaGetLastError();
}

// Relative errors of two fields, bound by reading both once (100^3: 131 us, now 8.5).
__global__ void __launch_bounds__(kColX * kColY) k_errors(const double* a, const double* b, double* acc, Geo g) {
    double v[4] = {0., 0., 0., 0.};  // sum (a-b)^2, sum b^2, max |a-b|, max |a|
    for_column(g, [&](int x, int y, int z) {
        const long long o = cell_at(g, x, y, z);
        const double va = a[o], vb = b[o], d = va - vb;
        v[0] += d * d;
        v[1] += vb * vb;
        v[2] = fmax(v[2], fabs(d));
        v[3] = fmax(v[3], fabs(va));
    });
    block_accumulate<2, 2>(v, acc);
}

cudaError_t launch_errors(const Geo& g, const double* a, const double* b, double* acc4, cudaStream_t s) {
    add_launches(1);
    k_errors<<<column_grid(g), dim3(kColX, kColY), 0, s>>>(a, b, acc4, g);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(kColX * kColY)
    k_misfit(const double* a, const double* b, double* lam, double* jacc, Geo g) {
    double s[1] = {0.};
    for_column(g, [&](int x, int y, int z) {
        const long long o = cell_at(g, x, y, z);
        const double d = a[o] - b[o];
        s[0] += 0.5 * d * d;
        put_img<double>(lam + g.origin, g, x, y, z, d);
    });
    block_accumulate<1, 0>(s, jacc);
}

cudaError_t launch_misfit(const Geo& g, const double* a, const double* b, double* lam, double* jacc, cudaStream_t s) {
    add_launches(1);
    k_misfit<<<column_grid(g), dim3(kColX, kColY), 0, s>>>(a, b, lam, jacc, g);
    return cudaGetLastError();
}

}  // namespace sp
