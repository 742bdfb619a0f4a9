// mhd_kernels.cuh -- sm_100a kernels of the RK4 Hall-MHD step (reference: t3dsdsc.f).
//
// Storage: structure-of-arrays, one array per field, node (i,j,k) at i + mx*(j + my*k),
// no ghost nodes.  x and y are periodic (index wrap); z rows 0,1,mz-2,mz-1 are the wall
// rows of the reference (outer row 0, next row one half of its inner neighbour).
// Every field is stored as the perturbation from the FP64 z-profile equilibrium
// (rho0, B0, p0; momentum has no equilibrium part), in type T (double or float).
//
// Each kernel is launched on a 3-D grid: blockIdx.x covers x in chunks of blockDim.x,
// blockIdx.y = j, blockIdx.z = k, so a warp reads consecutive x (coalesced).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"

namespace dasha {

constexpr int NF = 8;

template <class T>
struct Geo {
    int mx, my, mz;
    long sy, sz;
    // 4th-order first / second derivative coefficients (t3dsdsc.f:336-504), zero where the
    // reference leaves them undefined (z rows outside 2..mz-3)
    const T *a1x, *b1x, *c1x, *d1x, *a1y, *b1y, *c1y, *d1y, *a1z, *b1z, *c1z, *d1z;
    const T *a2x, *b2x, *c2x, *d2x, *a2y, *b2y, *c2y, *d2y, *a2z, *b2z, *c2z, *d2z;
    // difc weights: difc = (f+ - f0)*wp - (f0 - f-)*wm  (t3dsdsc.f:5618-5619)
    const T *wpx, *wmx, *wpy, *wmy, *wpz, *wmz;
    const T *cbx;    // (1/32)(1 - tanh((x+3)/8)), smoothing coefficient of B (t3dsdsc.f:5636-5642)
    const T* cr;     // FP64 contexts: the radial coefficient below at every node, made once (k_radial_field)
    const T *xc, *yc, *zc;   // node coordinates: the radial coefficient 1/32 + 3/32 (1 + tanh((r-3)/3))/2
                             // (t3dsdsc.f:5659-5661); FP32 passes evaluate it per node
    // equilibrium z-profiles (FP64)
    const double *rho0, *bx0, *by0, *bz0, *p0;
    const double *dzp0;               // Dz p0 (interior rows)
    const double *d2rho0, *d2p0;      // D2z rho0, D2z p0 (interior rows)
    const double *rsx, *rsy, *rsz;    // xresd profiles (interior rows)
    const double *j0x, *j0y, *j0z;    // J0 profiles for j0_mode FULL (null otherwise)
    const double *dzp0r;              // Dz p0 / rho0 (interior rows)
    T eta, di, gamma, mu, drho, dp;
    int hall, viscos, diffu;
    // first plane of setdt's region: 0, except on a z-slab above the lowest one, whose planes 0
    // and 1 are ghost copies of the slab below (halo.h)
    int kcfl0;
};

template <class T>
struct F8 { T* f[NF]; };
template <class T>
struct F3 { T* f[3]; };

__device__ __forceinline__ int wrapi(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// -DDASHA_BOUNDS (a checking build for tests): the z-marching kernels test every global node
// span they load or store against the field extent n; the first violation of a launch is kept
// in g_bounds_hit as (site + 1) << 48 | index, the access is skipped (no trap, no fault), and the
// C-ABI call that launched it returns DASHA_E_CUDA naming the site and index.  In the normal
// build DASHA_SPAN is `true` and costs nothing.
enum BoundsSite {
    BS_ZPV_LOAD, BS_ZPV_STORE, BS_ZPV_WALL_LOAD, BS_ZPV2_LOAD, BS_ZPV2_STORE, BS_ZCURL_LOAD, BS_ZCURL_STORE,
    BS_ZHYDRO_LOAD, BS_ZHYDRO_NODE_LOAD, BS_ZHYDRO_STORE, BS_ZEH_LOAD, BS_ZEH_NODE_LOAD, BS_ZEH_STORE, BS_COUNT
};
#ifdef DASHA_BOUNDS
static __device__ unsigned long long g_bounds_hit;
__device__ __forceinline__ bool dasha_span(long first, long count, long n, int site) {
    if (first >= 0 && first + count <= n) return true;
    atomicCAS(&g_bounds_hit, 0ull, ((unsigned long long)(site + 1) << 48) | ((unsigned long long)first & 0xFFFFFFFFFFFFull));
    return false;
}
#define DASHA_SPAN(first, count, n, site) dasha_span((long)(first), (long)(count), (long)(n), (int)(site))
#else
#define DASHA_SPAN(first, count, n, site) true
#endif

template <class T>
__device__ __forceinline__ T d1fc(T fm2, T fm, T f0, T fp, T fp2, T a, T b, T c, T d) {
    return a * (fp - f0) + b * (f0 - fm) + c * (fp2 - f0) + d * (f0 - fm2);
}

// d1fc on two FP32 values at once (packed FADD2 / FMUL2 / FFMA2 on sm_100): a (fp - f0), then
// + b (f0 - fm), + c (fp2 - f0), + d (f0 - fm2) by fused multiply-adds.  (Spelling the scalar
// form the same way made the FP64 hydro RHS 25 % slower on B200: one serial chain of DFMAs.)
__device__ __forceinline__ float2 neg2(float2 v) { return make_float2(-v.x, -v.y); }
__device__ __forceinline__ float2 d1fc2(float2 fm2, float2 fm, float2 f0, float2 fp, float2 fp2, float2 a, float2 b,
                                        float2 c, float2 d) {
    float2 t = __fmul2_rn(a, __fadd2_rn(fp, neg2(f0)));
    t = __ffma2_rn(b, __fadd2_rn(f0, neg2(fm)), t);
    t = __ffma2_rn(c, __fadd2_rn(fp2, neg2(f0)), t);
    return __ffma2_rn(d, __fadd2_rn(f0, neg2(fm2)), t);
}
__device__ __forceinline__ float2 bc2(float v) { return make_float2(v, v); }

// 1/v rounded to nearest: the same value as the IEEE division 1/v, without its slow path
__device__ __forceinline__ float recip(float v) { return __frcp_rn(v); }
__device__ __forceinline__ double recip(double v) { return __drcp_rn(v); }

// Stencil helper: neighbour offsets of node (i,j,k) in a periodic-x/y, bounded-z array.
template <class T>
struct Nbr {
    long c;              // centre
    long xm2, xm1, xp1, xp2, ym2, ym1, yp1, yp2;   // absolute indices
    int i, j, k;
    __device__ __forceinline__ Nbr(const Geo<T>& g, int i_, int j_, int k_) : i(i_), j(j_), k(k_) {
        long row = (long)j * g.sy + (long)k * g.sz;
        c = row + i;
        xm2 = row + wrapi(i - 2, g.mx); xm1 = row + wrapi(i - 1, g.mx);
        xp1 = row + wrapi(i + 1, g.mx); xp2 = row + wrapi(i + 2, g.mx);
        long col = (long)i + (long)k * g.sz;
        ym2 = col + (long)wrapi(j - 2, g.my) * g.sy; ym1 = col + (long)wrapi(j - 1, g.my) * g.sy;
        yp1 = col + (long)wrapi(j + 1, g.my) * g.sy; yp2 = col + (long)wrapi(j + 2, g.my) * g.sy;
    }
    __device__ __forceinline__ T Dx(const Geo<T>& g, const T* f) const {
        return d1fc(f[xm2], f[xm1], f[c], f[xp1], f[xp2], g.a1x[i], g.b1x[i], g.c1x[i], g.d1x[i]);
    }
    __device__ __forceinline__ T Dy(const Geo<T>& g, const T* f) const {
        return d1fc(f[ym2], f[ym1], f[c], f[yp1], f[yp2], g.a1y[j], g.b1y[j], g.c1y[j], g.d1y[j]);
    }
    __device__ __forceinline__ T Dz(const Geo<T>& g, const T* f) const {
        return d1fc(f[c - 2 * g.sz], f[c - g.sz], f[c], f[c + g.sz], f[c + 2 * g.sz],
                    g.a1z[k], g.b1z[k], g.c1z[k], g.d1z[k]);
    }
};

// ---------------------------------------------------------------------------------------
// NFLD field pointers (the transposed smoothing passes of the adjoint)
template <class T, int NFLD>
struct FS { T* f[NFLD]; };

// ---------------------------------------------------------------------------------------
// E = -v x B + eta*J at every node (t3dsdsc.f:1367-1372).
template <class T>
__global__ void k_efield(Geo<T> g, F8<T> x, F3<T> cur, F3<T> e) {
    wait_for_stream();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.mx) return;
    int jj = blockIdx.y, k = blockIdx.z;
    long c = (long)i + (long)jj * g.sy + (long)k * g.sz;
    T r = T(g.rho0[k]) + x.f[0][c];
    T m1 = x.f[1][c], m2 = x.f[2][c], m3 = x.f[3][c];
    T b1 = T(g.bx0[k]) + x.f[4][c], b2 = T(g.by0[k]) + x.f[5][c], b3 = T(g.bz0[k]) + x.f[6][c];
    const T ri = T(1) / r;
    e.f[0][c] = (-m2 * b3 + m3 * b2) * ri + g.eta * cur.f[0][c];
    e.f[1][c] = (-m3 * b1 + m1 * b3) * ri + g.eta * cur.f[1][c];
    e.f[2][c] = (-m1 * b2 + m2 * b1) * ri + g.eta * cur.f[2][c];
}

// ---------------------------------------------------------------------------------------
// J0 added to the smoothed J1 (j0_mode FULL).
template <class T>
__global__ void k_add_j0(Geo<T> g, F3<T> cur) {
    wait_for_stream();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.mx) return;
    int jj = blockIdx.y, k = blockIdx.z;
    long c = (long)i + (long)jj * g.sy + (long)k * g.sz;
    cur.f[0][c] += T(g.j0x[k]);
    cur.f[1][c] += T(g.j0y[k]);
    cur.f[2][c] += T(g.j0z[k]);
}

// ---------------------------------------------------------------------------------------
// FP64 reductions
__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// CFL in rate form: the reference's per-direction step h / (vp/cfl + visc/(2h)) is the
// inverse of the rate vp * (1/(cfl h)) + visc/(2 h^2), so dt = min(100, 1 / max rate) over
// the region k 0..mz-3, j 0..my-2, i 0..mx-3 (t3dsdsc.f:4709-4736).  Tables per axis:
// ich = 1/(cfl |h|), vv = visc/(2 h^2), ih = 1/|h| (whistler term).  NaN wins so that a corrupted
// state is reported.
__device__ __forceinline__ double nanmax(double a, double b) { return (a != a || b != b) ? (a != a ? a : b) : fmax(a, b); }

// The CFL rate of node c (totals = equilibrium profile at the node's plane + stored
// perturbation), max over the three directions.
template <class T>
__device__ __forceinline__ double cfl_node_rate(const F8<T>& x, long c, double r0, double bx0, double by0, double bz0,
                                                double p0, double gamma, double whistler, double cx, double vx_,
                                                double hx, double cy, double vy_, double hy, double cz, double vz_,
                                                double hz) {
    double rinv = 1.0 / (r0 + (double)x.f[0][c]);
    double vx = (double)x.f[1][c] * rinv, vy = (double)x.f[2][c] * rinv, vz = (double)x.f[3][c] * rinv;
    double b1 = bx0 + (double)x.f[4][c], b2 = by0 + (double)x.f[5][c], b3 = bz0 + (double)x.f[6][c];
    double bb = b1 * b1 + b2 * b2 + b3 * b3;
    double vf = sqrt(fabs((bb + gamma * (p0 + (double)x.f[7][c])) * rinv));
    double w = whistler != 0.0 ? whistler * sqrt(bb) * rinv : 0.0;
    double rx = (fabs(vx) + vf + w * hx) * cx + vx_;
    double ry = (fabs(vy) + vf + w * hy) * cy + vy_;
    double rz = (fabs(vz) + vf + w * hz) * cz + vz_;
    return nanmax(rx, nanmax(ry, rz));
}

// the 16 bytes of a field at p (aligned: rows are multiples of 4 values)
__device__ __forceinline__ void load16(const float* p, float (&v)[4]) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void load16(const double* p, double (&v)[2]) {
    const double2 q = *reinterpret_cast<const double2*>(p);
    v[0] = q.x; v[1] = q.y;
}

// setdt's sweep.  The rate needs FP64 (a division and two square roots a node: the FP64 pipe took 386 us for the
// 33.5M nodes of 512x256x256 FP32, where memory needs 167), but only at nodes that can be the maximum: each
// node first gets an upper bound in FP32, and cfl_node_rate runs where the bound reaches the largest rate known so far
// (this warp's, and other CTAs' at the start), so the result is the full sweep's to the last bit.  The bound: rho, B and p
// totals are formed in the field's precision; FP32 totals are off by 2^-24 (|background| + |total|), which is added to |B| and
// |p| as 1e-6 |background| and kept below 8e-6 relative in rho by taking nodes with |rho| < |rho0| / 128
// or outside 1e-10 .. 1e10 as unbounded; |B^2 + gamma p| <= B^2 + gamma |p|; the 1e-36 and 1e-25 cover
// underflow; everything else is a sum of non-negative products whose roundings stay far below
// the factor 1 + 3e-5.  NaN compares false and is evaluated, and NaN wins the maximum.
// A thread owns 16 bytes of a row (4 FP32 or 2 FP64 nodes) and marches over `planes` planes, so
// the x and y tables are read once; one atomicMax a CTA on the bits of the rate (rates are >= 0, a NaN pattern
// lies above every finite one).  512x256x256 FP32 386 + 42 (a one-block reduction of the rows) -> 229 us,
// 256x128x256 FP64 116 + 23 -> 108.  It also replaces a tap on the post-step filter's last launch, which
// read the 8 fields back there and made that launch 500 us (512x256x256 FP32), 230 us (256x128x256 FP64) longer;
// on 64x32x64 both ways take a step the same time.  Capped at 3 CTAs an SM (80 registers) 250 us, at 4 375.
template <class T>
__global__ void __launch_bounds__(256) k_cfl_rate(Geo<T> g, F8<T> x, const double* ich, const double* vv, const double* ih,
                                                  double gamma, double whistler, int planes, unsigned long long* out,
                                                  unsigned long long* next) {
    constexpr int V = 16 / (int)sizeof(T);
    constexpr unsigned ALL = 0xffffffffu;
    wait_for_stream();
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *next = 0;   // the word the next sweep takes
    const int nq = g.mx / V, id = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = id < nq * (g.my - 1);
    const int jj = on ? id / nq : 0, i0 = on ? V * (id - jj * nq) : 0;
    const double *ichy = ich + g.mx, *ichz = ichy + g.my, *vvy = vv + g.mx, *vvz = vvy + g.my, *ihy = ih + g.mx, *ihz = ihy + g.my;
    float cx[V], ux[V], hx[V];
#pragma unroll
    for (int e = 0; e < V; ++e) { cx[e] = (float)ich[i0 + e]; ux[e] = fabsf((float)vv[i0 + e]); hx[e] = (float)ih[i0 + e]; }
    const float cy = (float)ichy[jj], uy = fabsf((float)vvy[jj]), hy = (float)ihy[jj];
    const float ga = fabsf((float)gamma), wh = fabsf((float)whistler);
    const int ka = g.kcfl0 + blockIdx.y * planes, kb = min(ka + planes, g.mz - 2);
    auto down = [](double b) { return b != b ? __int_as_float(0x7f800000) : __double2float_rd(b); };
    double best = 0.0;
    float thr = down(__longlong_as_double((long long)*(volatile unsigned long long*)out));
    for (int k = ka; k < kb; ++k) {
        const double r0 = g.rho0[k], bx0 = g.bx0[k], by0 = g.by0[k], bz0 = g.bz0[k], p0 = g.p0[k];
        const double czd = ichz[k], vzd = vvz[k], hzd = ihz[k];
        const float cz = (float)czd, uz = fabsf((float)vzd), hz = (float)hzd;
        const long c = (long)i0 + (long)jj * g.sy + (long)k * g.sz;
        float est[V], top = -1.f;
        {
            T f[8][V];
#pragma unroll
            for (int m = 0; m < 8; ++m) load16(x.f[m] + c, f[m]);
#pragma unroll
            for (int e = 0; e < V; ++e) {
                float r, b1, b2, b3, p;
                bool ok = true;
                if constexpr (sizeof(T) == 4) {
                    const float R0 = (float)r0, X0 = (float)bx0, Y0 = (float)by0, Z0 = (float)bz0, P0 = (float)p0;
                    r = fabsf(R0 + f[0][e]);
                    ok = r >= 0.0078125f * fabsf(R0);
                    b1 = fmaf(1e-6f, fabsf(X0), fabsf(X0 + f[4][e]));
                    b2 = fmaf(1e-6f, fabsf(Y0), fabsf(Y0 + f[5][e]));
                    b3 = fmaf(1e-6f, fabsf(Z0), fabsf(Z0 + f[6][e]));
                    p = fmaf(1e-6f, fabsf(P0), fabsf(P0 + f[7][e]));
                } else {
                    r = fabsf((float)(r0 + f[0][e]));
                    b1 = (float)(bx0 + f[4][e]); b2 = (float)(by0 + f[5][e]); b3 = (float)(bz0 + f[6][e]);
                    p = fabsf((float)(p0 + f[7][e]));
                }
                const float ri = __fdividef(1.f, r);
                const float bb = fmaf(b1, b1, fmaf(b2, b2, fmaf(b3, b3, 1e-36f)));
                const float q = fmaf(ga, p, bb) * ri;
                const float vf = q * rsqrtf(q);
                const float w = wh != 0.f ? wh * (bb * rsqrtf(bb)) * ri : 0.f;
                const float ex = fmaf(fmaf(fabsf((float)f[1][e]), ri, fmaf(w, hx[e], vf)), cx[e], ux[e]);
                const float ey = fmaf(fmaf(fabsf((float)f[2][e]), ri, fmaf(w, hy, vf)), cy, uy);
                const float ez = fmaf(fmaf(fabsf((float)f[3][e]), ri, fmaf(w, hz, vf)), cz, uz);
                const float s = ex + ey + ez;   // NaN and infinity of any of the three
                float b = fmaxf(ex, fmaxf(ey, ez)) * 1.00003f + 1e-25f;
                if (!(ok && r >= 1e-10f && r <= 1e10f && s < 3e38f)) b = __int_as_float(0x7f800000);
                est[e] = on && i0 + e <= g.mx - 3 ? b : -1.f;
                top = fmaxf(top, est[e]);
            }
        }
        if (!__any_sync(ALL, top >= thr)) continue;
        auto exact = [&](int e) {
            const int i = i0 + e;
            best = nanmax(best, cfl_node_rate(x, c + e, r0, bx0, by0, bz0, p0, gamma, whistler, ich[i], vv[i], ih[i],
                                              ichy[jj], vvy[jj], ihy[jj], czd, vzd, hzd));
        };
        // the warp's highest bound first: its rate mostly rules the others out
        const unsigned high = __reduce_max_sync(ALL, __float_as_uint(fmaxf(top, 0.f)));
        if (top >= thr && __float_as_uint(top) == high) {
            int m = 0;
#pragma unroll
            for (int e = V - 1; e >= 0; --e) if (est[e] == top) m = e;
            exact(m);
        }
        thr = fmaxf(thr, __uint_as_float(__reduce_max_sync(ALL, __float_as_uint(down(best)))));
#pragma unroll
        for (int e = 0; e < V; ++e)
            if (est[e] >= thr) exact(e);
        thr = fmaxf(thr, __uint_as_float(__reduce_max_sync(ALL, __float_as_uint(down(best)))));
    }
    __shared__ double sh[8];
    double v = best;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = nanmax(v, __shfl_down_sync(ALL, v, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < 8; ++q) v = nanmax(v, sh[q]);
        if (v != 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(v));
    }
}

// sum over the CTA (at most 32 warps), in thread 0; sh is free again after the next barrier
__device__ __forceinline__ double cta_sum(double v, double* sh) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = threadIdx.x < nw ? sh[lane] : 0.;
    return wid == 0 ? warp_sum(v) : v;
}

// Diagnostics partial results, one launch for the three kinds of CTA (128 threads):
//  - DIAG_J rows of a plane: mass and energy with the trapezoid weights, part[2 b], part[2 b + 1].  Planes klo..khi
//    count (a z-slab's own planes and the walls it holds); the others give zero;
//  - reconnected flux of a row j: sum_x sqrt(Bz(z=0)^2+eps^2)*wx, with Bz on the central plane ka (odd mz, kb = ka)
//    or the mean of the two central planes ka, kb = ka + 1 (even mz); ka < 0: a z-slab that does not own
//    the (first) central plane;
//  - J extrema of a plane k's row my/2 (diagn t3dsdsc.f:1199-1214).
// 16-byte loads, DIAG_J rows a CTA: an eighth of the partial results for the reduction that follows, and one launch
// for three.  dasha_diagnostics of 256x128x256 FP32, its current included: 0.48 -> 0.38 ms.
constexpr int DIAG_J = 8;
template <class T>
__global__ void __launch_bounds__(128) k_diag_parts(Geo<T> g, F8<T> x, F3<T> cur, const double* wx, const double* wy,
                                                    const double* wz, double gamma, double* part, double* fl, double* jext,
                                                    int klo, int khi, int ka, int kb) {
    wait_for_stream();
    constexpr int V = 16 / (int)sizeof(T);
    __shared__ double s1[32], s2[32];
    const int tid = threadIdx.x, nj = (g.my + DIAG_J - 1) / DIAG_J;
    const long rows = (long)nj * g.mz;
    const long b = blockIdx.x;
    if (b < rows) {
        const int k = (int)(b / nj), j0 = (int)(b - (long)k * nj) * DIAG_J, nr = min(DIAG_J, g.my - j0), nq = g.mx / V;
        double sm = 0., se = 0.;
        if (k >= klo && k <= khi) {
            const double r0 = g.rho0[k], bx0 = g.bx0[k], by0 = g.by0[k], bz0 = g.bz0[k], p0 = g.p0[k];
            for (int n = tid; n < nr * nq; n += blockDim.x) {
                const int j = j0 + n / nq, i0 = V * (n % nq);
                const long c = (long)i0 + (long)j * g.sy + (long)k * g.sz;
                T f[8][V];
#pragma unroll
                for (int m = 0; m < 8; ++m) load16(x.f[m] + c, f[m]);
                const double w = wy[j];
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const double rho = r0 + (double)f[0][e], m1 = f[1][e], m2 = f[2][e], m3 = f[3][e];
                    const double b1 = bx0 + (double)f[4][e], b2 = by0 + (double)f[5][e], b3 = bz0 + (double)f[6][e];
                    const double p = p0 + (double)f[7][e], vol = wx[i0 + e] * w;
                    sm += rho * vol;
                    se += (0.5 * (m1 * m1 + m2 * m2 + m3 * m3) / rho + p / (gamma - 1.) + 0.5 * (b1 * b1 + b2 * b2 + b3 * b3)) * vol;
                }
            }
        }
        sm = cta_sum(sm, s1);
        se = cta_sum(se, s2);
        if (tid == 0) { part[2 * b] = sm * wz[k]; part[2 * b + 1] = se * wz[k]; }
    } else if (b < rows + g.my) {
        const int j = (int)(b - rows);
        double s = 0.;
        for (int i = tid; i < g.mx && ka >= 0; i += blockDim.x) {
            const long c = (long)i + (long)j * g.sy;
            double bz = g.bz0[ka] + (double)x.f[6][c + (long)ka * g.sz];
            if (ka != kb) bz = 0.5 * (bz + (g.bz0[kb] + (double)x.f[6][c + (long)kb * g.sz]));
            s += sqrt(bz * bz + 1e-20) * wx[i];
        }
        s = cta_sum(s, s1);
        if (tid == 0) fl[j] = s;
    } else {
        const int k = (int)(b - rows - g.my), lane = tid & 31, wid = tid >> 5;
        double mx[3] = {-1e300, -1e300, -1e300}, mn[3] = {1e300, 1e300, 1e300};
        for (int i = tid; i < g.mx && k >= klo && k <= khi; i += blockDim.x) {
            const long c = (long)i + (long)(g.my / 2) * g.sy + (long)k * g.sz;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const double v = cur.f[m][c];
                mx[m] = fmax(mx[m], v);
                mn[m] = fmin(mn[m], v);
            }
        }
        __shared__ double sh[6][4];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const double a = warp_max(mx[m]), d = warp_min(mn[m]);
            if (lane == 0) { sh[2 * m][wid] = a; sh[2 * m + 1][wid] = d; }
        }
        __syncthreads();
        if (tid < 6) {
            double v = sh[tid][0];
            for (int q = 1; q < 4; ++q) v = tid & 1 ? fmin(v, sh[tid][q]) : fmax(v, sh[tid][q]);
            jext[6 * k + tid] = v;
        }
    }
}

// Final diagnostics reduction (one block, fixed order) -> out[9]; also raises the blow-up
// flag when max Jy >= 1e7 (t3dsdsc.f:1232).  Every thread takes part in each sum and extremum: with the flux and the
// extrema left to one thread and a row's result per (j, k) it took 105 us on 256x128x256, 138 us on 512x256x256.
static __global__ void __launch_bounds__(1024) k_diag_final(const double* rows, long nrows, const double* fl, int my,
                                                            const double* jext, int mz, double* out, int* blowup) {
    wait_for_stream();
    __shared__ double sh[3][32], ex[6][32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double sm = 0., se = 0., f = 0.;
#pragma unroll 4
    for (long q = tid; q < nrows; q += blockDim.x) {
        const double2 v = *reinterpret_cast<const double2*>(rows + 2 * q);
        sm += v.x;
        se += v.y;
    }
    for (int j = tid; j < my; j += blockDim.x) f += fl[j];
    double e[6] = {-1e300, 1e300, -1e300, 1e300, -1e300, 1e300};
    for (int k = tid; k < mz; k += blockDim.x)
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            e[2 * m] = fmax(e[2 * m], jext[6 * k + 2 * m]);
            e[2 * m + 1] = fmin(e[2 * m + 1], jext[6 * k + 2 * m + 1]);
        }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const double v = q & 1 ? warp_min(e[q]) : warp_max(e[q]);
        if (lane == 0) ex[q][wid] = v;
    }
    sm = cta_sum(sm, sh[0]);
    se = cta_sum(se, sh[1]);
    f = cta_sum(f, sh[2]);
    if (wid == 0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) e[q] = q & 1 ? warp_min(ex[q][lane]) : warp_max(ex[q][lane]);
        if (tid == 0) {
            out[0] = sm; out[1] = se; out[2] = f / my;
            for (int q = 0; q < 6; ++q) out[3 + q] = e[q];
            if (blowup && (fabs(e[2]) >= 1e7 || e[2] != e[2])) *blowup = 1;
        }
    }
}

}  // namespace dasha
