// adjoint.cuh -- discrete adjoint (vector-Jacobian products) of the RK4 Hall-MHD step, FP64.
//
// The forward step (stepon, t3dsdsc.f:1063-1185) is X -> F(X + dt/6 (k1 + 2 k2 + 2 k3 + k4))
// with k = G(S) = avrg(right(S)) and F the post-step filter (avrgtt).  With dt held fixed
// (the recorded sequence is replayed) every piece is either linear -- the smoothing passes
// with their wall rows, the curls, the 4th-order derivatives -- or pointwise: E = -v x B +
// eta J, the Hall term, the fluxes and the pressure equation.  Each linear piece is
// transposed here as a gather (one thread per node reads the adjoint at the nodes whose
// stencils touch it); the wall rows y(1) = y(2)/2, y(0) = 0 transpose to a fold of the row
// adjoints into row 2 (and mz-3).  No reference counterpart: the reference has no adjoint.
#pragma once
#include "mhd_kernels.cuh"
#include "zm_kernels.cuh"

namespace dasha {

// One thread per x-y column and run of ZB planes (the engine's choice is 1); x and y flattened so that a
// warp is full whatever mx is.  Bound by the latency of a thread's loads, so a run away from the walls
// loads without conditions, and the launch bounds trade registers for warps.  Measured on B200, 128x64x128 /
// 44x24x50, us a launch, against one node a thread with the wall conditions at every load: 3-field pass 34 -> 25 /
// 10.7 -> 10.1, 8 fields 108 (two launches) -> 63 / 26 -> 12.7, pointwise 208 -> 86 + 19 (velocities) / 23 -> 11 + 8,
// gather 201 -> 113 / 25 -> 13; the copies and fills around them (20 of 8 fields a step) are gone.
struct AdjCol {
    int i, j, im, ip, jm, jp;
    unsigned c0, xm, xp, ym, yp;                      // offsets of the node and its neighbours in a plane
    bool on;
    __device__ __forceinline__ AdjCol(const Geo<double>& g) {
        const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
        on = q < (unsigned)(g.mx * g.my);
        j = (int)(q / (unsigned)g.mx);
        i = (int)(q - (unsigned)j * (unsigned)g.mx);
        im = wrapi(i - 1, g.mx); ip = wrapi(i + 1, g.mx); jm = wrapi(j - 1, g.my); jp = wrapi(j + 1, g.my);
        c0 = q;
        xm = c0 - i + im; xp = c0 - i + ip;
        ym = (unsigned)(jm * g.mx + i); yp = (unsigned)(jp * g.mx + i);
    }
};

// Transpose of one smoothing pass on planes 2 .. mz-3 (fields in, out; KINDS as in k_zpv).  The input
// ybar is the adjoint of the pass output with its wall rows; folding them (y(1) = y(2)/2 -> ybar(2) +=
// ybar(1)/2, same at the top; rows 0 and mz-1 constant) is done on the fly.  With c the coefficient
// and u = c ybar on the interior planes,
//   x(n) = ybar(n) - W u(n) + sum over neighbours m of w(m -> n) u(m),   W the sum of n's six weights,
// and the wall rows 1 and mz-2 take w u of rows 2 and mz-3.  FOLD: the result's wall rows folded in
// the same way (rows 0, 1, mz-2, mz-1 zero), for the last pass of a chain whose input had its rows from a
// boundary rule.
// EDGE: the run holds row 2 or mz-3, or ends beyond it; all others load without a condition, so that a
// thread's loads are in flight together.
template <int NF, unsigned KINDS, int ZB, bool EDGE>
__device__ __forceinline__ void adj_pass_run(const Geo<double>& g, const AdjCol& t, int kb, const FS<double, NF>& in,
                                             const FS<double, NF>& out, bool fold) {
    const int kt = g.mz - 3;
    const double wxy = g.wpx[t.i] + g.wmx[t.i] + g.wpy[t.j] + g.wmy[t.j];
    const double wxm = g.wpx[t.im], wxp = g.wmx[t.ip], wym = g.wpy[t.jm], wyp = g.wmy[t.jp];
    constexpr bool RAD = any_kind0(KINDS, NF);
    // the radial coefficient: of the column, planes kb-1 .. kb+ZB, and of the x and y neighbours
    double cr[ZB + 2], cn[ZB][4];
    if constexpr (RAD) {
#pragma unroll
        for (int z = 0; z < ZB + 2; ++z) cr[z] = g.cr[t.c0 + (long)(EDGE ? min(kb - 1 + z, kt) : kb - 1 + z) * g.sz];
#pragma unroll
        for (int z = 0; z < ZB; ++z) {
            const double* p = g.cr + (long)(EDGE ? min(kb + z, kt) : kb + z) * g.sz;
            cn[z][0] = p[t.xm] * wxm; cn[z][1] = p[t.xp] * wxp; cn[z][2] = p[t.ym] * wym; cn[z][3] = p[t.yp] * wyp;
        }
    }
#pragma unroll
    for (int q = 0; q < NF; ++q) {
        constexpr unsigned K = KINDS;
        const unsigned kind = (K >> (2 * q)) & 3u;
        const double* y = in.f[q];
        // folded ybar at offset o of plane k, 0 off the interior planes
        auto Y = [&](unsigned o, int k) {
            if (!EDGE) return y[o + (long)k * g.sz];
            double v = 0.0;
            if (k >= 2 && k <= kt) {
                v = y[o + (long)k * g.sz];
                if (k == 2) v += 0.5 * y[o + g.sz];
                if (k == kt) v += 0.5 * y[o + (long)(k + 1) * g.sz];
            }
            return v;
        };
        double yc[ZB + 2], yn[ZB][4];
#pragma unroll
        for (int z = 0; z < ZB + 2; ++z) yc[z] = Y(t.c0, kb - 1 + z);
#pragma unroll
        for (int z = 0; z < ZB; ++z) {
            yn[z][0] = Y(t.xm, kb + z); yn[z][1] = Y(t.xp, kb + z); yn[z][2] = Y(t.ym, kb + z); yn[z][3] = Y(t.yp, kb + z);
        }
        const double cc = kind == 1u ? 0.125 : g.cbx[t.i];
        const double cxm = (kind == 1u ? 0.125 : g.cbx[t.im]) * wxm, cxp = (kind == 1u ? 0.125 : g.cbx[t.ip]) * wxp;
        auto cz = [&](int z) { return kind == 0u ? cr[RAD ? z : 0] : cc; };
#pragma unroll
        for (int z = 1; z <= ZB; ++z) {
            const int k = kb - 1 + z;
            if (EDGE && k > kt) continue;
            const double* n = yn[z - 1];
            double v = yc[z] * (1.0 - cz(z) * (wxy + g.wpz[k] + g.wmz[k]));
            if (kind == 0u) {
                const double* c = cn[RAD ? z - 1 : 0];
                v += n[0] * c[0] + n[1] * c[1] + n[2] * c[2] + n[3] * c[3];
            } else {
                v += n[0] * cxm + n[1] * cxp + (n[2] * wym + n[3] * wyp) * cc;
            }
            if (!EDGE || k > 2) v += yc[z - 1] * cz(z - 1) * g.wpz[k - 1];
            if (!EDGE || k < kt) v += yc[z + 1] * cz(z + 1) * g.wmz[k + 1];
            const long ko = t.c0 + (long)k * g.sz;
            if (EDGE && (k == 2 || k == kt)) {        // the wall rows 1 and mz-2 (both where mz = 5)
                double lo = k == 2 ? yc[z] * cz(z) * g.wmz[2] : 0.0, hi = k == kt ? yc[z] * cz(z) * g.wpz[kt] : 0.0;
                if (fold) { v += 0.5 * (lo + hi); lo = 0.0; hi = 0.0; }
                if (k == 2) { out.f[q][t.c0 + g.sz] = lo; out.f[q][t.c0] = 0.0; }
                if (k == kt) { out.f[q][ko + g.sz] = hi; out.f[q][ko + 2 * g.sz] = 0.0; }
            }
            out.f[q][ko] = v;
        }
    }
}
template <int NF, unsigned KINDS, int ZB>
__device__ __forceinline__ void adj_pass_body(const Geo<double>& g, const FS<double, NF>& in, const FS<double, NF>& out,
                                              bool fold) {
    const AdjCol t(g);
    const int kb = 2 + (int)blockIdx.y * ZB, kt = g.mz - 3;
    if (!t.on || kb > kt) return;
    if (kb > 3 && kb + ZB < kt) adj_pass_run<NF, KINDS, ZB, false>(g, t, kb, in, out, fold);
    else adj_pass_run<NF, KINDS, ZB, true>(g, t, kb, in, out, fold);
}
template <unsigned KINDS, int ZB>
static __global__ void __launch_bounds__(128, 8) k_adj_pass3(const __grid_constant__ Geo<double> g, const __grid_constant__ FS<double, 3> in,
                                                         const __grid_constant__ FS<double, 3> out, bool fold) {
    wait_for_stream();
    adj_pass_body<3, KINDS, ZB>(g, in, out, fold);
}
// the 8 state-like fields: (rho, m) and (B, p) by blockIdx.z
template <unsigned KINDS_B, int ZB>
static __global__ void __launch_bounds__(128, 8) k_adj_pass8(const __grid_constant__ Geo<double> g, const __grid_constant__ F8<double> in,
                                                         const __grid_constant__ F8<double> out, bool fold) {
    wait_for_stream();
    FS<double, 4> a, b;
    const int lo = 4 * (int)blockIdx.z;
#pragma unroll
    for (int q = 0; q < 4; ++q) { a.f[q] = lo ? in.f[4 + q] : in.f[q]; b.f[q] = lo ? out.f[4 + q] : out.f[q]; }
    if (lo) adj_pass_body<4, KINDS_B, ZB>(g, a, b, fold);
    else adj_pass_body<4, 0u, ZB>(g, a, b, fold);
}

// Transposed first derivatives at a column: (D^T w)(n) for the stencil with per-node coefficients
//   D f(c) = a_c f(c+1) + (-a+b-c+d)_c f(c) - b_c f(c-1) + c_c f(c+2) - d_c f(c-2)
struct DTCol : AdjCol {
    unsigned xm2, xp2, ym2, yp2;
    double ax[5], ay[5];                              // weights of n, n-1, n+1, n-2, n+2
    __device__ __forceinline__ DTCol(const Geo<double>& g) : AdjCol(g) {
        if (!on) return;
        const int i2 = wrapi(i - 2, g.mx), p2 = wrapi(i + 2, g.mx), j2 = wrapi(j - 2, g.my), q2 = wrapi(j + 2, g.my);
        xm2 = c0 - i + i2; xp2 = c0 - i + p2;
        ym2 = (unsigned)(j2 * g.mx + i); yp2 = (unsigned)(q2 * g.mx + i);
        ax[0] = -g.a1x[i] + g.b1x[i] - g.c1x[i] + g.d1x[i];
        ax[1] = g.a1x[im]; ax[2] = g.b1x[ip]; ax[3] = g.c1x[i2]; ax[4] = g.d1x[p2];
        ay[0] = -g.a1y[j] + g.b1y[j] - g.c1y[j] + g.d1y[j];
        ay[1] = g.a1y[jm]; ay[2] = g.b1y[jp]; ay[3] = g.c1y[j2]; ay[4] = g.d1y[q2];
    }
    __device__ __forceinline__ double x(const double* w, long ko, double w0) const {
        return w0 * ax[0] + w[xm + ko] * ax[1] - w[xp + ko] * ax[2] + w[xm2 + ko] * ax[3] - w[xp2 + ko] * ax[4];
    }
    __device__ __forceinline__ double y(const double* w, long ko, double w0) const {
        return w0 * ay[0] + w[ym + ko] * ay[1] - w[yp + ko] * ay[2] + w[ym2 + ko] * ay[3] - w[yp2 + ko] * ay[4];
    }
};
// the z weights of plane k (w is zero outside the interior planes, the z coefficients are too)
struct DTz {
    double a[5];
    __device__ __forceinline__ DTz(const Geo<double>& g, int k, bool inner) {
        if (inner) {                                  // k-2 .. k+2 on the grid
            a[0] = -g.a1z[k] + g.b1z[k] - g.c1z[k] + g.d1z[k];
            a[1] = g.a1z[k - 1]; a[2] = g.b1z[k + 1]; a[3] = g.c1z[k - 2]; a[4] = g.d1z[k + 2];
            return;
        }
        auto A = [&](const double* t, int kk) { return (kk >= 0 && kk < g.mz) ? t[kk] : 0.0; };
        a[0] = -A(g.a1z, k) + A(g.b1z, k) - A(g.c1z, k) + A(g.d1z, k);
        a[1] = A(g.a1z, k - 1); a[2] = A(g.b1z, k + 1); a[3] = A(g.c1z, k - 2); a[4] = A(g.d1z, k + 2);
    }
    // col: planes k-2 .. k+2
    __device__ __forceinline__ double of(const double* col) const {
        return col[2] * a[0] + col[1] * a[1] - col[3] * a[2] + col[0] * a[3] - col[4] * a[4];
    }
};
// ZB + 4 values of a column from plane k0-2 on, 0 beyond the grid
template <int ZB>
__device__ __forceinline__ void dt_column(const Geo<double>& g, const double* w, unsigned c0, int k0, bool inner,
                                          double (&col)[ZB + 4]) {
    if (inner) {
#pragma unroll
        for (int z = 0; z < ZB + 4; ++z) col[z] = w[c0 + (long)(k0 - 2 + z) * g.sz];
        return;
    }
#pragma unroll
    for (int z = 0; z < ZB + 4; ++z) {
        const int k = k0 - 2 + z;
        col[z] = (k >= 0 && k < g.mz) ? w[c0 + (long)k * g.sz] : 0.0;
    }
}

// out (+)= s * curl^T(w):  curl(B) = (Dy B3 - Dz B2, Dz B1 - Dx B3, Dx B2 - Dy B1), so
//   curl^T(w) = (Dz^T w2 - Dy^T w3, Dx^T w3 - Dz^T w1, Dy^T w1 - Dx^T w2)
// Every plane of the grid (row 0 and 1 take from rows 2 and 3).
template <int ZB>
static __global__ void __launch_bounds__(128) k_adj_curlT(const __grid_constant__ Geo<double> g, const __grid_constant__ F3<double> w,
                                                         const __grid_constant__ F3<double> out, double s, int accumulate) {
    wait_for_stream();
    const DTCol t(g);
    if (!t.on) return;
    const int k0 = (int)blockIdx.y * ZB;
    const bool inner = k0 >= 2 && k0 + ZB + 2 <= g.mz;
    double c1[ZB + 4], c2[ZB + 4];
    dt_column<ZB>(g, w.f[0], t.c0, k0, inner, c1);
    dt_column<ZB>(g, w.f[1], t.c0, k0, inner, c2);
#pragma unroll
    for (int z = 0; z < ZB; ++z) {
        const int k = k0 + z;
        if (k >= g.mz) break;
        const long ko = (long)k * g.sz;
        const DTz dz(g, k, inner);
        const double w3 = w.f[2][t.c0 + ko];
        const double o0 = dz.of(c2 + z) - t.y(w.f[2], ko, w3);
        const double o1 = t.x(w.f[2], ko, w3) - dz.of(c1 + z);
        const double o2 = t.y(w.f[0], ko, c1[z + 2]) - t.x(w.f[1], ko, c2[z + 2]);
        const long c = t.c0 + ko;
        if (accumulate) { out.f[0][c] += s * o0; out.f[1][c] += s * o1; out.f[2][c] += s * o2; }
        else { out.f[0][c] = s * o0; out.f[1][c] = s * o1; out.f[2][c] = s * o2; }
    }
}

// v_d = m_d / rho at every node, for the divergence in k_adj_pointwise (13 divisions a node there otherwise)
static __global__ void __launch_bounds__(256) k_adj_velocity(long n, int mz, const __grid_constant__ Geo<double> g,
                                                            const __grid_constant__ F8<double> s, const __grid_constant__ F3<double> v) {
    wait_for_stream();
    const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double ri = 1.0 / (g.rho0[c / g.sz] + s.f[0][c]);
    v.f[0][c] = s.f[1][c] * ri;
    v.f[1][c] = s.f[2][c] * ri;
    v.f[2][c] = s.f[3][c] * ri;
}

// Pointwise adjoints at every node, given
//   eb  = adjoint of E0 (all nodes), hb = adjoint of the Hall field H0 (rows folded),
//   ob  = adjoint of the hydro outputs xdif 0,1,2,3,7 (rows folded)
// and the state S (perturbation form), its velocity and smoothed current J.  Produces
//   sb   = direct adjoints of rho, m1..3, B1..3, p (8 fields)
//   jb   = adjoint of J (3)
//   wq   = weighted fields for the stencil transposes done by k_adj_gather:
//          0..2: -di*hb_d/rho (Hall grad p) - ob7*v_d (v . grad p)   3: ob7*gamma*p (gamma p div v)
//   ub   = pointwise adjoint of u_d = m_d/rho at the node from the pressure equation (3)
//   eta  partial sums (one per block)
struct AdjPtw {
    F8<double> s;
    F3<double> j, eb, hb, jb, ub, v;
    const double* ob[5];
    F8<double> sb;
    double* wq[4];
    double* etapart;
    int hall;
};

static __global__ void __launch_bounds__(128, 4) k_adj_pointwise(const __grid_constant__ Geo<double> g, const __grid_constant__ AdjPtw a) {
    wait_for_stream();
    const unsigned node = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned plane = (unsigned)g.sz, row = (unsigned)g.mx;
    double eta_acc = 0.0;
    if (node < plane * (unsigned)g.mz) {
        const int k = (int)(node / plane), j = (int)((node - k * plane) / row), i = (int)(node - k * plane - j * row);
        const long c = node;
        const double rho = g.rho0[k] + a.s.f[0][c];
        const double ri = 1.0 / rho;
        const double m1 = a.s.f[1][c], m2 = a.s.f[2][c], m3 = a.s.f[3][c];
        const double b1 = g.bx0[k] + a.s.f[4][c], b2 = g.by0[k] + a.s.f[5][c], b3 = g.bz0[k] + a.s.f[6][c];
        const double j1 = a.j.f[0][c], j2 = a.j.f[1][c], j3 = a.j.f[2][c];
        double rb = 0, m1b = 0, m2b = 0, m3b = 0, b1b = 0, b2b = 0, b3b = 0, pb = 0, j1b = 0, j2b = 0, j3b = 0;
        // E0 = (-m x B)/rho + eta J
        const double e1 = a.eb.f[0][c], e2 = a.eb.f[1][c], e3 = a.eb.f[2][c];
        {
            const double n1 = -m2 * b3 + m3 * b2, n2 = -m3 * b1 + m1 * b3, n3 = -m1 * b2 + m2 * b1;
            m1b += (b3 * e2 - b2 * e3) * ri;
            m2b += (-b3 * e1 + b1 * e3) * ri;
            m3b += (b2 * e1 - b1 * e2) * ri;
            b1b += (-m3 * e2 + m2 * e3) * ri;
            b2b += (m3 * e1 - m1 * e3) * ri;
            b3b += (-m2 * e1 + m1 * e2) * ri;
            rb += -(n1 * e1 + n2 * e2 + n3 * e3) * ri * ri;
            j1b += g.eta * e1; j2b += g.eta * e2; j3b += g.eta * e3;
            eta_acc += j1 * e1 + j2 * e2 + j3 * e3;
        }
        const bool intr = k >= 2 && k <= g.mz - 3;
        double wq0 = 0, wq1 = 0, wq2 = 0, wq3 = 0, u1 = 0, u2 = 0, u3 = 0;
        if (intr) {
            Nbr<double> n(g, i, j, k);
            const double px = n.Dx(g, a.s.f[7]), py = n.Dy(g, a.s.f[7]), pz = n.Dz(g, a.s.f[7]) + g.dzp0[k];
            if (a.hall) {   // H0 = di (J x B - grad p)/rho
                const double h1 = a.hb.f[0][c], h2 = a.hb.f[1][c], h3 = a.hb.f[2][c];
                const double q1 = j2 * b3 - j3 * b2 - px, q2 = j3 * b1 - j1 * b3 - py, q3 = j1 * b2 - j2 * b1 - pz;
                const double d = g.di * ri;
                j1b += d * (-b3 * h2 + b2 * h3);
                j2b += d * (b3 * h1 - b1 * h3);
                j3b += d * (-b2 * h1 + b1 * h2);
                b1b += d * (j3 * h2 - j2 * h3);
                b2b += d * (-j3 * h1 + j1 * h3);
                b3b += d * (j2 * h1 - j1 * h2);
                rb += -d * ri * (q1 * h1 + q2 * h2 + q3 * h3);
                wq0 = -d * h1; wq1 = -d * h2; wq2 = -d * h3;
            }
            // hydro outputs: J x B in the momentum, the pressure equation
            const double o1 = a.ob[1][c], o2 = a.ob[2][c], o3 = a.ob[3][c], o7 = a.ob[4][c];
            j2b += o1 * b3; j3b -= o1 * b2; b3b += o1 * j2; b2b -= o1 * j3;
            j3b += o2 * b1; j1b -= o2 * b3; b1b += o2 * j3; b3b -= o2 * j1;
            j1b += o3 * b2; j2b -= o3 * b1; b2b += o3 * j1; b1b -= o3 * j2;
            // o7 = -(px v1 + py v2 + pz v3) + gamma p divv + (gamma-1) eta |J|^2
            const double v1 = m1 * ri, v2 = m2 * ri, v3 = m3 * ri;
            const double divv = -n.Dx(g, a.v.f[0]) - n.Dy(g, a.v.f[1]) - n.Dz(g, a.v.f[2]);
            const double p = g.p0[k] + a.s.f[7][c];
            u1 = -o7 * px; u2 = -o7 * py; u3 = -o7 * pz;   // adjoint of the centre velocity
            pb += o7 * g.gamma * divv;
            wq0 -= o7 * v1; wq1 -= o7 * v2; wq2 -= o7 * v3;
            wq3 = o7 * g.gamma * p;
            const double ce = (g.gamma - 1.0) * g.eta;
            j1b += o7 * 2.0 * ce * j1; j2b += o7 * 2.0 * ce * j2; j3b += o7 * 2.0 * ce * j3;
            eta_acc += o7 * (g.gamma - 1.0) * (j1 * j1 + j2 * j2 + j3 * j3);
        }
        a.sb.f[0][c] = rb; a.sb.f[1][c] = m1b; a.sb.f[2][c] = m2b; a.sb.f[3][c] = m3b;
        a.sb.f[4][c] = b1b; a.sb.f[5][c] = b2b; a.sb.f[6][c] = b3b; a.sb.f[7][c] = pb;
        a.jb.f[0][c] = j1b; a.jb.f[1][c] = j2b; a.jb.f[2][c] = j3b;
        a.wq[0][c] = wq0; a.wq[1][c] = wq1; a.wq[2][c] = wq2; a.wq[3][c] = wq3;
        a.ub.f[0][c] = u1; a.ub.f[1][c] = u2; a.ub.f[2][c] = u3;
    }
    // block partial of d/d eta
    __shared__ double sh[32];
    double v = warp_sum(eta_acc);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        int nw = (blockDim.x + 31) >> 5;
        double t = 0;
        for (int w2 = 0; w2 < nw; ++w2) t += sh[w2];
        a.etapart[blockIdx.x] = t;
    }
}

// Gather of the stencil transposes of the hydro and Hall adjoints, then the pointwise chain
// rule through the fluxes m_d m_k / rho (+ dp on the diagonal), u_d = m_d/rho and p.
//   ob: adjoints of xdif 0,1,2,3,7 (rows folded);  wq, ub from k_adj_pointwise
struct AdjGat {
    F8<double> s, sb;
    const double* wq[4];
    F3<double> ub;
    const double* ob[5];
};

template <int ZB>
static __global__ void __launch_bounds__(128, 4) k_adj_gather(const __grid_constant__ Geo<double> g, const __grid_constant__ AdjGat a) {
    wait_for_stream();
    const DTCol t(g);
    if (!t.on) return;
    const int k0 = (int)blockIdx.y * ZB;
    const bool inner = k0 >= 2 && k0 + ZB + 2 <= g.mz;
    double m[ZB][3], ri[ZB], mb[ZB][3], rb[ZB], pb[ZB], ub[ZB][3];
#pragma unroll
    for (int z = 0; z < ZB; ++z) {
        const int k = min(k0 + z, g.mz - 1);
        const long c = t.c0 + (long)k * g.sz;
        ri[z] = 1.0 / (g.rho0[k] + a.s.f[0][c]);
        rb[z] = 0.0;
        pb[z] = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) { m[z][d] = a.s.f[1 + d][c]; mb[z][d] = 0.0; ub[z][d] = a.ub.f[d][c]; }
    }
    double col[ZB + 4];
    // flux adjoints ab[d] = -(D_d^T ob_q)(n), q = 0 continuity, 1..3 momentum
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double* w = a.ob[q];
        dt_column<ZB>(g, w, t.c0, k0, inner, col);
#pragma unroll
        for (int z = 0; z < ZB; ++z) {
            const int k = min(k0 + z, g.mz - 1);
            const long ko = (long)k * g.sz;
            const DTz dz(g, k0 + z, inner);
            const double ab[3] = {-t.x(w, ko, col[z + 2]), -t.y(w, ko, col[z + 2]), -dz.of(col + z)};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (q == 0) { mb[z][d] += ab[d]; continue; }
                const double f = ab[d] * ri[z];       // flux m_d m_q / rho, dp on the diagonal
                mb[z][d] += f * m[z][q > 0 ? q - 1 : 0];
                mb[z][q > 0 ? q - 1 : 0] += f * m[z][d];
                rb[z] -= f * m[z][d] * m[z][q > 0 ? q - 1 : 0] * ri[z];
                if (d == q - 1) pb[z] += ab[d];
            }
        }
    }
    // pressure: D_d^T of the Hall weights less D_d^T(ob7 v_d) (v.grad p);  u_d gets -D_d^T(ob7 gamma p)
#pragma unroll
    for (int z = 0; z < ZB; ++z) {
        const long ko = (long)min(k0 + z, g.mz - 1) * g.sz;
        pb[z] += t.x(a.wq[0], ko, a.wq[0][t.c0 + ko]) + t.y(a.wq[1], ko, a.wq[1][t.c0 + ko]);
        const double w3 = a.wq[3][t.c0 + ko];
        ub[z][0] -= t.x(a.wq[3], ko, w3);
        ub[z][1] -= t.y(a.wq[3], ko, w3);
    }
    dt_column<ZB>(g, a.wq[2], t.c0, k0, inner, col);
#pragma unroll
    for (int z = 0; z < ZB; ++z) pb[z] += DTz(g, k0 + z, inner).of(col + z);
    dt_column<ZB>(g, a.wq[3], t.c0, k0, inner, col);
#pragma unroll
    for (int z = 0; z < ZB; ++z) ub[z][2] -= DTz(g, k0 + z, inner).of(col + z);
#pragma unroll
    for (int z = 0; z < ZB; ++z) {
        if (k0 + z >= g.mz) break;
        const long c = t.c0 + (long)(k0 + z) * g.sz;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            mb[z][d] += ub[z][d] * ri[z];
            rb[z] -= ub[z][d] * m[z][d] * ri[z] * ri[z];
        }
        a.sb.f[0][c] += rb[z];
        a.sb.f[1][c] += mb[z][0];
        a.sb.f[2][c] += mb[z][1];
        a.sb.f[3][c] += mb[z][2];
        a.sb.f[7][c] += pb[z];
    }
}

// *acc += sum(part[0..n)), one block, fixed order
static __global__ void k_reduce_add(const double* part, long n, double* acc) {
    wait_for_stream();
    double v = 0.0;
    for (long q = threadIdx.x; q < n; q += blockDim.x) v += part[q];
    __shared__ double sh[32];
    v = warp_sum(v);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) t += sh[w];
        *acc += t;
    }
}

// The vector algebra between two stages of the RK adjoint over 8 fields: tot += sig (sig null: tot = mu),
// then kap = a mu + b sig (kap null: none).  One launch for what were three of y = a x + b y.
static __global__ void __launch_bounds__(256) k_adj_stage(long n, const __grid_constant__ F8<double> mu, const __grid_constant__ F8<double> sig,
                                                         const __grid_constant__ F8<double> tot, const __grid_constant__ F8<double> kap,
                                                         double a, double b) {
    wait_for_stream();
    const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int m = blockIdx.y;
    const double s = sig.f[0] ? sig.f[m][c] : 0.0;
    if (sig.f[0]) tot.f[m][c] += s;
    else tot.f[m][c] = mu.f[m][c];
    if (kap.f[0]) kap.f[m][c] = a * mu.f[m][c] + b * s;
}

// objective: Phi = (1/my) sum_j sum_i sqrt(Bz(z=0)^2 + eps^2) w_i -> its gradient in Bz
static __global__ void k_adj_flux_seed(Geo<double> g, const double* dbz, const double* wx, double* lam_bz) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.mx) return;
    int j = blockIdx.y;
    if (g.mz % 2) {
        int kc = (g.mz - 1) / 2;
        long c = (long)i + (long)j * g.sy + (long)kc * g.sz;
        double bz = g.bz0[kc] + dbz[c];
        lam_bz[c] = wx[i] * bz / sqrt(bz * bz + 1e-20) / g.my;
    } else {
        int ka = g.mz / 2 - 1, kb = g.mz / 2;
        long ca = (long)i + (long)j * g.sy + (long)ka * g.sz, cb = (long)i + (long)j * g.sy + (long)kb * g.sz;
        double bz = 0.5 * ((g.bz0[ka] + dbz[ca]) + (g.bz0[kb] + dbz[cb]));
        double d = wx[i] * bz / sqrt(bz * bz + 1e-20) / g.my * 0.5;
        lam_bz[ca] = d;
        lam_bz[cb] = d;
    }
}

// psi map transpose: dPhi/dpsi(i,k) = sum_j [ -(Dz^T lam_Bx)(i,j,k) + (Dx^T lam_Bz)(i,j,k) ], the sums
// over y taken first (by k_adj_ysum, in ascending j): sbx, sbz on the (x, z) nodes
static __global__ void k_adj_ysum(Geo<double> g, const double* lbx, const double* lbz, double* sbx, double* sbz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.mx) return;
    const long o = (long)i + (long)blockIdx.y * g.sz;
    double a = 0.0, b = 0.0;
    for (int j = 0; j < g.my; ++j) { a += lbx[o + j * g.sy]; b += lbz[o + j * g.sy]; }
    sbx[(long)i + (long)blockIdx.y * g.mx] = a;
    sbz[(long)i + (long)blockIdx.y * g.mx] = b;
}
static __global__ void k_adj_psi(Geo<double> g, const double* sbx, const double* sbz, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.mx) return;
    const int k = blockIdx.y;
    const DTz dz(g, k, k >= 2 && k + 3 <= g.mz);
    double col[5];
#pragma unroll
    for (int z = 0; z < 5; ++z) {
        const int kk = k - 2 + z;
        col[z] = (kk >= 0 && kk < g.mz) ? sbx[(long)i + (long)kk * g.mx] : 0.0;
    }
    const double* b = sbz + (long)k * g.mx;
    const int i1 = wrapi(i - 1, g.mx), i2 = wrapi(i - 2, g.mx), p1 = wrapi(i + 1, g.mx), p2 = wrapi(i + 2, g.mx);
    out[(long)i + (long)k * g.mx] = -dz.of(col) + b[i] * (-g.a1x[i] + g.b1x[i] - g.c1x[i] + g.d1x[i]) + b[i1] * g.a1x[i1] -
                                    b[p1] * g.b1x[p1] + b[i2] * g.c1x[i2] - b[p2] * g.d1x[p2];
}

}  // namespace dasha
