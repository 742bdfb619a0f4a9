// walls_core.cuh -- the reference's own bounded configuration: the dipole magnetosphere of
// initia (t3dsdsc.f:612-850) with walls on all six sides (periodx = periody = periodz = .false.,
// mhd03.for), the x-min inflow driver (bndry, T:1710-1773), the inner-sphere mask r <= rcr (every
// bndry* routine), the radial Hall coefficient (T:1398) and a 3-D equilibrium (rhoi, bxi, byi, bzi,
// pri).  FP64 throughout, on the reference's own local layout at a 1x1 process grid: arrays
// (mxpr, my, mzpr) with mxpr = mx + 4, mzpr = mz + 4, x fastest, a field stride of
// mxpr*my*mzpr (so an 8-field state is x(mxpr, my, mzpr, 8) exactly), indices written 1-based
// as in the reference: physical nodes jx = 3..mx+2, jy = 1..my, jz = 3..mz+2; interior
// x_first..x_last = 5..mx, 3..my-2, z_first..z_last = 5..mz; boundary rows 3, 4 / mx+1, mx+2,
// 1, 2 / my-1, my and 3, 4 / mz+1, mz+2.
//
// Every routine is a sequence of loops over index boxes; each loop body is a per-node lambda
// run by an executor (`Exec::run(box, f)`; the GPU executor in walls.cu launches one thread per node).  Within a loop no node reads
// what another node of the same loop writes.  Arithmetic follows the reference's expressions term
// by term, with its single-precision constants (REAL*4 literals such as 0.15 or 1.1) as the
// float values they are, so every value has the reference's bits.
//
// The reference runs a smoothing pass as a loop into a work field, a copy back and, for all fields,
// four boundary loops that feed one another (mask, x rows, y rows, z rows): 10 launches a pass of
// three fields and 831 a step.  Here a pass is one loop from one set of fields into another
// (RowRule::each gives a boundary node its final values straight from the interior values they
// derive from, the chain of rules the boundary loops apply), the flux, velocity and E loops are
// one, and the stage update ends the last pass: 87 launches a step with the Hall term on.
// Measured on B200 (ms a step of 41x25x33 / 129x72x101 nodes): 4.24 -> 0.88 / 10.9 -> 4.5.  The passes swap fields
// that are free at that time (J: efld; E: xdh; Hall: xdif 4..6; xdif and the filter: cur, efld, xdh), and the
// work fields w, u, v hold the smoothing coefficient, its x profile and the Hall coefficient of
// every node, which depend on the grid only, so that tanh is not taken per pass.
#pragma once
#include <cmath>
#include <vector>

#include "quotient.h"

#if !defined(__CUDACC__)
#define __host__
#define __device__
#endif
#define WHD __host__ __device__
#ifdef __CUDACC__
#define WALLS_UNROLL _Pragma("unroll")
#else
#define WALLS_UNROLL
#endif

namespace dasha {
namespace walls {

struct Box { int x0, x1, y0, y1, z0, z1; };   // inclusive, 1-based

struct Dims {
    int mx, my, mz, mxpr, mzpr;
    long sy, sz, n;                            // strides (1, mxpr, mxpr*my) and field size
    int x_first, x_last, z_first, z_last, xfirst, xlast, zfirst, zlast;
    WHD long at(int jx, int jy, int jz) const { return (long)(jx - 1) + sy * (jy - 1) + sz * (jz - 1); }
    WHD bool inside(int jx, int jy, int jz) const {   // off the boundary rows
        return jx >= x_first && jx <= x_last && jy >= 3 && jy <= my - 2 && jz >= z_first && jz <= z_last;
    }
};

// 1-D tables, indexed 1-based like the reference's arrays (entry 0 unused)
struct Tables {
    const double *xx, *yy, *zz, *dx, *dy, *dz;
    const double *ax1, *bx1, *cx1, *dx1, *ay1, *by1, *cy1, *dy1, *az1, *bz1, *cz1, *dz1;
    const double *ax2, *bx2, *cx2, *dx2, *ay2, *by2, *cy2, *dy2, *az2, *bz2, *cz2, *dz2;
    const double *axp, *bxp, *cxp;
    const double *hx, *hy, *hz, *rx, *ry, *rz;     // x(j+1) - x(j-1) and its reciprocal (smoothing)
};

struct Par {
    double gamma, eta, mu, drho, dp, cfl, rcr, chall;
    int hall, viscos, diffu;
    int uyzlimiter;
};

// device arrays of one context (padded layout); 8-field arrays hold field m at m*n
struct Arr {
    double *x, *xm, *xfold, *xdif;                 // 8 fields each
    double *cur, *efld, *xdh, *xresd;              // 3 fields each
    double *w, *fs, *gs, *hs, *u, *v;              // work fields
    double *rhoi, *bxi, *byi, *bzi, *pri, *rr0, *rr1;
    unsigned long long* dtbits;                    // setdt minimum (bits of a positive double)
};

WHD inline double d1fc(double fm2, double fm, double f0, double fp, double fp2, double a, double b, double c, double d) {
    return a * (fp - f0) + b * (f0 - fm) + c * (fp2 - f0) + d * (f0 - fm2);
}
// a / b rounded to nearest, r the reciprocal 1 / b rounded to nearest: on the device by two remainder corrections, five
// operations instead of the division's branch and some thirty.  Quotients that could overflow or be subnormal in between, zeros,
// infinities and NaN take the division.
WHD inline double div_by(double a, double b, double r) {
#ifdef __CUDA_ARCH__
    return div_by_steps(a, b, r);
#else
    (void)r;
    return a / b;
#endif
}
// one direction of the smoothing difference: hp, hm the spacings x+ - x0, x0 - x-, h2 = x+ - x-, r2 = 1 / h2
WHD inline double difc(double fm, double f0, double fp, double hp, double hm, double h2, double r2) {
    return div_by(2. * ((fp - f0) * hp - (f0 - fm) * hm), h2, r2);
}
// REAL*4 constants of the reference, widened as Fortran widens them
WHD inline double real4(float v) { return (double)v; }

// ---- derivative helpers at node (jx, jy, jz) of field f ----
struct Deriv {
    Dims d;
    Tables t;
    template <class V>
    WHD double Dx(const V& f, int jx, int jy, int jz) const {
        const long c = d.at(jx, jy, jz);
        return d1fc(f[c - 2], f[c - 1], f[c], f[c + 1], f[c + 2], t.ax1[jx], t.bx1[jx], t.cx1[jx], t.dx1[jx]);
    }
    template <class V>
    WHD double Dy(const V& f, int jx, int jy, int jz) const {
        const long c = d.at(jx, jy, jz), s = d.sy;
        return d1fc(f[c - 2 * s], f[c - s], f[c], f[c + s], f[c + 2 * s], t.ay1[jy], t.by1[jy], t.cy1[jy], t.dy1[jy]);
    }
    template <class V>
    WHD double Dz(const V& f, int jx, int jy, int jz) const {
        const long c = d.at(jx, jy, jz), s = d.sz;
        return d1fc(f[c - 2 * s], f[c - s], f[c], f[c + s], f[c + 2 * s], t.az1[jz], t.bz1[jz], t.cz1[jz], t.dz1[jz]);
    }
    WHD double L2(const double* f, int jx, int jy, int jz) const {   // d2fc x + y + z
        const long c = d.at(jx, jy, jz), sy = d.sy, sz = d.sz;
        return d1fc(f[c - 2], f[c - 1], f[c], f[c + 1], f[c + 2], t.ax2[jx], t.bx2[jx], t.cx2[jx], t.dx2[jx]) +
               d1fc(f[c - 2 * sy], f[c - sy], f[c], f[c + sy], f[c + 2 * sy], t.ay2[jy], t.by2[jy], t.cy2[jy], t.dy2[jy]) +
               d1fc(f[c - 2 * sz], f[c - sz], f[c], f[c + sz], f[c + 2 * sz], t.az2[jz], t.bz2[jz], t.cz2[jz], t.dz2[jz]);
    }
    // the sum of the three difc terms of a smoothing pass (avrg* routines, e.g. T:5643-5648)
    WHD double difc3(const double* f, int jx, int jy, int jz) const {
        const long c = d.at(jx, jy, jz), sy = d.sy, sz = d.sz;
        return difc(f[c - 1], f[c], f[c + 1], t.dx[jx], t.dx[jx - 1], t.hx[jx], t.rx[jx]) +
               difc(f[c - sy], f[c], f[c + sy], t.dy[jy], t.dy[jy - 1], t.hy[jy], t.ry[jy]) +
               difc(f[c - sz], f[c], f[c + sz], t.dz[jz], t.dz[jz - 1], t.hz[jz], t.rz[jz]);
    }
    // the radial smoothing coefficient (avrg, avrgtt, avrgE, avrgc: T:5659-5661 and alike)
    WHD double coef_r(int jx, int jy, int jz) const {
        const double r = sqrt(t.xx[jx] * t.xx[jx] + t.yy[jy] * t.yy[jy] + t.zz[jz] * t.zz[jz]);
        return 1.0 / 32.0 + 0.046875 * (1 + tanh((r - 3.) / 3.));
    }
    // the x profile of the B fields in avrg / avrgtt (T:5636-5642): coef_avrg (1 - tanh((x+3)/8))
    WHD double coef_b(int jx) const { return (1.0 / 32.0) * (1 - tanh((t.xx[jx] + 3) / 8.)); }
};

// Smoothing coefficient kinds: RADIAL (coef_r * sum), BX (coef_b * sum), EIGHTH (1/8 * sum)
enum SmoothKind { SM_RADIAL = 0, SM_BX = 1, SM_EIGHTH = 2 };
// Boundary routine kinds: bndryc, bndryh, bndryE (3 fields, extrapolated x-min rows, y and z rows
// over all x), bndrytt (8 fields, extrapolated x-min rows, y and z rows from x_first), bndry (8
// fields, x-min inflow driver)
enum RowKind { ROWS_C = 0, ROWS_H = 1, ROWS_E = 2, ROWS_TT = 3, ROWS_XDIF = 4 };

// up to 8 fields by pointer
struct Fields { double* f[8]; };

// The nodes of the boundary rows (two at each end of each axis) by number: whole z planes, then y rows
// and x rows between them.
struct Shell {
    int nx, ny, nz, zlast;
    explicit Shell(const Dims& d) : nx(d.mx), ny(d.my), nz(d.mz), zlast(d.zlast) {}
    int count() const { return 4 * (nx * ny + nx * (nz - 4) + (ny - 4) * (nz - 4)); }
    static WHD int end(int q, int n) { return q < 2 ? q : n - 4 + q; }   // rows 0, 1, n-2, n-1
    WHD void node(int i, int& jx, int& jy, int& jz) const {
        const int a = 4 * nx * ny, b = a + 4 * nx * (nz - 4);
        if (i < a) {
            const int r = i / nx;
            jx = i - r * nx; jy = r % ny; jz = end(r / ny, nz);
        } else if (i < b) {
            const int r = (i - a) / nx;
            jx = i - a - r * nx; jy = end(r & 3, ny); jz = 2 + (r >> 2);
        } else {
            const int r = (i - b) >> 2;
            jx = end((i - b) & 3, nx); jy = 2 + r % (ny - 4); jz = 2 + r / (ny - 4);
        }
        jx += 3; jy += 1; jz += 3;
    }
};

// Values before a boundary routine: s(m, jx, jy, jz) of field m.
// A smoothing pass (f + coef * sum difc) on the interior, the field itself elsewhere.
struct Smooth {
    Deriv dv;
    Fields in;
    const double *w, *u;                           // the coefficients of GridCoef
    int kind;
    unsigned bx;                                   // fields (bits) with the x profile
    WHD double operator()(int m, int jx, int jy, int jz) const {
        const long c = dv.d.at(jx, jy, jz);
        const double* f = in.f[m];
        if (!dv.d.inside(jx, jy, jz)) return f[c];
        const double s = dv.difc3(f, jx, jy, jz);
        if (kind == SM_EIGHTH) return f[c] + (1.0 / 8.0) * s;
        if ((bx >> m) & 1u) return f[c] + u[jx - 1] * s;
        return f[c] + w[c] * s;
    }
    // the same at one interior node for several fields: what does not depend on the field, once
    struct At {
        const Smooth& s;
        long c, sy, sz;
        double hp[3], hm[3], h2[3], r2[3], cw, cu;
        WHD double operator()(int m) const {
            const double* f = s.in.f[m] + c;
            const double d3 = difc(f[-1], f[0], f[1], hp[0], hm[0], h2[0], r2[0]) +
                              difc(f[-sy], f[0], f[sy], hp[1], hm[1], h2[1], r2[1]) +
                              difc(f[-sz], f[0], f[sz], hp[2], hm[2], h2[2], r2[2]);
            if (s.kind == SM_EIGHTH) return f[0] + (1.0 / 8.0) * d3;
            if ((s.bx >> m) & 1u) return f[0] + cu * d3;
            return f[0] + cw * d3;
        }
    };
    WHD At at(int jx, int jy, int jz) const {
        const Tables& t = dv.t;
        const long c = dv.d.at(jx, jy, jz);
        return At{*this, c, dv.d.sy, dv.d.sz,
                  {t.dx[jx], t.dy[jy], t.dz[jz]}, {t.dx[jx - 1], t.dy[jy - 1], t.dz[jz - 1]},
                  {t.hx[jx], t.hy[jy], t.hz[jz]}, {t.rx[jx], t.ry[jy], t.rz[jz]},
                  kind == SM_EIGHTH ? 0. : w[c], bx ? u[jx - 1] : 0.};
    }
};
// a value functor at one node, for those with nothing to share between fields
template <class S>
struct NodeOf {
    const S& s;
    int jx, jy, jz;
    WHD double operator()(int m) const { return s(m, jx, jy, jz); }
};
// field m of a value functor as field 0
template <class S>
struct OfField {
    const S& s;
    int m;
    WHD double operator()(int, int jx, int jy, int jz) const { return s(m, jx, jy, jz); }
    WHD NodeOf<OfField> at(int jx, int jy, int jz) const { return {*this, jx, jy, jz}; }
};
// The x-min extrapolation reaches three nodes in, which on a grid of 5 or 6 x nodes is an x-max boundary
// row.  Where the field was just formed on the interior, the reference finds there what the
// last evaluation left: 0 on the outer row (mx = 5), half of the last interior row on the other (kept
// in u behind the coefficient's profile; q = 0 the current, 1 the Hall field).
struct NarrowRows {
    Dims d;
    double* u;
    WHD bool at(int jx) const { return jx > d.x_last; }
    WHD double* row(int q, int m, int jy, int jz) const {
        return u + (3 + 3 * q + m) * ((long)d.my * d.mzpr) + (jy - 1) + (long)d.my * (jz - 1);
    }
    WHD double kept(int q, int m, int jx, int jy, int jz) const { return jx == d.xlast ? 0. : *row(q, m, jy, jz); }
};
// B - B0 at a node and its curl (T:2468-2491; interior nodes)
struct Curl {
    Deriv dv;
    Arr a;
    long n;
    NarrowRows nr;
    struct Pert {
        const double *x, *e;
        WHD double operator[](long c) const { return x[c] - e[c]; }
    };
    WHD double operator()(int m, int jx, int jy, int jz) const {
        if (nr.at(jx)) return nr.kept(0, m, jx, jy, jz);
        const Pert u{a.x + 4 * n, a.bxi}, v{a.x + 5 * n, a.byi}, w{a.x + 6 * n, a.bzi};
        if (m == 0) return dv.Dy(w, jx, jy, jz) - dv.Dz(v, jx, jy, jz);
        if (m == 1) return dv.Dz(u, jx, jy, jz) - dv.Dx(w, jx, jy, jz);
        return dv.Dx(v, jx, jy, jz) - dv.Dy(u, jx, jy, jz);
    }
    WHD NodeOf<Curl> at(int jx, int jy, int jz) const { return {*this, jx, jy, jz}; }
};
// xdh (T:1404-1420; interior nodes)
struct HallField {
    Deriv dv;
    Arr a;
    long n;
    NarrowRows nr;
    WHD double operator()(int m, int jx, int jy, int jz) const {
        if (nr.at(jx)) return nr.kept(1, m, jx, jy, jz);
        const long c = dv.d.at(jx, jy, jz);
        const double* x = a.x;
        const double* cu = a.cur;
        const double* p8 = x + 7 * n;
        const double cht = a.v[c];
        if (m == 0) return cht * (cu[n + c] * x[6 * n + c] - cu[2 * n + c] * x[5 * n + c] - dv.Dx(p8, jx, jy, jz)) / x[c];
        if (m == 1) return cht * (cu[2 * n + c] * x[4 * n + c] - cu[c] * x[6 * n + c] - dv.Dy(p8, jx, jy, jz)) / x[c];
        return cht * (cu[c] * x[5 * n + c] - cu[n + c] * x[4 * n + c] - dv.Dz(p8, jx, jy, jz)) / x[c];
    }
    WHD NodeOf<HallField> at(int jx, int jy, int jz) const { return {*this, jx, jy, jz}; }
};
struct Stored {
    const double* f;
    Dims d;
    long n;
    WHD double operator()(int m, int jx, int jy, int jz) const { return f[m * n + d.at(jx, jy, jz)]; }
    WHD NodeOf<Stored> at(int jx, int jy, int jz) const { return {*this, jx, jy, jz}; }
};

// The boundary routines (bndry*, T:1677-3027), a loop each in the reference: mask (0 inside the
// sphere r <= rcr), x rows, y rows, z rows, each reading what the one before left.  each() gives a
// node the values all of them leave there, from the values s before them.
struct RowRule {
    Dims d;
    Tables t;
    int kind;
    const double* rr1;
    double rcr;
    bool uyz;
    const double *rhoi, *bxi, *byi, *bzi, *pri;    // ROWS_XDIF: the driver
    const double* ref;                             // the state at the start of the step
    double tt, ddt;

    template <class S>
    WHD double masked(const S& s, int m, int jx, int jy, int jz) const {
        return rr1[d.at(jx, jy, jz)] <= rcr ? 0. : s(m, jx, jy, jz);
    }
    // the state of the x-min rows 4 and 3 under the inflow driver (T:1710-1773): the equilibrium
    // plus a time-dependent density / velocity / pressure pulse.  rhoi(4,jz,jz) and rhoi(3,jz,jz)
    // index y by jz as the reference does (its defect D3), read at the same linear position of the
    // array.  (products in the reference's left-to-right order)
    WHD double driven_state(int m, int row, int jy, int jz) const {
        if (m == 2 || m == 3) return 0.;
        const long c = d.at(row, jy, jz);
        if (m >= 4 && m <= 6) {
            // B pulse times the file field bxinfc, byinfc, bzinfc, which is 0 without the fcinp/ files
            // (mxdatfc = .false.)
            const double bpulse = 0. * real4(0.0017f) * sqrt(tt * tt * tt * real4(7.25f) * real4(7.25f) * real4(7.25f)) /
                                  (exp(tt * real4(7.25f) * real4(0.0069f)) + 1.);
            return (m == 4 ? bxi : (m == 5 ? byi : bzi))[c] + bpulse;
        }
        const double zz = t.zz[jz], yy = t.yy[jy];
        const double at = tanh((tt - 9.) / 1.) - tanh((tt - 39.) / 1.5);
        const double bz6 = tanh((zz + real4(0.6f)) / real4(0.15f)) - tanh((zz - real4(0.6f)) / real4(0.15f));
        const double by4 = tanh((yy + real4(0.4f)) / real4(0.15f)) - tanh((yy - real4(0.4f)) / real4(0.15f));
        if (m == 7) return pri[c] + (double)(0.2f * 0.5f) * at * 0.5 * bz6 * 0.5 * by4;
        const double x1 = rhoi[d.at(row, jz, jz)] + 0.5 * at * 0.5 * bz6 * 0.5 * by4;
        if (m == 0) return x1;
        const double bz2 = tanh((zz + real4(0.2f)) / real4(0.15f)) - tanh((zz - real4(0.2f)) / real4(0.15f));
        const double by3 = tanh((yy + real4(0.3f)) / real4(0.15f)) - tanh((yy - real4(0.3f)) / real4(0.15f));
        return real4(0.8f) * x1 * 0.5 * at * 0.5 * bz2 * 0.5 * by3;
    }
    // the x-min rows 3 and 4 at (jy, jz), before the y and z rows
    template <class S>
    WHD double x_min(const S& s, int m, int jx, int jy, int jz) const {
        if (kind == ROWS_XDIF)                     // the rate (state - start of the step) / (ddt + 1e-9)
            return (driven_state(m, jx, jy, jz) - ref[m * d.n + d.at(jx, jy, jz)]) / (ddt + 1.e-9);
        // third-order extrapolation with the one-sided weights axp, bxp, cxp (T:505-517)
        const double f5 = masked(s, m, 5, jy, jz), f6 = masked(s, m, 6, jy, jz), f7 = masked(s, m, 7, jy, jz);
        const double f4 = (t.axp[4] * f5 + t.bxp[4] * f6 + t.cxp[4] * f7) / (t.axp[4] + t.bxp[4] + t.cxp[4]);
        if (jx == 4) return f4;
        return (t.axp[3] * f4 + t.bxp[3] * f5 + t.cxp[3] * f6) / (t.axp[3] + t.bxp[3] + t.cxp[3]);
    }
    // the uy/uz limiter of bndry and bndrytt (T:1928-1975, 2231-2278): on the two wall rows at each z
    // end the z momentum, on the two rows at each y end the y momentum, may only point into
    // the domain
    WHD double limited(double v, int m, int jx, int jy, int jz) const {
        if (uyz && jx >= d.x_first) {
            if (m == 3 && ((jz <= 4 && v >= 0.) || (jz >= d.zlast - 1 && v <= 0.))) v = 0.;
            if (m == 2 && ((jy <= 2 && v >= 0.) || (jy >= d.my - 1 && v <= 0.))) v = 0.;
        }
        return v;
    }
    // out(m, value of field m at the node) for fields 0 .. NF-1, behind the x-min rows (jx > 4)
    template <int NF, class S, class Out>
    WHD void each(const S& s, int jx, int jy, int jz, const Out& out) const {
        // the rows next to a wall are half of their inner neighbours, the walls 0
        if (jz == 3 || jz == d.zlast || jy == 1 || jy == d.my || jx == d.xlast) {
            for (int m = 0; m < NF; ++m) out(m, 0.);
            return;
        }
        const bool hz = jz == 4 || jz == d.zlast - 1, hy = jy == 2 || jy == d.my - 1, hx = jx == d.xlast - 1;
        const int sx = hx ? jx - 1 : jx, sy = hy ? (jy == 2 ? 3 : d.my - 2) : jy, sz = hz ? (jz == 4 ? 5 : d.zlast - 2) : jz;
        const bool off = rr1[d.at(sx, sy, sz)] <= rcr;
        const auto at = s.at(sx, sy, sz);
        WALLS_UNROLL
        for (int m = 0; m < NF; ++m) {
            double v = off ? 0. : at(m);
            if (hx) v = 0.5 * v;
            if (hy) v = 0.5 * v;
            if (hz) v = 0.5 * v;
            out(m, limited(v, m, jx, jy, jz));
        }
    }
    // field m on the x-min rows 3 and 4
    template <class S>
    WHD double x_min_row(const S& s, int m, int jx, int jy, int jz) const {
        if (kind == ROWS_TT) return x_min(s, m, jx, jy, jz);   // bndrytt's y and z rows start behind them
        if (jz == 3 || jz == d.zlast || jy == 1 || jy == d.my) return 0.;
        const bool hz = jz == 4 || jz == d.zlast - 1, hy = jy == 2 || jy == d.my - 1;
        double v = x_min(s, m, jx, hy ? (jy == 2 ? 3 : d.my - 2) : jy, hz ? (jz == 4 ? 5 : d.zlast - 2) : jz);
        if (hy) v = 0.5 * v;
        if (hz) v = 0.5 * v;
        return v;
    }
};

// A loop over the physical nodes that gives every field its values after a boundary routine: out(m, c,
// value) with c the node's index.  The nodes behind the x-min rows take a thread for all NF fields, or one
// per field (split) on small grids.  Split threads are shorter, but do what the fields share NF times, so they
// win while they all run at once.  Loops of 3 fields turn a little above one wave of eight blocks of 128 an SM (the threads of
// the boundary rows are short): ms a step with their loops split / not, 52896 nodes 0.681 / 0.748, 54180 0.721 / 0.736, 58800
// 0.855 / 0.781, 60000 0.936 / 0.809.  Loops of 8 fields, which share more of the work, turn at the same
// size (52896 0.733 / 0.748, 58800 0.771 / 0.781, 60000 0.828 / 0.809, 64000 0.792 / 0.771), so one line serves
// both: 9/8 of a wave of 3-field threads.  All loops: 9600 nodes 0.549 / 0.648, 33825 0.632 / 0.745,
// 84150 0.964 / 0.849, 464520 3.63 / 2.87, 997458 7.41 / 5.79.  Those of the x-min rows, three smoothed values each, come after
// them with a thread per field, so that no warp holds both (10.3 ms a step with them in line).
template <int NF, class S, class Out>
struct RowLoop {
    S s;
    RowRule rr;
    Out out;
    bool split;
    WHD void operator()(int i, int, int) const {
        const Dims& d = rr.d;
        const unsigned nx = (unsigned)(d.mx - 2), ny = (unsigned)d.my;
        const unsigned main = nx * ny * (unsigned)d.mz * (split ? NF : 1);
        unsigned q = (unsigned)(i - 1);
        if (split && q < main) {
            const int m = (int)(q % NF);
            q /= NF;
            const unsigned r = q / nx;
            const int jx = 5 + (int)(q - r * nx), jy = 1 + (int)(r % ny), jz = 3 + (int)(r / ny);
            const long c = d.at(jx, jy, jz);
            rr.template each<1>(OfField<S>{s, m}, jx, jy, jz, [&](int, double v) { out(m, c, rr.limited(v, m, jx, jy, jz)); });
        } else if (q < main) {
            const unsigned r = q / nx;
            const int jx = 5 + (int)(q - r * nx), jy = 1 + (int)(r % ny), jz = 3 + (int)(r / ny);
            const long c = d.at(jx, jy, jz);
            rr.template each<NF>(s, jx, jy, jz, [&](int m, double v) { out(m, c, v); });
        } else {
            q -= main;
            const int m = (int)(q % NF), jx = 3 + (int)(q / NF & 1u);
            const unsigned r = q / NF >> 1;
            const int jy = 1 + (int)(r % ny), jz = 3 + (int)(r / ny);
            out(m, d.at(jx, jy, jz), rr.x_min_row(s, m, jx, jy, jz));
        }
    }
};

template <class Exec>
struct Core {
    Exec& ex;
    Dims d;
    Tables t;
    Par p;
    Arr a;

    Deriv D() const { return Deriv{d, t}; }
    Box physical() const { return {d.x_first - 2, d.x_last + 2, 1, d.my, d.z_first - 2, d.z_last + 2}; }
    Box interior() const { return {d.x_first, d.x_last, 3, d.my - 2, d.z_first, d.z_last}; }

    Fields fields(double* base, int nf = 8) const {
        Fields r{};
        for (int m = 0; m < nf; ++m) r.f[m] = base + m * d.n;
        return r;
    }
    // 8 fields free while xdif (or the filtered perturbation) is smoothed
    Fields spare8() const {
        Fields r{};
        for (int m = 0; m < 3; ++m) { r.f[m] = a.cur + m * d.n; r.f[3 + m] = a.efld + m * d.n; }
        r.f[6] = a.xdh;
        r.f[7] = a.xdh + d.n;
        return r;
    }
    RowRule rule(int kind, double tt = 0., double ddt = 0., int km = 1) const {
        RowRule r{};
        r.d = d; r.t = t; r.kind = kind; r.rr1 = a.rr1; r.rcr = p.rcr;
        r.uyz = p.uyzlimiter && (kind == ROWS_XDIF || kind == ROWS_TT);
        r.rhoi = a.rhoi; r.bxi = a.bxi; r.byi = a.byi; r.bzi = a.bzi; r.pri = a.pri;
        r.ref = km == 1 ? a.xfold : a.xm;
        r.tt = tt; r.ddt = ddt;
        return r;
    }
    Smooth smoother(const Fields& in, int kind, unsigned bx = 0) const { return Smooth{D(), in, a.w, a.u, kind, bx}; }

    // ---- coefficients of the grid: w the radial smoothing coefficient, u(jx) its x profile for the B
    // fields (at linear position jx-1), v the Hall coefficient cht = 0.5 chall (tanh((r0 - 1.1)/8) -
    // tanh((r0 - 2)/10)) (T:1396-1399) ----
    struct GridCoef {
        Deriv dv;
        Arr a;
        double chall;
        WHD void operator()(int jx, int jy, int jz) const {
            const long c = dv.d.at(jx, jy, jz);
            a.w[c] = dv.coef_r(jx, jy, jz);
            const double r0 = a.rr0[c];
            a.v[c] = 0.5 * chall * (tanh((r0 - real4(1.1f)) / 8.) - tanh((r0 - 2.) / 10.));
            if (jy == 1 && jz == 3) a.u[jx - 1] = dv.coef_b(jx);
        }
    };
    GridCoef grid_coef() const { return GridCoef{D(), a, p.chall}; }

    // ---- one smoothing pass with its boundary routine, `in` into `out` ----
    template <int NF>
    void pass(const Smooth& sm, const RowRule& rr, const Fields& out) {
        rows<NF>(sm, rr, [=] WHD(int m, long c, double v) { out.f[m][c] = v; });
    }
    template <int NF, class S, class Out>
    void rows(const S& s, const RowRule& rr, const Out& out) {
        const bool split = 3L * d.mx * d.my * d.mz <= 148L * 9 * 128;
        ex.run({1, ((d.mx - 2) * (split ? NF : 1) + 2 * NF) * d.my * d.mz, 1, 1, 1, 1}, RowLoop<NF, S, Out>{s, rr, out, split});
    }

    // ---- current (T:2452-2500): J = curl(B - B0), bndryc, avrgc(1,3,4) ----
    void current() {
        ex.run(physical(), grid_coef());
        smoothed_current();
    }
    void smoothed_current() {
        const Dims dd = d;
        const RowRule rc = rule(ROWS_C);
        const NarrowRows nr{d, a.u};
        const Curl cu{D(), a, d.n, nr};
        double* cur = a.cur;
        const long n = d.n;
        rows<3>(cu, rc, [=] WHD(int m, long c, double v) { cur[m * n + c] = v; });
        const Fields j = fields(a.cur, 3), q = fields(a.efld, 3);
        for (int k = 0; k < 2; ++k) {
            pass<3>(smoother(j, SM_RADIAL), rc, q);
            pass<3>(smoother(q, SM_RADIAL), rc, j);
        }
        if (d.mx <= 6)
            ex.run({d.xlast - 1, d.xlast - 1, 1, d.my, 3, d.zlast}, [=] WHD(int jx, int jy, int jz) {
                for (int m = 0; m < 3; ++m) *nr.row(0, m, jy, jz) = j.f[m][dd.at(jx, jy, jz)];
            });
    }

    // ---- right (T:1297-1673) with totalE = .true.: xdif = dx/dt of the state x ----
    void right(double tt, double ddt, int km) {
        ex.run(physical(), grid_coef());
        rates(tt, ddt, km);
        if (tt != 0.) {                                              // avrg(t, ddt, km, 1, 8, 0, 2)
            const RowRule rx = rule(ROWS_XDIF, tt, ddt, km);
            const Fields k = fields(a.xdif), q = spare8();
            pass<8>(smoother(k, SM_RADIAL, 0x70u), rx, q);
            pass<8>(smoother(q, SM_RADIAL, 0x70u), rx, k);
        }
    }

    // xdif with its boundary rows, before avrg
    void rates(double tt, double ddt, int km) {
        const Dims dd = d;
        const Deriv dv = D();
        const Arr aa = a;
        const Par pp = p;
        const long n = d.n;
        smoothed_current();
        // every node: the six products of the momentum fluxes (flux, T:2286-2347; xdh and xdif 4..6 are
        // free here), velocity and E = (-v x B) + eta J (T:1348-1373)
        ex.run(physical(), [=] WHD(int jx, int jy, int jz) {
            const long c = dd.at(jx, jy, jz);
            const double* x = aa.x;
            const double* cu = aa.cur;
            const double x1 = x[c], x2 = x[n + c], x3 = x[2 * n + c], x4 = x[3 * n + c], dp = x[7 * n + c] - aa.pri[c];
            double* p1 = aa.xdh;
            double* p2 = aa.xdif + 4 * n;
            const double r1 = 1. / x1;
            p1[c] = div_by(x2 * x2, x1, r1) + dp;
            p1[n + c] = div_by(x2 * x3, x1, r1);
            p1[2 * n + c] = div_by(x2 * x4, x1, r1);
            p2[c] = div_by(x3 * x3, x1, r1) + dp;
            p2[n + c] = div_by(x4 * x3, x1, r1);
            p2[2 * n + c] = div_by(x4 * x4, x1, r1) + dp;
            aa.fs[c] = div_by(x2, x1, r1);
            aa.gs[c] = div_by(x3, x1, r1);
            aa.hs[c] = div_by(x4, x1, r1);
            aa.efld[c] = div_by(-x3 * x[6 * n + c] + x4 * x[5 * n + c], x1, r1) + pp.eta * cu[c];
            aa.efld[n + c] = div_by(-x4 * x[4 * n + c] + x2 * x[6 * n + c], x1, r1) + pp.eta * cu[n + c];
            aa.efld[2 * n + c] = div_by(-x2 * x[5 * n + c] + x3 * x[4 * n + c], x1, r1) + pp.eta * cu[2 * n + c];
        });
        // continuity and momentum: -div of the fluxes, J x B - xresd
        ex.run(interior(), [=] WHD(int jx, int jy, int jz) {
            const long c = dd.at(jx, jy, jz);
            const double* x = aa.x;
            const double* cu = aa.cur;
            const double* p1 = aa.xdh;
            const double* p2 = aa.xdif + 4 * n;
            WALLS_UNROLL
            for (int m = 0; m < 4; ++m) {
            const double* fs = m == 0 ? x + n : (m == 1 ? p1 : (m == 2 ? p1 + n : p1 + 2 * n));
            const double* gs = m == 0 ? x + 2 * n : (m == 1 ? p1 + n : (m == 2 ? p2 : p2 + n));
            const double* hs = m == 0 ? x + 3 * n : (m == 1 ? p1 + 2 * n : (m == 2 ? p2 + n : p2 + 2 * n));
            double r = -dv.Dx(fs, jx, jy, jz) - dv.Dy(gs, jx, jy, jz) - dv.Dz(hs, jx, jy, jz);
            if (m == 1) r = r - aa.xresd[c] + cu[n + c] * x[6 * n + c] - cu[2 * n + c] * x[5 * n + c];
            if (m == 2) r = r - aa.xresd[n + c] + cu[2 * n + c] * x[4 * n + c] - cu[c] * x[6 * n + c];
            if (m == 3) r = r - aa.xresd[2 * n + c] + cu[c] * x[5 * n + c] - cu[n + c] * x[4 * n + c];
            aa.xdif[m * n + c] = r;
            }
        });
        const RowRule re = rule(ROWS_E);
        const Fields e = fields(a.efld, 3), h = fields(a.xdh, 3), q = fields(a.xdif + 4 * n, 3);
        for (int k = 0; k < 2; ++k) {                               // avrgE(t, 1, 3, 4)
            pass<3>(smoother(e, SM_RADIAL), re, h);
            pass<3>(smoother(h, SM_RADIAL), re, e);
        }
        if (p.hall) {
            const RowRule rh = rule(ROWS_H);
            const NarrowRows nr{d, a.u};
            const HallField hf{dv, aa, n, nr};
            rows<3>(hf, rh, [=] WHD(int m, long c, double v) { h.f[m][c] = v; });
            for (int k = 0; k < 2; ++k) {                           // avrgh(1, 3, 5)
                pass<3>(smoother(h, SM_EIGHTH), rh, q);
                pass<3>(smoother(q, SM_EIGHTH), rh, h);
            }
            const Smooth sm = smoother(h, SM_EIGHTH);               // the fifth, added to E
            if (d.mx <= 6)
                ex.run({d.xlast - 1, d.xlast - 1, 1, d.my, 3, d.zlast}, [=] WHD(int jx, int jy, int jz) {
                    rh.template each<3>(sm, jx, jy, jz, [&](int m, double v) { *nr.row(1, m, jy, jz) = v; });
                });
            rows<3>(sm, rh, [=] WHD(int m, long c, double v) { e.f[m][c] = e.f[m][c] + v; });
        }
        // induction -curl E and the pressure equation (T:1434-1566); viscosity and diffusion
        // (T:1585-1663), where with a zero coefficient the reference adds zero
        const bool visc = p.viscos && p.mu != 0., diff = p.diffu && (p.drho != 0. || p.dp != 0.);
        ex.run(interior(), [=] WHD(int jx, int jy, int jz) {
            const long c = dd.at(jx, jy, jz);
            const double* e = aa.efld;
            const double* x = aa.x;
            double* xd = aa.xdif;
            const double* cu = aa.cur;
            xd[4 * n + c] = -dv.Dy(e + 2 * n, jx, jy, jz) + dv.Dz(e + n, jx, jy, jz);
            xd[5 * n + c] = -dv.Dz(e, jx, jy, jz) + dv.Dx(e + 2 * n, jx, jy, jz);
            xd[6 * n + c] = -dv.Dx(e + n, jx, jy, jz) + dv.Dy(e, jx, jy, jz);
            const double* p8 = x + 7 * n;
            double r = -dv.Dx(p8, jx, jy, jz) * aa.fs[c] - dv.Dy(p8, jx, jy, jz) * aa.gs[c] -
                       dv.Dz(p8, jx, jy, jz) * aa.hs[c] +
                       (-dv.Dx(aa.fs, jx, jy, jz) - dv.Dy(aa.gs, jx, jy, jz) - dv.Dz(aa.hs, jx, jy, jz)) *
                           pp.gamma * x[7 * n + c] +
                       (pp.gamma - 1.) * pp.eta * (cu[c] * cu[c] + cu[n + c] * cu[n + c] + cu[2 * n + c] * cu[2 * n + c]);
            if (visc) {
                const double af = dv.L2(aa.fs, jx, jy, jz), ag = dv.L2(aa.gs, jx, jy, jz), ah = dv.L2(aa.hs, jx, jy, jz);
                xd[n + c] = xd[n + c] + pp.mu * af;
                xd[2 * n + c] = xd[2 * n + c] + pp.mu * ag;
                xd[3 * n + c] = xd[3 * n + c] + pp.mu * ah;
                r = r + pp.mu * (aa.fs[c] * af + aa.gs[c] * ag + aa.hs[c] * ah);
            }
            if (diff) {
                xd[c] = xd[c] + pp.drho * dv.L2(aa.x, jx, jy, jz);
                r = r + pp.dp * dv.L2(p8, jx, jy, jz);
            }
            xd[7 * n + c] = r;
            if (aa.rr1[c] <= pp.rcr)                                 // the mask of bndry
                for (int m = 0; m < 8; ++m) xd[m * n + c] = 0.;
        });
        // the boundary rows (from interior values), and the driven rows of the state
        const RowRule rx = rule(ROWS_XDIF, tt, ddt, km);
        const Stored st{aa.xdif, dd, n};
        const Shell sh(d);
        ex.run({1, 8 * sh.count(), 1, 1, 1, 1}, [=] WHD(int i, int, int) {
            int jx, jy, jz;
            const int m = (i - 1) & 7;
            sh.node((i - 1) >> 3, jx, jy, jz);
            const long c = dd.at(jx, jy, jz);
            if (jx <= 4) {
                aa.xdif[m * n + c] = rx.x_min_row(st, m, jx, jy, jz);
                aa.x[m * n + c] = rx.driven_state(m, jx, jy, jz);
            } else {
                rx.template each<1>(OfField<Stored>{st, m}, jx, jy, jz, [&](int, double v) { aa.xdif[m * n + c] = rx.limited(v, m, jx, jy, jz); });
            }
        });
    }

    // ---- stepon (T:1063-1172): RK4 registers xfold, xm, x; then avrgtt on x - eq ----
    void stepon(double time, double dt) {
        const Dims dd = d;
        const Arr aa = a;
        const long n = d.n;
        const GridCoef gc = grid_coef();
        ex.run(physical(), [=] WHD(int jx, int jy, int jz) {
            const long c = dd.at(jx, jy, jz);
            gc(jx, jy, jz);
            for (int m = 0; m < 8; ++m) aa.xfold[m * n + c] = aa.x[m * n + c];
        });
        const double tts[4] = {time + dt / 2, time + dt / 2, time + dt, time + dt};
        const double ddts[4] = {dt / 2., dt / 2., dt, dt / 6.};
        const Fields q = spare8(), xd = fields(a.xdif);
        // the equilibrium parts of the state (null: none)
        Fields eq{};
        eq.f[0] = a.rhoi; eq.f[4] = a.bxi; eq.f[5] = a.byi; eq.f[6] = a.bzi; eq.f[7] = a.pri;
        for (int s = 0; s < 4; ++s) {
            const int km = s == 3 ? 2 : 1;
            const double tt = tts[s], ddt = ddts[s];
            rates(tt, ddt, km);
            RowRule rx = rule(ROWS_XDIF, tt, ddt, km);
            if (tt != 0.) pass<8>(smoother(xd, SM_RADIAL, 0x70u), rx, q);   // avrg(t, ddt, km, 1, 8, 0, 2)
            const Smooth sm = smoother(q, SM_RADIAL, 0x70u);
            // the second pass and the stage update; after the last stage x - eq goes to xdif
            const auto update = [=] WHD(int m, long c, double k) {
                    const long i = m * n + c;
                    if (s == 0) { aa.xm[i] = aa.xfold[i] + k * dt / 6.; aa.x[i] = aa.xfold[i] + k * dt / 2.; }
                    else if (s == 1) { aa.xm[i] = aa.xm[i] + k * dt / 3.; aa.x[i] = aa.xfold[i] + k * dt / 2.; }
                    else if (s == 2) { aa.xm[i] = aa.xm[i] + k * dt / 3.; aa.x[i] = aa.xfold[i] + k * dt; }
                    else {
                        const double v = aa.xm[i] + k * dt / 6.;
                        aa.xdif[i] = eq.f[m] ? v - eq.f[m][c] : v;
                    }
            };
            if (tt != 0.) rows<8>(sm, rx, update);
            else ex.run(physical(), [=] WHD(int jx, int jy, int jz) {
                const long c = dd.at(jx, jy, jz);
                for (int m = 0; m < 8; ++m) update(m, c, aa.xdif[m * n + c]);
            });
        }
        const RowRule rt = rule(ROWS_TT, time + dt);                 // avrgtt(tt, 1, 8, 0, 2)
        pass<8>(smoother(xd, SM_RADIAL, 0x70u), rt, q);
        const Smooth sm = smoother(q, SM_RADIAL, 0x70u);
        rows<8>(sm, rt, [=] WHD(int m, long c, double v) { aa.x[m * n + c] = eq.f[m] ? v + eq.f[m][c] : v; });
    }

    // ---- setdt (T:4694-4810): min over the cells with r >= 1 of the region zfirst..z_last,
    // 1..my-1, xfirst..x_last; one atomicMin on the bits of the positive double ----
    void setdt_launch() {
        const Dims dd = d;
        const Tables tb = t;
        const Arr aa = a;
        const Par pp = p;
        const long n = d.n;
        ex.run({d.xfirst, d.x_last, 1, d.my - 1, d.zfirst, d.z_last}, [=] WHD(int jx, int jy, int jz) {
            const long c = dd.at(jx, jy, jz);
            if (!(aa.rr1[c] >= 1.)) return;
            const double* x = aa.x;
            const double vx = x[n + c] / x[c], vy = x[2 * n + c] / x[c], vz = x[3 * n + c] / x[c];
            const double va2 = (x[4 * n + c] * x[4 * n + c] + x[5 * n + c] * x[5 * n + c] + x[6 * n + c] * x[6 * n + c]) / x[c];
            const double cs2 = pp.gamma * x[7 * n + c] / x[c];
            const double vpx = fabs(vx) + sqrt(fabs(va2 + cs2));
            const double vpy = fabs(vy) + sqrt(fabs(va2 + cs2));
            const double vpz = fabs(vz) + sqrt(fabs(va2 + cs2));
            const double vis = pp.eta + pp.mu;
            const double dtx = fabs(tb.dx[jx]) / (vpx / pp.cfl + vis / tb.dx[jx] / 2.);
            const double dty = fabs(tb.dy[jy]) / (vpy / pp.cfl + vis / tb.dy[jy] / 2.);
            const double dtz = fabs(tb.dz[jz]) / (vpz / pp.cfl + vis / tb.dz[jz] / 2.);
            const double dt1 = dtx < dty ? dtx : dty;
            const double dt2 = dtz < dt1 ? dtz : dt1;
            Exec::atomic_min_bits(aa.dtbits, dt2);
        });
    }
};


// ---- host set-up, shared by the device engine (walls.cu) and host builds of this core ----

// index ranges of a 1x1 process grid (t3dsdsc.f:60-81)
inline Dims make_dims(int mx, int my, int mz) {
    Dims d{};
    d.mx = mx; d.my = my; d.mz = mz; d.mxpr = mx + 4; d.mzpr = mz + 4;
    d.sy = d.mxpr; d.sz = (long)d.mxpr * my; d.n = d.sz * d.mzpr;
    d.x_first = 5; d.x_last = mx; d.z_first = 5; d.z_last = mz;
    d.xfirst = 3; d.xlast = mx + 2; d.zfirst = 3; d.zlast = mz + 2;
    return d;
}

// x**k as the reference's translation evaluates integer powers: repeated multiplication
inline double ipow2(double a) { return a * a; }
inline double ipow3(double a) { return a * a * a; }
inline double ipow4(double a) { const double b = a * a; return b * b; }

// The 1-D tables of input on the padded index (entry 0 unused), in the order of the members of
// Tables: xx yy zz dx dy dz; the first-derivative weights a b c d of x, y, z (T:439-504); the
// second-derivative weights (T:336-364); the one-sided weights axp bxp cxp toward +x
// (T:505-517); the spans x(j+1) - x(j-1) of x, y, z and their reciprocals (interior nodes).
// Spacings are forward differences, the last one repeated.
constexpr int NTAB = 6 + 12 + 12 + 3 + 6;
inline std::vector<std::vector<double>> make_tables(const Dims& d, const double* xc, const double* yc,
                                                    const double* zc) {
    const int mx = d.mx, my = d.my, mz = d.mz;
    const int L[3] = {d.mxpr + 1, my + 1, d.mzpr + 1};
    std::vector<double> xx(L[0], 0.), yy(L[1], 0.), zz(L[2], 0.), dx(L[0], 0.), dy(L[1], 0.), dz(L[2], 0.);
    auto fwd = [](const double* c, int nn, int i) { return i + 1 < nn ? c[i + 1] - c[i] : c[i] - c[i - 1]; };
    for (int i = 0; i < mx; ++i) { xx[i + 3] = xc[i]; dx[i + 3] = fwd(xc, mx, i); }
    for (int j = 0; j < my; ++j) { yy[j + 1] = yc[j]; dy[j + 1] = fwd(yc, my, j); }
    for (int k = 0; k < mz; ++k) { zz[k + 3] = zc[k]; dz[k + 3] = fwd(zc, mz, k); }
    std::vector<double> c1[3][4], c2[3][4], cp[3];
    const std::vector<double>* crd[3] = {&xx, &yy, &zz};
    const int lo[3] = {d.x_first, 3, d.z_first}, hi[3] = {d.x_last, my - 2, d.z_last};
    for (int ax = 0; ax < 3; ++ax) {
        for (int q = 0; q < 4; ++q) { c1[ax][q].assign(L[ax], 0.); c2[ax][q].assign(L[ax], 0.); }
        const std::vector<double>& c = *crd[ax];
        for (int j = lo[ax]; j <= hi[ax]; ++j) {
            const double dxp1 = c[j + 1] - c[j], dxm1 = c[j] - c[j - 1], dxp2 = c[j + 2] - c[j], dxm2 = c[j] - c[j - 2];
            {   // second derivative (T:336-364)
                const double f1 = ipow2(dxp1) + dxp1 * dxm2, f2 = ipow3(dxp1) - dxp1 * ipow2(dxm2),
                             f3 = ipow4(dxp1) + dxp1 * ipow3(dxm2);
                const double g1 = -ipow2(dxm1) + dxm1 * dxm2, g2 = ipow3(dxm1) - dxm1 * ipow2(dxm2),
                             g3 = -ipow4(dxm1) + dxm1 * ipow3(dxm2);
                const double h1 = ipow2(dxp2) + dxp2 * dxm2, h2 = ipow3(dxp2) - dxp2 * ipow2(dxm2),
                             h3 = ipow4(dxp2) + dxp2 * ipow3(dxm2);
                const double ca = (f1 * h3 - f3 * h1) * (g2 * h3 - g3 * h2) - (g1 * h3 - g3 * h1) * (f2 * h3 - f3 * h2);
                const double a2 = 2. * h3 * (g2 * h3 - g3 * h2) / ca, b2 = 2. * h3 * (h2 * f3 - h3 * f2) / ca;
                const double cc2 = 2. * h3 * (f2 * g3 - f3 * g2) / ca;
                c2[ax][0][j] = a2; c2[ax][1][j] = b2; c2[ax][2][j] = cc2;
                c2[ax][3][j] = -(dxp1 * a2 + dxm1 * b2 + dxp2 * cc2) / dxm2;
            }
            {   // first derivative (T:439-504)
                const double f1 = dxp1 + ipow4(dxp1) / ipow3(dxm2), f2 = ipow2(dxp1) - ipow4(dxp1) / ipow2(dxm2),
                             f3 = ipow3(dxp1) + ipow4(dxp1) / dxm2;
                const double g1 = dxm1 - ipow4(dxm1) / ipow3(dxm2), g2 = -ipow2(dxm1) + ipow4(dxm1) / ipow2(dxm2),
                             g3 = ipow3(dxm1) - ipow4(dxm1) / dxm2;
                const double h1 = dxp2 + ipow4(dxp2) / ipow3(dxm2), h2 = ipow2(dxp2) - ipow4(dxp2) / ipow2(dxm2),
                             h3 = ipow3(dxp2) + ipow4(dxp2) / dxm2;
                const double ca = (f1 * h3 - f3 * h1) * (g2 * h3 - g3 * h2) - (g1 * h3 - g3 * h1) * (f2 * h3 - f3 * h2);
                const double a1 = h3 * (g2 * h3 - g3 * h2) / ca, b1 = h3 * (h2 * f3 - h3 * f2) / ca,
                             cc1 = h3 * (f2 * g3 - f3 * g2) / ca;
                c1[ax][0][j] = a1; c1[ax][1][j] = b1; c1[ax][2][j] = cc1;
                c1[ax][3][j] = (ipow2(dxp1) * a1 - ipow2(dxm1) * b1 + ipow2(dxp2) * cc1) / ipow2(dxm2);
            }
        }
    }
    for (int q = 0; q < 3; ++q) cp[q].assign(L[0], 0.);
    for (int j = d.xfirst; j <= d.xlast - 3; ++j) {
        const double dxp1 = xx[j + 1] - xx[j], dxp2 = xx[j + 2] - xx[j], dxp3 = xx[j + 3] - xx[j];
        const double f1 = dxp1 - ipow3(dxp1) / ipow2(dxp3), f2 = ipow2(dxp1) - ipow3(dxp1) / dxp3;
        const double g1 = dxp2 - ipow3(dxp2) / ipow2(dxp3), g2 = ipow2(dxp2) - ipow3(dxp2) / dxp3;
        const double ca = f1 * g2 - f2 * g1;
        cp[0][j] = g2 / ca;
        cp[1][j] = -f2 / ca;
        cp[2][j] = (1 - cp[0][j] * dxp1 - cp[1][j] * dxp2) / dxp3;
    }
    std::vector<std::vector<double>> out{xx, yy, zz, dx, dy, dz};
    for (int ax = 0; ax < 3; ++ax) for (int q = 0; q < 4; ++q) out.push_back(c1[ax][q]);
    for (int ax = 0; ax < 3; ++ax) for (int q = 0; q < 4; ++q) out.push_back(c2[ax][q]);
    for (int q = 0; q < 3; ++q) out.push_back(cp[q]);
    for (int inverse = 0; inverse < 2; ++inverse)
        for (int ax = 0; ax < 3; ++ax) {
            std::vector<double> h(L[ax], 0.);
            for (int j = lo[ax]; j <= hi[ax]; ++j) {
                const double span = (*crd[ax])[j + 1] - (*crd[ax])[j - 1];
                h[j] = inverse ? 1. / span : span;
            }
            out.push_back(h);
        }
    return out;
}

// Tables from NTAB pointers in the order of make_tables
inline void bind_tables(Tables& t, const double* const* p) {
    int o = 0;
    t.xx = p[o++]; t.yy = p[o++]; t.zz = p[o++]; t.dx = p[o++]; t.dy = p[o++]; t.dz = p[o++];
    const double** d1[12] = {&t.ax1, &t.bx1, &t.cx1, &t.dx1, &t.ay1, &t.by1, &t.cy1, &t.dy1, &t.az1, &t.bz1, &t.cz1, &t.dz1};
    const double** d2[12] = {&t.ax2, &t.bx2, &t.cx2, &t.dx2, &t.ay2, &t.by2, &t.cy2, &t.dy2, &t.az2, &t.bz2, &t.cz2, &t.dz2};
    for (auto* q : d1) *q = p[o++];
    for (auto* q : d2) *q = p[o++];
    t.axp = p[o++]; t.bxp = p[o++]; t.cxp = p[o++];
    t.hx = p[o++]; t.hy = p[o++]; t.hz = p[o++]; t.rx = p[o++]; t.ry = p[o++]; t.rz = p[o++];
}

// r of every physical node, zero elsewhere (initia, T:771-776; rr0 and rr1 alike, the centre of
// rr1 at x = 0.0); tab: the tables of make_tables
inline std::vector<double> make_radius(const Dims& d, const std::vector<std::vector<double>>& tab) {
    const std::vector<double>&xx = tab[0], &yy = tab[1], &zz = tab[2];
    std::vector<double> r(d.n, 0.);
    for (int jz = 3; jz <= d.mz + 2; ++jz)
        for (int jy = 1; jy <= d.my; ++jy)
            for (int jx = 3; jx <= d.mx + 2; ++jx)
                r[d.at(jx, jy, jz)] = std::sqrt(xx[jx] * xx[jx] + yy[jy] * yy[jy] + zz[jz] * zz[jz]);
    return r;
}

// Fields of one context, carved from consecutive blocks: take(k) returns k fields
template <class Take>
inline void carve(Arr& a, Take take) {
    a.x = take(8); a.xm = take(8); a.xfold = take(8); a.xdif = take(8);
    a.cur = take(3); a.efld = take(3); a.xdh = take(3); a.xresd = take(3);
    a.w = take(1); a.fs = take(1); a.gs = take(1); a.hs = take(1); a.u = take(1); a.v = take(1);
    a.rhoi = take(1); a.bxi = take(1); a.byi = take(1); a.bzi = take(1); a.pri = take(1);
    a.rr0 = take(1); a.rr1 = take(1);
}
constexpr int NFIELDS = 4 * 8 + 4 * 3 + 6 + 7;   // fields carve takes

}  // namespace walls
}  // namespace dasha
