// noalloc.cu -- dasha_current_noalloc: the smoothed current density J = S^4(curl(B - B0))
// computed without allocating any device memory.
//
// Who needs this: callers whose device memory is not theirs to allocate -- a host code that
// hands the GPU over to a memory manager owning every byte up front (a fixed pool sized at
// start-up, a cap enforced by a scheduler), code running where the CUDA allocator may not be
// called (inside a no-allocation phase of a larger application or while another component
// holds the allocator lock), and diagnostics that must not perturb a tight memory budget.
// dasha_current needs a context, whose buffers come from cudaMalloc; this entry point takes
// the caller's device input and output arrays and does its ping-pong passes in a fixed
// scratch array that is part of the library image.
//
// The scratch is a file-scope __device__ array of NOALLOC_SCRATCH_DOUBLES doubles (about 26 MB):
// every GPU that loads this library holds it until the process exits.  It holds one
// 3-field ping-pong buffer of at most NOALLOC_MAX_CELLS nodes and the 1-D stencil tables.
// All calls share it and it keeps the last call's contents; every byte a call reads is
// written earlier in the same call, so nothing has to be cleared.  Calls that overlap on the
// GPU (two streams, two host threads) race on it: serialise them.
#include "dasha_capi.h"
#include "mhd_kernels.cuh"
#include "coef.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

using namespace dasha;

namespace {
constexpr long kMaxCells = DASHA_NOALLOC_MAX_CELLS;
constexpr int kAxisMax = DASHA_NOALLOC_MAX_AXIS;
constexpr int kTabPerAxis = 7;   // a1 b1 c1 d1 (first derivative), wp wm (difc), coordinate
constexpr long kTabDoubles = 3L * kTabPerAxis * kAxisMax;
constexpr long kScratchDoubles = 3 * kMaxCells + kTabDoubles;
static_assert(kScratchDoubles == DASHA_NOALLOC_SCRATCH_DOUBLES, "scratch size mismatch with dasha_capi.h");
constexpr int kMaxDevices = 64;

std::mutex g_mu;
double* g_dev_ptr[kMaxDevices] = {};   // device address of the scratch, per device ordinal
double g_host_tab[kTabDoubles];        // host staging of the tables (static: no heap use)
}  // namespace

static __device__ __align__(256) double g_noalloc_scratch[kScratchDoubles];

// Both kernels: a thread per node of the interior planes (blockIdx.y), x and y flattened so that a warp is full
// whatever mx is; the threads of planes 2 and mz-3 also write the wall rows beside them.  Bound by
// the latency of a thread's loads; eight blocks an SM.  Measured on B200 at 128x64x100: a pass 20.4 -> 15.7 us against a thread
// for every node of rows of 128 with the coefficient by tanh, the curl 18.6 -> 15.5 us.
struct NoallocNode {
    int i, j, k;
    unsigned q;                                       // offset in the plane
    long c;
    bool on;
    __device__ __forceinline__ NoallocNode(const Geo<double>& g) {
        q = blockIdx.x * 128u + threadIdx.x;
        on = q < (unsigned)(g.mx * g.my);
        j = (int)(q / (unsigned)g.mx);
        i = (int)(q - (unsigned)j * (unsigned)g.mx);
        k = 2 + (int)blockIdx.y;
        c = q + (long)k * g.sz;
    }
    __device__ __forceinline__ void store(const Geo<double>& g, double* f, double v) const {
        f[c] = v;
        if (k == 2) { f[q + g.sz] = 0.5 * v; f[q] = 0.0; }
        if (k == g.mz - 3) { f[c + g.sz] = 0.5 * v; f[c + 2 * g.sz] = 0.0; }
    }
};

// J1 = curl(B - B0) with the wall rows (current t3dsdsc.f:2468-2491, bndryc)
__global__ void __launch_bounds__(128, 8) k_noalloc_curl(const __grid_constant__ Geo<double> g, F3<double> b, F3<double> o) {
    wait_for_stream();
    const NoallocNode t(g);
    if (!t.on) return;
    const Nbr<double> n(g, t.i, t.j, t.k);
    // all before the first store, which might alias the loads for all that the compiler knows
    const double j1 = n.Dy(g, b.f[2]) - n.Dz(g, b.f[1]);
    const double j2 = n.Dz(g, b.f[0]) - n.Dx(g, b.f[2]);
    const double j3 = n.Dx(g, b.f[1]) - n.Dy(g, b.f[0]);
    t.store(g, o.f[0], j1);
    t.store(g, o.f[1], j2);
    t.store(g, o.f[2], j3);
}

// One smoothing pass with the radial coefficient of avrgc (t3dsdsc.f:5981-5992) evaluated
// from the node coordinates, wall rows re-applied (bndryc t3dsdsc.f:2614-2642).  1/32 + 3/64 (1 + tanh u) =
// 1/32 + (3/32) / (1 + exp(-2u)), u = (r-3)/3: half the operations of tanh.
__global__ void __launch_bounds__(128, 8) k_noalloc_smooth(const __grid_constant__ Geo<double> g, F3<double> in, F3<double> out) {
    wait_for_stream();
    const NoallocNode t(g);
    if (!t.on) return;
    const int im = wrapi(t.i - 1, g.mx) - t.i, ip = wrapi(t.i + 1, g.mx) - t.i;
    const long jm = (long)(wrapi(t.j - 1, g.my) - t.j) * g.sy, jp = (long)(wrapi(t.j + 1, g.my) - t.j) * g.sy;
    double f0[3], fx[3][2], fy[3][2], fz[3][2];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double* f = in.f[q] + t.c;
        f0[q] = f[0];
        fx[q][0] = f[im]; fx[q][1] = f[ip];
        fy[q][0] = f[jm]; fy[q][1] = f[jp];
        fz[q][0] = f[-g.sz]; fz[q][1] = f[g.sz];
    }
    const double x = g.xc[t.i], y = g.yc[t.j], z = g.zc[t.k];
    const double coef = 1.0 / 32.0 + (3.0 / 32.0) / (1.0 + exp((6.0 - 2.0 * sqrt(x * x + y * y + z * z)) / 3.0));
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double d = (fx[q][1] - f0[q]) * g.wpx[t.i] - (f0[q] - fx[q][0]) * g.wmx[t.i] + (fy[q][1] - f0[q]) * g.wpy[t.j] -
                         (f0[q] - fy[q][0]) * g.wmy[t.j] + (fz[q][1] - f0[q]) * g.wpz[t.k] - (f0[q] - fz[q][0]) * g.wmz[t.k];
        t.store(g, out.f[q], f0[q] + coef * d);
    }
}

// The 1-D tables of axis blockIdx.y from the coordinates x | y | z (`coord`): the first-derivative weights
// as the derivatives at x0 of the Lagrange polynomials through the five nodes, and the difc weights.
__global__ void k_noalloc_tables(double* dtab, const double* coord, int mx, int my, int mz) {
    wait_for_stream();
    const int d = blockIdx.y, n = d == 0 ? mx : (d == 1 ? my : mz), i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* t = dtab + (long)d * kTabPerAxis * kAxisMax;
    const double* c = coord + (d == 0 ? 0 : (d == 1 ? mx : mx + my));
    const bool periodic = d < 2;
    const double L = c[n - 1] - c[0] + (c[1] - c[0]);
    auto at = [&](int q) {
        if (!periodic) return c[q];
        const int w = q < 0 ? -1 : (q >= n ? 1 : 0);
        return c[q - w * n] + w * L;
    };
    const double x0 = c[i];
    double a[4] = {0, 0, 0, 0}, wp = 0.0, wm = 0.0;
    if (periodic || (i >= 2 && i <= n - 3)) {
        const double h1 = at(i + 1) - x0, g1 = x0 - at(i - 1), h2 = at(i + 2) - x0, g2 = x0 - at(i - 2);
        a[0] = g1 * h2 * g2 / (h1 * (h1 + g1) * (h2 - h1) * (h1 + g2));
        a[1] = h1 * h2 * g2 / (g1 * (g1 + h1) * (g1 + h2) * (g2 - g1));
        a[2] = -h1 * g1 * g2 / (h2 * (h2 - h1) * (h2 + g1) * (h2 + g2));
        a[3] = -h1 * g1 * h2 / (g2 * (g2 + h1) * (g2 - g1) * (g2 + h2));
    }
    if (periodic || (i >= 1 && i <= n - 2)) {
        const double xm = at(i - 1), xp = at(i + 1);
        wp = 2.0 * (xp - x0) / (xp - xm);
        wm = 2.0 * (x0 - xm) / (xp - xm);
    }
    for (int q = 0; q < 4; ++q) t[(long)q * kAxisMax + i] = a[q];
    t[4L * kAxisMax + i] = wp;
    t[5L * kAxisMax + i] = wm;
}

// Spacings of ordinary size and neighbours within a factor of 1000: the weights' products neither
// overflow nor cancel to nothing, and the 4x4 systems of coef.h have no zero pivot.
static bool ordinary_spacings(const double* c, int n, bool periodic) {
    double last = c[1] - c[0];
    if (periodic) last = c[n - 1] - c[n - 2];        // the wrap repeats c[1] - c[0] after it
    for (int i = periodic ? -1 : 0; i + 1 < n; ++i) {
        const double h = i < 0 ? c[1] - c[0] : c[i + 1] - c[i];
        if (!(h > 1e-60 && h < 1e60 && h < 1e3 * last && last < 1e3 * h)) return false;
        last = h;
    }
    return true;
}

// One-time set-up per device: the device address of the scratch array.  Host code must not
// use the symbol's name as an address (it is a host-side stand-in).
static int scratch_for_current_device(double** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return DASHA_E_CUDA;
    if (!g_dev_ptr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) return DASHA_E_CUDA;
        g_dev_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_dev_ptr[dev];
    return DASHA_OK;
}

// The 1-D tables into g_host_tab (host FP64), same construction as dasha_create
static int host_tables(const double* const coords[3], const int n[3]) {
    for (int d = 0; d < 3; ++d) {
        const double* c = coords[d];
        const bool periodic = d < 2;
        const double L = periodic ? c[n[d] - 1] - c[0] + (c[1] - c[0]) : 0.0;
        auto at = [&](int i) {
            if (!periodic) return c[i];
            int q = 0;
            while (i < 0) { i += n[d]; --q; }
            while (i >= n[d]) { i -= n[d]; ++q; }
            return c[i] + q * L;
        };
        double* t = g_host_tab + (long)d * kTabPerAxis * kAxisMax;
        for (int q = 0; q < kTabPerAxis; ++q)
            for (int i = 0; i < n[d]; ++i) t[(long)q * kAxisMax + i] = 0.0;
        for (int i = 0; i < n[d]; ++i) {
            if (periodic || (i >= 2 && i <= n[d] - 3)) {
                double x0 = at(i), w1[4];
                if (!stencil_weights(at(i + 1) - x0, x0 - at(i - 1), at(i + 2) - x0, x0 - at(i - 2), 1, w1))
                    return DASHA_E_INVALID;
                for (int q = 0; q < 4; ++q) t[(long)q * kAxisMax + i] = w1[q];
            }
            if (periodic || (i >= 1 && i <= n[d] - 2)) {
                double xm = at(i - 1), x0 = at(i), xp = at(i + 1);
                t[4L * kAxisMax + i] = 2.0 * (xp - x0) / (xp - xm);
                t[5L * kAxisMax + i] = 2.0 * (x0 - xm) / (xp - xm);
            }
            t[6L * kAxisMax + i] = c[i];
        }
    }
    return DASHA_OK;
}

extern "C" int dasha_current_noalloc(const dasha_grid_c* grid, const double* db_dev, double* cur_dev, void* stream) {
    if (!grid || !grid->x || !grid->y || !grid->z || !db_dev || !cur_dev) return DASHA_E_INVALID;
    const int mx = grid->mx, my = grid->my, mz = grid->mz;
    if (mx < 5 || my < 5 || mz < 7) return DASHA_E_INVALID;
    if (!(grid->periodic[0] == 1 && grid->periodic[1] == 1 && grid->periodic[2] == 0)) return DASHA_E_UNSUPPORTED;
    if ((long)mx * my * mz > kMaxCells || mx > kAxisMax || my > kAxisMax || mz > kAxisMax) return DASHA_E_NOSCRATCH;
    {   // the curl reads neighbours of B while it writes J: the two ranges must be disjoint
        const uintptr_t nb = 3u * sizeof(double) * (uintptr_t)mx * my * mz;
        const uintptr_t a = reinterpret_cast<uintptr_t>(db_dev), b = reinterpret_cast<uintptr_t>(cur_dev);
        if (a < b + nb && b < a + nb) return DASHA_E_INVALID;
    }
    const double* coords[3] = {grid->x, grid->y, grid->z};
    const int n[3] = {mx, my, mz};
    for (int d = 0; d < 3; ++d)
        for (int i = 0; i + 1 < n[d]; ++i)
            if (!(coords[d][i + 1] > coords[d][i])) return DASHA_E_INVALID;

    std::lock_guard<std::mutex> lock(g_mu);
    double* scratch = nullptr;
    if (int rc = scratch_for_current_device(&scratch)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    double* dtab = scratch + 3 * kMaxCells;
    // the coordinates: entry 6 of each axis' table, or all three in that of x
    const double* xyz[3];
    for (int d = 0; d < 3; ++d) xyz[d] = dtab + ((long)d * kTabPerAxis + 6) * kAxisMax;
    bool ordinary = mx + my + mz <= kAxisMax;
    for (int d = 0; d < 3; ++d) ordinary = ordinary && ordinary_spacings(coords[d], n[d], d < 2);
    if (ordinary) {
        // the coordinates go over and a kernel makes the tables: 16 powers and a 4x4 system a node on the host
        // took 100 us of a 128x64x100 call, and 688 KB of tables to copy
        double* h = g_host_tab + 6L * kAxisMax;
        int at = 0;
        for (int d = 0; d < 3; ++d) {
            std::memcpy(h + at, coords[d], sizeof(double) * n[d]);
            xyz[d] = dtab + 6L * kAxisMax + at;
            at += n[d];
        }
        if (cudaMemcpyAsync(dtab + 6L * kAxisMax, h, sizeof(double) * at, cudaMemcpyHostToDevice, st) != cudaSuccess)
            return DASHA_E_CUDA;
        const int most = std::max(mx, std::max(my, mz));
        k_noalloc_tables<<<dim3((unsigned)((most + 127) / 128), 3), 128, 0, st>>>(dtab, xyz[0], mx, my, mz);
    } else {
        if (int rc = host_tables(coords, n)) return rc;
        if (cudaMemcpyAsync(dtab, g_host_tab, sizeof(double) * kTabDoubles, cudaMemcpyHostToDevice, st) != cudaSuccess)
            return DASHA_E_CUDA;
    }

    Geo<double> g{};
    g.mx = mx; g.my = my; g.mz = mz; g.sy = mx; g.sz = (long)mx * my;
    const double* T[3];
    for (int d = 0; d < 3; ++d) T[d] = dtab + (long)d * kTabPerAxis * kAxisMax;
    g.a1x = T[0]; g.b1x = T[0] + kAxisMax; g.c1x = T[0] + 2 * kAxisMax; g.d1x = T[0] + 3 * kAxisMax;
    g.a1y = T[1]; g.b1y = T[1] + kAxisMax; g.c1y = T[1] + 2 * kAxisMax; g.d1y = T[1] + 3 * kAxisMax;
    g.a1z = T[2]; g.b1z = T[2] + kAxisMax; g.c1z = T[2] + 2 * kAxisMax; g.d1z = T[2] + 3 * kAxisMax;
    g.wpx = T[0] + 4 * kAxisMax; g.wmx = T[0] + 5 * kAxisMax;
    g.wpy = T[1] + 4 * kAxisMax; g.wmy = T[1] + 5 * kAxisMax;
    g.wpz = T[2] + 4 * kAxisMax; g.wmz = T[2] + 5 * kAxisMax;
    g.xc = xyz[0]; g.yc = xyz[1]; g.zc = xyz[2];

    const long N = (long)mx * my * mz;
    F3<double> b, cur, tmp;
    for (int q = 0; q < 3; ++q) {
        b.f[q] = const_cast<double*>(db_dev) + q * N;
        cur.f[q] = cur_dev + q * N;
        tmp.f[q] = scratch + q * N;
    }
    const dim3 grd((unsigned)((mx * my + 127) / 128), (unsigned)(mz - 4));
    // J1 = curl(B - B0) with the wall rows, then 4 passes cur -> scratch -> cur -> scratch -> cur
    launch_overlapped(st, true, k_noalloc_curl, grd, 128, 0, g, b, cur);
    for (int pass = 0; pass < 4; ++pass) {
        if (pass % 2 == 0) launch_overlapped(st, true, k_noalloc_smooth, grd, 128, 0, g, cur, tmp);
        else launch_overlapped(st, true, k_noalloc_smooth, grd, 128, 0, g, tmp, cur);
    }
    return cudaGetLastError() == cudaSuccess ? DASHA_OK : DASHA_E_CUDA;
}
