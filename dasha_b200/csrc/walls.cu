// walls.cu -- the engine of the reference's own bounded configuration (walls_core.cuh): a
// context created with periodic = {0, 0, 0}.  FP64, one thread per node for every loop of the
// reference's routines, on the reference's padded local layout.  Built with -fmad=false: the
// reference's expressions are rounded as written (no contraction to FMA), so the results follow
// the reference's own arithmetic to the rounding of the transcendental functions.
#include "dasha_capi.h"
#include "engine.cuh"
#include "walls_core.cuh"

#include <cstring>
#include <vector>

namespace dasha {

namespace {

using walls::Box;

// one thread per node of the box: x and y of a plane flattened (rows of 41 or 129 nodes would leave
// a third to a half of the threads of row-wise blocks idle), z in blockIdx.y.  Bound by the latency of
// each thread's loads: eight blocks an SM (64 registers a thread) measured 4.50 ms a 129x72x101 step, five or six
// (up to 96 registers, the compiler's choice) 4.67.
template <class F>
__global__ void __launch_bounds__(128, 8) k_walls(const __grid_constant__ Box b, const __grid_constant__ F f) {
    wait_for_stream();
    const unsigned nx = (unsigned)(b.x1 - b.x0 + 1), i = blockIdx.x * 128u + threadIdx.x, jy = i / nx;
    if (jy > (unsigned)(b.y1 - b.y0)) return;
    f(b.x0 + (int)(i - jy * nx), b.y0 + (int)jy, b.z0 + (int)blockIdx.y);
}
struct GpuExec {
    cudaStream_t st;
    static bool empty(const Box& b) { return b.x1 < b.x0 || b.y1 < b.y0 || b.z1 < b.z0; }
    static dim3 grid(const Box& b) {
        const long plane = (long)(b.x1 - b.x0 + 1) * (b.y1 - b.y0 + 1);
        return dim3((unsigned)((plane + 127) / 128), (unsigned)(b.z1 - b.z0 + 1));
    }
    template <class F>
    void run(Box b, F f) {
        if (!empty(b)) launch_overlapped(st, true, k_walls<F>, grid(b), 128, 0, b, f);
    }
    // the minimum of positive doubles through their bit patterns (ordered as unsigned integers)
    __host__ __device__ static void atomic_min_bits(unsigned long long* p, double v) {
#ifdef __CUDA_ARCH__
        // one atomic per warp, and only if it lowers the minimum so far: an atomic per node on one
        // address took 594 us of a 129x72x101 setdt
        const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
        const unsigned on = __activemask(), hi = (unsigned)(bits >> 32), hm = __reduce_min_sync(on, hi);
        const unsigned lm = __reduce_min_sync(on, hi == hm ? (unsigned)bits : 0xffffffffu);
        const unsigned long long least = (unsigned long long)hm << 32 | lm;
        if ((threadIdx.x & 31) == (unsigned)__ffs(on) - 1 && least < *(volatile unsigned long long*)p) atomicMin(p, least);
#else
        (void)p; (void)v;
#endif
    }
};

class WallEngine : public EngineBase {
public:
    GpuExec ex{};
    walls::Dims d{};
    walls::Par par{};
    walls::Arr a{};
    walls::Tables t{};
    void* pool = nullptr;
    double* tab = nullptr;
    cudaStream_t st = nullptr;
    long n = 0;
    bool eq_set = false;

    // no kernel here waits on a ring: stepon enqueues, and setdt waits for its own copy
    bool own_wait_status() const override { return true; }

    ~WallEngine() override {
        if (pool) cudaFree(pool);
        if (tab) cudaFree(tab);
        for (int b = 0; b < 2; ++b) {
            if (pin[b] && small_buf.empty()) cudaFreeHost(pin[b]);
            if (pev[b]) cudaEventDestroy(pev[b]);
        }
    }
    walls::Core<GpuExec> core() { return walls::Core<GpuExec>{ex, d, t, par, a}; }

    Status init(int mx, int my, int mz, const dasha_params_c& p, cudaStream_t st_, const double* xc, const double* yc,
                const double* zc) {
        st = st_;
        ex.st = st_;
        d = walls::make_dims(mx, my, mz);
        n = d.n;
        par.gamma = p.gamma; par.eta = p.eta; par.mu = p.viscos ? p.mu : 0.; par.drho = p.diffu ? p.drho : 0.;
        par.dp = p.diffu ? p.dp : 0.; par.cfl = p.cfl; par.rcr = p.rcr; par.chall = p.di;
        par.hall = p.hall; par.viscos = p.viscos; par.diffu = p.diffu; par.uyzlimiter = p.uyzlimiter;
        DASHA_CK(cudaMalloc(&pool, sizeof(double) * n * walls::NFIELDS + 256));
        DASHA_CK(cudaMemsetAsync(pool, 0, sizeof(double) * n * walls::NFIELDS + 256, st));
        DASHA_CK(cudaStreamSynchronize(st));          // the stream does not order with the copies below
        double* q = static_cast<double*>(pool);
        walls::carve(a, [&](int k) { double* r = q; q += (size_t)k * n; return r; });
        a.dtbits = reinterpret_cast<unsigned long long*>(q);
        // the 1-D tables, concatenated in one device buffer
        const std::vector<std::vector<double>> tabs = walls::make_tables(d, xc, yc, zc);
        std::vector<double> ht;
        std::vector<size_t> off;
        for (const auto& v : tabs) { off.push_back(ht.size()); ht.insert(ht.end(), v.begin(), v.end()); }
        DASHA_CK(cudaMalloc(&tab, sizeof(double) * ht.size()));
        DASHA_CK(cudaMemcpy(tab, ht.data(), sizeof(double) * ht.size(), cudaMemcpyHostToDevice));
        const double* tp[walls::NTAB];
        for (int k = 0; k < walls::NTAB; ++k) tp[k] = tab + off[k];
        walls::bind_tables(t, tp);
        {
            const std::vector<double> r = walls::make_radius(d, tabs);
            DASHA_CK(cudaMemcpy(a.rr0, r.data(), sizeof(double) * n, cudaMemcpyHostToDevice));
            DASHA_CK(cudaMemcpy(a.rr1, r.data(), sizeof(double) * n, cudaMemcpyHostToDevice));
        }
        DASHA_CK(cudaStreamSynchronize(st));
        return Status::ok();
    }

    // Physical nodes of a host array in the reference's layout (leading dimensions ld1, ld2, node
    // (i+2) + ld1 (j + ld2 ((k+2) + (mz+4) m))) to / from a padded device array.  The rows move packed, in
    // chunks through two pinned buffers (the host threads' gather or scatter of one chunk runs beside the DMA of the
    // other) and a device array that is free meanwhile, which one kernel unpacks or packs: a copy of
    // the padded arrays by one host thread and pageable memory took 17 ms each way at 129x72x101, this 5 and 6 ms.
    // Eight fields of less than 4 MB go in one piece through pageable memory: to pin the buffers would take longer
    // (20 ms more to set up a 41x25x33 context) than their transfers ever give back.
    double* pin[2] = {nullptr, nullptr};
    cudaEvent_t pev[2] = {nullptr, nullptr};
    std::vector<double> small_buf;
    static constexpr size_t PIN = size_t(8) << 20, SMALL = size_t(4) << 20;
    // rows of one pinned buffer: two of them hold an 8-field array of up to 16 MB (to pin memory takes about 1 ms a MB)
    long chunk_rows() const {
        const long most = std::max(1L, (long)(PIN / sizeof(double)) / d.mx);
        return small_buf.empty() ? std::min(most, 4L * d.my * d.mz) : most;
    }
    Status pins() {
        if (pev[1]) return Status::ok();
        const size_t all = 8 * sizeof(double) * (size_t)d.mx * d.my * d.mz;
        if (all < SMALL) {
            small_buf.resize(all / sizeof(double));
            pin[0] = pin[1] = small_buf.data();
        }
        for (int b = 0; b < 2; ++b) {
            if (!pin[b]) DASHA_CK(cudaMallocHost(&pin[b], sizeof(double) * (size_t)chunk_rows() * d.mx));
            if (!pev[b]) DASHA_CK(cudaEventCreateWithFlags(&pev[b], cudaEventDisableTiming));
        }
        return Status::ok();
    }
    // the rows [0, n) of a chunk, by the calling thread alone in a transfer of at most `alone` bytes, by the host threads above.
    // To wake the threads takes some 20 us, and rows on their way up leave the cache of the thread that the caller
    // filled them on, from which the copy to the GPU then reads slower.  Median ms a call, threads / alone (the padded copy
    // before), set_state: 10x10x10 0.103 / 0.062 (0.043), 41x25x33 (2.2 MB) 0.55 / 0.30 (0.40), 49x30x40 0.84 / 0.50 (0.66),
    // 74x45x59 (12.6 MB) 1.6-2.0 / 0.88-1.0 (2.0), 98x60x79 (30 MB) 2.6-3.1 / 2.0-2.2 (5.0), 115x70x92 (47 MB) 3.8 / 3.2 (10),
    // 200x120x150 (230 MB) 17.6 / 17.5 (71); get_state: 10x10x10 0.077 / 0.048 (0.055), 41x25x33 0.39-0.41 / 0.36-0.42 (0.41),
    // 49x30x40 0.57-0.63 / 0.58-0.65 (0.66), 55x34x45 (5.4 MB) 0.74-0.98 / 0.50-0.59 (0.9), 66x40x53 (9 MB) 1.0-1.6 / 0.8-1.0 (1.4),
    // 74x45x59 0.98-1.7 / 0.95-1.2 (1.9), 98x60x79 1.1-3.0 / 2.2-2.7 (4.4), 200x120x150 15.3 / 25.4 (45).
    static constexpr size_t ALONE_UP = size_t(32) << 20, ALONE_DOWN = size_t(10) << 20;
    template <class F>
    void spread(long rows, size_t alone, long n, const F& f) const {
        if (sizeof(double) * (size_t)rows * d.mx <= alone) f(0L, n);
        else HostPool::get().run(n, f);
    }
    // host address of row r = j + my (k + mz m) of the caller's array
    long row_at(long r, long ld1, long ld2) const {
        const long j = r % d.my, q = r / d.my, k = q % d.mz, m = q / d.mz;
        return 2 + ld1 * (j + ld2 * ((k + 2) + (long)(d.mz + 4) * m));
    }
    Status upload(const double* src, long ld1, long ld2, int nf, double* dst, double* stage) {
        Status s = pins();
        if (s.code) return s;
        const long rows = (long)nf * d.mz * d.my, step = chunk_rows();
        int q = 0;
        for (long r0 = 0; r0 < rows; r0 += step, ++q) {
            const long r1 = std::min(rows, r0 + step);
            double* h = pin[q & 1];
            DASHA_CK(cudaEventSynchronize(pev[q & 1]));
            spread(rows, ALONE_UP, r1 - r0, [&](long a0, long a1) {
                for (long r = a0; r < a1; ++r) std::memcpy(h + r * d.mx, src + row_at(r0 + r, ld1, ld2), sizeof(double) * d.mx);
            });
            DASHA_CK(cudaMemcpyAsync(stage + r0 * d.mx, h, sizeof(double) * (size_t)(r1 - r0) * d.mx, cudaMemcpyHostToDevice, st));
            DASHA_CK(cudaEventRecord(pev[q & 1], st));
        }
        move(nf, [=] __device__(double* packed, double* padded) { *padded = *packed; }, stage, dst);
        DASHA_CK(cudaGetLastError());
        DASHA_CK(cudaStreamSynchronize(st));
        return Status::ok();
    }
    Status download(double* dst, long ld1, long ld2, int nf, double* src, double* stage) {
        Status s = pins();
        if (s.code) return s;
        move(nf, [=] __device__(double* packed, double* padded) { *packed = *padded; }, stage, src);
        DASHA_CK(cudaGetLastError());
        const long rows = (long)nf * d.mz * d.my, step = chunk_rows();
        auto copy = [&](long q) {
            const long r0 = q * step, r1 = std::min(rows, r0 + step);
            cudaError_t e = cudaMemcpyAsync(pin[q & 1], stage + r0 * d.mx, sizeof(double) * (size_t)(r1 - r0) * d.mx, cudaMemcpyDeviceToHost, st);
            return e ? e : cudaEventRecord(pev[q & 1], st);
        };
        const long chunks = (rows + step - 1) / step;
        DASHA_CK(copy(0));
        for (long q = 0; q < chunks; ++q) {
            if (q + 1 < chunks) DASHA_CK(copy(q + 1));
            DASHA_CK(cudaEventSynchronize(pev[q & 1]));
            const long r0 = q * step, r1 = std::min(rows, r0 + step);
            const double* h = pin[q & 1];
            spread(rows, ALONE_DOWN, r1 - r0, [&](long a0, long a1) {
                for (long r = a0; r < a1; ++r) std::memcpy(dst + row_at(r0 + r, ld1, ld2), h + r * d.mx, sizeof(double) * d.mx);
            });
        }
        return Status::ok();
    }
    // f(packed, padded) at every physical node of nf fields
    template <class F>
    void move(int nf, F f, double* packed, double* padded) {
        const walls::Dims dd = d;
        const long nn = n;
        ex.run(core().physical(), [=] __device__(int jx, int jy, int jz) {
            const long i = (jx - 3) + (long)dd.mx * ((jy - 1) + (long)dd.my * (jz - 3)), np = (long)dd.mx * dd.my * dd.mz;
            const long c = dd.at(jx, jy, jz);
            for (int m = 0; m < nf; ++m) f(packed + m * np + i, padded + m * nn + c);
        });
    }

    // the equilibrium, then xresd as initia computes it (T:805-834): the state set to the
    // equilibrium, right(0, 1e-9, 1) with eta = 0 (foreta runs after it), xresd = the momentum rates
    Status equilibrium_from(const double* src, long ld1, long ld2) {
        // rho0 bx0 by0 bz0 p0 by way of xm, zero off the physical nodes: the driver reads rhoi beyond the last
        // plane where mz - 1 >= 3 my (RowRule::driven_state), and rhs() packs its rates in xm
        DASHA_CK(cudaMemsetAsync(a.xm, 0, sizeof(double) * 5 * n, st));
        Status s = upload(src, ld1, ld2, 5, a.xm, a.xdif);
        if (s.code) return s;
        double* eq[5] = {a.rhoi, a.bxi, a.byi, a.bzi, a.pri};
        for (int q = 0; q < 5; ++q) DASHA_CK(cudaMemcpyAsync(eq[q], a.xm + q * n, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        const int from[8] = {0, -1, -1, -1, 1, 2, 3, 4};
        for (int m = 0; m < 8; ++m) {
            if (from[m] < 0) DASHA_CK(cudaMemsetAsync(a.x + m * n, 0, sizeof(double) * n, st));
            else DASHA_CK(cudaMemcpyAsync(a.x + m * n, eq[from[m]], sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        }
        DASHA_CK(cudaMemcpyAsync(a.xfold, a.x, sizeof(double) * 8 * n, cudaMemcpyDeviceToDevice, st));
        DASHA_CK(cudaMemsetAsync(a.xresd, 0, sizeof(double) * 3 * n, st));
        const double eta = par.eta;
        par.eta = 0.;
        core().right(0., 1.e-9, 1);
        par.eta = eta;
        DASHA_CK(cudaMemcpyAsync(a.xresd, a.xdif + n, sizeof(double) * 3 * n, cudaMemcpyDeviceToDevice, st));
        DASHA_CK(cudaGetLastError());
        DASHA_CK(cudaStreamSynchronize(st));
        eq_set = true;
        return Status::ok();
    }
    Status set_equilibrium(const double* rho0, const double* b0, const double* p0, const double*) override {
        // z-profiles broadcast over x and y
        std::vector<double> e(5 * (size_t)n, 0.);
        const double* prof[5] = {rho0, b0, b0 + d.mz, b0 + 2 * d.mz, p0};
        for (int q = 0; q < 5; ++q)
            for (int k = 0; k < d.mz; ++k)
                for (int j = 1; j <= d.my; ++j)
                    for (int i = 3; i <= d.mx + 2; ++i) e[q * n + d.at(i, j, k + 3)] = prof[q][k];
        return equilibrium_from(e.data(), d.mxpr, d.my);
    }
    Status set_equilibrium_3d(const double* eq, long ld1, long ld2) override {
        return equilibrium_from(eq, ld1, ld2);
    }
    Status set_j0(const double*) override { return Status::err(DASHA_E_UNSUPPORTED, "J0 is a periodic-context option"); }
    Status set_state(const double* x, long ld1, long ld2) override {
        return upload(x, ld1, ld2, 8, a.x, a.xdif);
    }
    Status get_state(double* x, long ld1, long ld2) override {
        return download(x, ld1, ld2, 8, a.x, a.xdif);
    }
    Status setdt(double* dt, int* blowup) override {
        const double hundred = 100.;
        unsigned long long bits;
        std::memcpy(&bits, &hundred, sizeof(bits));
        DASHA_CK(cudaMemcpyAsync(a.dtbits, &bits, sizeof(bits), cudaMemcpyHostToDevice, st));
        core().setdt_launch();
        DASHA_CK(cudaGetLastError());
        DASHA_CK(cudaMemcpyAsync(&bits, a.dtbits, sizeof(bits), cudaMemcpyDeviceToHost, st));
        DASHA_CK(cudaStreamSynchronize(st));
        std::memcpy(dt, &bits, sizeof(double));
        *blowup = 0;
        return Status::ok();
    }
    Status stepon(double time, double dt, int) override {
        NvtxRange range("stepon (bounded)");
        core().stepon(time, dt);
        DASHA_CK(cudaGetLastError());
        return Status::ok();
    }
    Status current(double* cur, long ld1, long ld2) override {
        core().current();
        DASHA_CK(cudaGetLastError());
        return download(cur, ld1, ld2, 3, a.cur, a.xdif);
    }
    // right(t, 1e-9, 1) with xfold = x, as initia calls it; the state is restored afterwards
    // (the inflow driver writes the x-min rows of x)
    Status rhs(double tt, double* xdif, long ld1, long ld2) override {
        DASHA_CK(cudaMemcpyAsync(a.xfold, a.x, sizeof(double) * 8 * n, cudaMemcpyDeviceToDevice, st));
        core().right(tt, 1.e-9, 1);
        DASHA_CK(cudaMemcpyAsync(a.x, a.xfold, sizeof(double) * 8 * n, cudaMemcpyDeviceToDevice, st));
        DASHA_CK(cudaGetLastError());
        return download(xdif, ld1, ld2, 8, a.xdif, a.xm);
    }
    static Status no(const char* what) {
        return Status::err(DASHA_E_UNSUPPORTED, std::string(what) + " is not available on a bounded (periodic 0,0,0) context");
    }
    Status state_in(const ChunkIn&) override { return no("streamed state transfer"); }
    Status state_out(const ChunkOut&) override { return no("streamed state transfer"); }
    Status current_out(const ChunkOut&) override { return no("streamed current transfer"); }
    int raw_fields() const override { return 8; }
    size_t raw_elem() const override { return sizeof(double); }
    Status raw_out(const std::function<bool(const void*, size_t)>&) override { return no("the exact-resume record"); }
    Status raw_in(const std::function<bool(void*, size_t)>&) override { return no("the exact-resume record"); }
    Status midplane(double*) override { return no("dasha_midplane"); }
    Status diagnostics(double*) override { return no("dasha_diagnostics"); }
    Status adjoint_flux_grad(int, const double*, int, double*, double*) override { return no("the adjoint"); }
    Status adjoint_rhs(const double*, double*, long, long) override { return no("the adjoint"); }
};

}  // namespace

EngineBase* make_engine_walls(int mx, int my, int mz, const dasha_params_c& p, cudaStream_t st, const double* x,
                              const double* y, const double* z, Status& s) {
    WallEngine* e = new WallEngine();
    s = e->init(mx, my, mz, p, st, x, y, z);
    if (s.code) { delete e; return nullptr; }
    return e;
}

}  // namespace dasha
