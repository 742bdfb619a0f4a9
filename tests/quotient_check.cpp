// Bit-for-bit check of the quotients by fused multiply-adds (dasha_b200/csrc/quotient.h) against the division, for
// g++ (the host's fma) and for nvcc -x cu (the device's): every case is a pair (dividend, divisor), and a
// result may differ from the division's only in a NaN's payload.  Prints the number of differences and the first few.
#include "quotient.h"

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

using namespace dasha;

template <class T>
struct Bits;
template <>
struct Bits<float> { using U = uint32_t; static constexpr int MANT = 23, EXP = 255; };
template <>
struct Bits<double> { using U = uint64_t; static constexpr int MANT = 52, EXP = 2047; };

template <class T>
static T make(bool neg, int e, uint64_t m) {
    using B = Bits<T>;
    const typename B::U u = ((typename B::U)neg << (8 * sizeof(T) - 1)) | ((typename B::U)e << B::MANT) |
                            ((typename B::U)m & (((typename B::U)1 << B::MANT) - 1));
    T v;
    std::memcpy(&v, &u, sizeof(v));
    return v;
}
static uint64_t g_seed = 88172645463325252ull;
static uint64_t rnd() { g_seed ^= g_seed << 13; g_seed ^= g_seed >> 7; g_seed ^= g_seed << 17; return g_seed; }

// dividends: all exponents with random mantissas, the ends of each binade, all patterns of the lowest magnitudes
template <class T>
static std::vector<T> dividends(long per_exponent) {
    using B = Bits<T>;
    std::vector<T> v;
    for (int e = 0; e <= B::EXP; ++e)
        for (int s = 0; s < 2; ++s) {
            for (uint64_t m : {0ull, 1ull, 2ull, 3ull, ~0ull, ~0ull - 1, 1ull << (B::MANT - 1)}) v.push_back(make<T>(s, e, m));
            for (long n = 0; n < per_exponent; ++n) v.push_back(make<T>(s, e, rnd()));
        }
    for (int s = 0; s < 2; ++s)
        for (uint64_t m = 0; m < 4096; ++m) v.push_back(make<T>(s, 0, m));
    return v;
}

struct Case3 { double a, b; };

#ifdef __CUDACC__
#define RUN(T, n, in, out, EXPR)                                                                        \
    {                                                                                                   \
        In* di;                                                                                         \
        T* dout;                                                                                        \
        cudaMalloc(&di, sizeof(In) * (n));                                                              \
        cudaMalloc(&dout, sizeof(T) * (n));                                                             \
        cudaMemcpy(di, (in).data(), sizeof(In) * (n), cudaMemcpyHostToDevice);                          \
        k_run<<<(unsigned)(((n) + 255) / 256), 256>>>((long)(n), di, dout);                             \
        cudaMemcpy((out).data(), dout, sizeof(T) * (n), cudaMemcpyDeviceToHost);                        \
        if (cudaGetLastError() != cudaSuccess) { std::printf("bad=-1\n"); std::exit(2); }               \
        cudaFree(di);                                                                                   \
        cudaFree(dout);                                                                                 \
    }
template <class T>
struct Over { T a, d; };
template <class T>
__global__ void k_run(long n, const Over<T>* in, T* out) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = over(in[i].a, in[i].d, T(1) / in[i].d);
}
__global__ void k_run(long n, const Case3* in, double* out) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = div_by_steps(in[i].a, in[i].b, 1. / in[i].b);
}
#else
#define RUN(T, n, in, out, EXPR) \
    for (long i = 0; i < (long)(n); ++i) { const In& c = (in)[i]; (out)[i] = EXPR; }
template <class T>
struct Over { T a, d; };
#endif

template <class T>
static bool same(T x, T y) { return std::memcmp(&x, &y, sizeof(T)) == 0 || (x != x && y != y); }

template <class T>
static long check_over(const char* name, long per_exponent) {
    using In = Over<T>;
    std::vector<In> in;
    for (T a : dividends<T>(per_exponent))
        for (T d : {T(3), T(6)}) in.push_back({a, d});
    std::vector<T> out(in.size());
    RUN(T, in.size(), in, out, (over(c.a, c.d, T(1) / c.d)));
    long bad = 0;
    for (size_t i = 0; i < in.size(); ++i) {
        const T want = in[i].a / in[i].d;
        if (!same(out[i], want) && ++bad <= 5)
            std::printf("%s %a / %a: %a, not %a\n", name, (double)in[i].a, (double)in[i].d, (double)out[i], (double)want);
    }
    return bad;
}

static long check_div_by(long per_exponent) {
    using In = Case3;
    std::vector<double> as = dividends<double>(per_exponent);
    std::vector<In> in;
    // divisors: every kind of exponent, both sides of the guards, mantissas all ones and all zeros
    const int eb[] = {0, 1, 2, 1023, 1022, 1024, 1000, 1046, 700, 1350, 1023 - 300, 1023 - 299, 1023 - 301, 1023 + 299, 1023 + 300,
                      1023 + 301, 2045, 2046, 2047};
    for (double a : as) {
        const int e = eb[rnd() % (sizeof(eb) / sizeof(eb[0]))];
        const uint64_t ms[] = {0ull, ~0ull, 1ull, rnd(), rnd(), rnd()};
        in.push_back({a, make<double>(rnd() & 1, e, ms[rnd() % 6])});
        in.push_back({a, make<double>(rnd() & 1, 1013 + (int)(rnd() % 20), rnd())});   // divisors of order one
    }
    // dividends next to a multiple of the divisor and next to the middle between two quotients
    for (long n = 0; n < 200000; ++n) {
        const double b = make<double>(0, 1013 + (int)(rnd() % 20), rnd()), q = make<double>(0, 1013 + (int)(rnd() % 20), rnd());
        const double half = 0.5 * (std::nextafter(q, 4.) - q), p = q * b, p2 = std::fma(half, b, p);
        for (double a : {p, std::nextafter(p, 0.), std::nextafter(p, 1e9), p2, std::nextafter(p2, 0.), std::nextafter(p2, 1e9)}) in.push_back({a, b});
    }
    std::vector<double> out(in.size());
    RUN(double, in.size(), in, out, (div_by_steps(c.a, c.b, 1. / c.b)));
    long bad = 0;
    for (size_t i = 0; i < in.size(); ++i) {
        const double want = in[i].a / in[i].b;
        if (!same(out[i], want) && ++bad <= 5) std::printf("div_by %a / %a: %a, not %a\n", in[i].a, in[i].b, out[i], want);
    }
    return bad;
}

int main() {
    const long f = check_over<float>("over<float>", 2000), d = check_over<double>("over<double>", 200), q = check_div_by(200);
    std::printf("over<float> bad=%ld over<double> bad=%ld div_by bad=%ld\n", f, d, q);
    return f || d || q ? 1 : 0;
}
