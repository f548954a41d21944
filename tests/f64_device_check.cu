// Largest errors of vp_f64.cuh's functions as the device computes them (its seeds are the hardware's approximations, which
// the host check replaces by roundings of the value) against the library's in long double: random arguments of many
// magnitudes, the tables' points and the halves between them, and both sides of every switch to the general functions.
// What the fast forms pass on is compared with CUDA's functions. Prints one line per function, in the units of the header.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "vp_f64.cuh"

typedef long double ld;
constexpr int NOUT = 7;  // rcp, rsqrt, sqrt, 1/sqrt with it, log, log<-1>, atan2(y, x)

__global__ void fast(int n, const double* x, const double* y, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* o = out + size_t(NOUT) * i;
    o[0] = f64::rcp(x[i]);
    o[1] = f64::rsqrt(x[i]);
    o[2] = f64::sqrt_inv(x[i], o[3]);
    o[4] = f64::log(x[i]);
    o[5] = f64::log<-1>(x[i]);
    o[6] = f64::atan2(y[i], x[i]);
}
__global__ void general(int n, const double* x, const double* y, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* o = out + size_t(NOUT) * i;
    o[0] = 1.0 / x[i];
    o[1] = rsqrt(x[i]);
    o[2] = sqrt(x[i]);
    o[3] = 1.0 / sqrt(x[i]);
    o[4] = log(x[i]);
    o[5] = log(0.5 * x[i]);
    o[6] = atan2(y[i], x[i]);
}

static bool run(bool lib, const std::vector<double>& x, const std::vector<double>& y, std::vector<double>& out) {
    const int n = int(x.size());
    double *dx = nullptr, *dy = nullptr, *d = nullptr;
    out.resize(size_t(NOUT) * n);
    bool ok = cudaMalloc(&dx, 8 * x.size()) == cudaSuccess && cudaMalloc(&dy, 8 * x.size()) == cudaSuccess &&
              cudaMalloc(&d, 8 * out.size()) == cudaSuccess &&
              cudaMemcpy(dx, x.data(), 8 * x.size(), cudaMemcpyHostToDevice) == cudaSuccess &&
              cudaMemcpy(dy, y.data(), 8 * x.size(), cudaMemcpyHostToDevice) == cudaSuccess;
    if (ok) {
        if (lib) general<<<(n + 255) / 256, 256>>>(n, dx, dy, d);
        else fast<<<(n + 255) / 256, 256>>>(n, dx, dy, d);
        ok = cudaGetLastError() == cudaSuccess &&
             cudaMemcpy(out.data(), d, 8 * out.size(), cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    cudaFree(dx);
    cudaFree(dy);
    cudaFree(d);
    return ok;
}

static double ulp(double x) {
    x = std::fabs(x);
    return std::nextafter(x, INFINITY) - x;
}

int main() {
    std::mt19937_64 rng(11);
    std::uniform_real_distribution<double> U(0, 1);
    std::vector<double> x, y, out;
    auto add = [&](double yy, double xx) {
        y.push_back(yy);
        x.push_back(xx);
    };
    auto sgn = [&]() { return rng() & 1 ? 1.0 : -1.0; };
    for (int k = 0; k < 200000; ++k) {
        add(sgn() * std::ldexp(1 + U(rng), int(rng() % 1900) - 950), std::ldexp(1 + U(rng), int(rng() % 1900) - 950));
        add((U(rng) - 0.5) * std::ldexp(1.0, -int(rng() % 60)), 1 + (U(rng) - 0.5) * std::ldexp(1.0, -int(rng() % 50)));
        const double s = std::ldexp(1.0, int(rng() % 120) - 60);
        add((U(rng) - 0.5) * s, (U(rng) - 0.5) * s);
    }
    for (int i = 0; i <= 128; ++i)
        for (int h = 0; h < 2; ++h)
            for (int d = -3; d <= 3; ++d) {
                double a = 1 + (i + 0.5 * h) / 128, t = (i + 0.5 * h) / 128;
                for (int k = 0; k < std::abs(d); ++k) {
                    a = std::nextafter(a, d > 0 ? INFINITY : 0.0);
                    t = std::nextafter(t, d > 0 ? INFINITY : -1.0);
                }
                for (int q = 0; q < 8 && t != 0; ++q) {
                    const double s = q & 1 ? -1.0 : 1.0, r = q & 2 ? -1.0 : 1.0;
                    q & 4 ? add(r, s * t) : add(s * t, r);
                }
                add(t, a);
            }
    for (int e : {-1022, -1021, -1020, -1019, -101, -100, -99, 99, 100, 101, 1019, 1020, 1021, 1023})  // the switches
        for (int d = -2; d <= 2; ++d) {
            double a = std::ldexp(1.0, e);
            for (int k = 0; k < std::abs(d); ++k) a = std::nextafter(a, d > 0 ? INFINITY : 0.0);
            if (a < std::ldexp(1.0, -1022)) continue;
            for (double c : {0.25, 1.0, 3.0}) add(c * a, a), add(-a, c * std::fmin(a, 1e307)), add(1.0, -a);
        }
    if (!run(false, x, y, out)) return 1;
    const double e52 = std::ldexp(1.0, -52);
    double w[NOUT] = {};
    for (size_t i = 0; i < x.size(); ++i) {
        const double* o = &out[NOUT * i];
        const ld X = x[i];
        const ld R = 1 / X, A = atan2l(y[i], X);
        auto worst = [&](int k, ld err, double unit) {
            const double e = double(fabsl(err)) / unit;
            if (!(e <= w[k])) w[k] = e;  // a NaN stays
        };
        if (std::isnormal(double(R))) worst(0, o[0] - R, ulp(double(R)));
        if (x[i] > 0) {
            const ld S = sqrtl(X), L = logl(X), H = logl(X / 2);
            if (std::isnormal(x[i])) worst(1, o[1] - 1 / S, ulp(double(1 / S)));  // rsqrt takes normal numbers only
            worst(2, o[2] - S, ulp(double(S)));
            worst(3, o[3] - 1 / S, ulp(double(1 / S)));
            worst(4, o[4] - L, e52 * std::fmax(1.0, double(fabsl(L))));
            worst(5, o[5] - H, e52 * std::fmax(1.0, double(fabsl(H))));
        }
        if (std::isnormal(double(A))) worst(6, o[6] - A, 2 * ulp(double(A)));
    }
    // zero, subnormal, infinite and NaN arguments: CUDA's values
    const double inf = INFINITY, den = 5e-324, nan = NAN;
    std::vector<double> sx, sy, so, sg;
    for (double a : {0.0, -0.0, den, -den, inf, -inf, 1e308, -1e308, 1e-308, 1.0, -1.0, nan})
        for (double b : {0.0, -0.0, den, -den, inf, -inf, 1e300, 1e-300, 1.0, -1.0, nan}) sx.push_back(a), sy.push_back(b);
    if (!run(false, sx, sy, so) || !run(true, sx, sy, sg)) return 1;
    int bad = 0;
    auto same = [&](double a, double b) { return (std::isnan(a) && std::isnan(b)) || (a == b && std::signbit(a) == std::signbit(b)); };
    for (size_t i = 0; i < sx.size(); ++i) {
        const double *f = &so[NOUT * i], *g = &sg[NOUT * i];
        const bool normal = std::isnormal(sx[i]);
        if (!normal || std::fabs(sx[i]) > 1e307 || std::fabs(sx[i]) < 1e-307) bad += !same(f[0], g[0]);
        if (!normal || sx[i] < 0)
            for (int k : {2, 3, 4}) bad += !same(f[k], g[k]);
        bad += !(same(f[6], g[6]) || (std::fabs(f[6] - g[6]) <= 4 * ulp(g[6]) && std::signbit(f[6]) == std::signbit(g[6])));
    }
    std::printf("rcp %.3f\nrsqrt %.3f\nsqrt %.3f\nsqrt_inv %.3f\nlog %.3f\nlog_half %.3f\natan2 %.3f\nspecial %d\n", w[0], w[1],
                w[2], w[3], w[4], w[5], w[6], bad);
    return 0;
}
