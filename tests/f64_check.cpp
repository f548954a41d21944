// Largest errors of vp_f64.cuh's functions (its host compilation: the seeds are 20-bit roundings) against the library's
// in long double, over random arguments of many magnitudes and over the edges of the tables and ranges. Prints one line
// per function: name, error in ulp (or in units of 2^-52 as the header states them).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

#include "vp_f64.cuh"

typedef long double ld;

static double ulp(double x) {
    x = std::fabs(x);
    return std::nextafter(x, INFINITY) - x;
}

int main() {
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> U(0, 1);
    const double e52 = std::ldexp(1.0, -52);
    double rcp = 0, rsq = 0, sq = 0, lg = 0, at = 0;
    auto one = [&](double x) {
        const ld X = x;
        rcp = std::fmax(rcp, double(std::fabs(f64::rcp(x) - 1 / X) / ulp(double(1 / X))));
        rsq = std::fmax(rsq, double(std::fabs(f64::rsqrt(x) - 1 / sqrtl(X)) / ulp(double(1 / sqrtl(X)))));
        sq = std::fmax(sq, double(std::fabs(f64::sqrt(x) - sqrtl(X)) / ulp(double(sqrtl(X)))));
        const ld L = logl(X);
        lg = std::fmax(lg, double(std::fabs(f64::log(x) - L) / (e52 * fmaxl(1, std::fabs(L)))));
        lg = std::fmax(lg, double(std::fabs(f64::log<-1>(x) - logl(X / 2)) / (e52 * fmaxl(1, std::fabs(logl(X / 2))))));
    };
    auto two = [&](double y, double x) {
        const ld T = atan2l(y, x);
        at = std::fmax(at, double(std::fabs(f64::atan2(y, x) - T) / std::fmax(2 * ulp(double(T)), 0.0)));
    };
    for (int k = 0; k < 2000000; ++k) {
        one(std::ldexp(1 + U(rng), int(rng() % 600) - 300));
        one(1 + (U(rng) - 0.5) * std::ldexp(1.0, -int(rng() % 50)));
        const double s = std::ldexp(1.0, int(rng() % 120) - 60);
        two((U(rng) - 0.5) * s, (U(rng) - 0.5) * s);
        two((U(rng) - 0.5) * std::ldexp(1.0, -int(rng() % 60)), (U(rng) - 0.5) * std::ldexp(1.0, -int(rng() % 60)));
    }
    for (int i = 0; i <= 128; ++i)  // the tables' points and the halves between them, and their neighbours
        for (int h = 0; h < 2; ++h)
            for (int d = -3; d <= 3; ++d) {
                double x = 1 + (i + 0.5 * h) / 128;
                for (int k = 0; k < std::abs(d); ++k) x = std::nextafter(x, d > 0 ? INFINITY : 0.0);
                one(x);
                double t = (i + 0.5 * h) / 128;
                for (int k = 0; k < std::abs(d); ++k) t = std::nextafter(t, d > 0 ? INFINITY : -1.0);
                for (int q = 0; q < 8; ++q) {
                    const double y = q & 1 ? -t : t, x2 = q & 2 ? -1.0 : 1.0;
                    if (t != 0) q & 4 ? two(x2, y) : two(y, x2);
                }
            }
    // what the fast forms pass on: the library's values
    int bad = 0;
    auto same = [&](double a, double b) { bad += !(a == b || (std::isnan(a) && std::isnan(b))) || std::signbit(a) != std::signbit(b); };
    const double inf = INFINITY, den = 5e-324;
    for (double x : {0.0, -0.0, den, -den, inf, -inf, 1e308, -1e308, 1e-308, double(NAN)}) same(f64::rcp(x), 1.0 / x);
    for (double x : {0.0, den, inf, -1.0, double(NAN)}) {
        if (x >= 0) same(f64::log(x), std::log(x));
        else bad += !std::isnan(f64::log(x));
        if (x >= 0) same(f64::sqrt(x), std::sqrt(x));
        else bad += !std::isnan(f64::sqrt(x));
    }
    for (double y : {0.0, -0.0, 1.0, -1.0, inf, -inf, den, 1e300, 1e-300})
        for (double x : {0.0, -0.0, 1.0, -1.0, inf, -inf, den, 1e300, 1e-300}) {
            const double a = f64::atan2(y, x), b = std::atan2(y, x);
            bad += !(std::fabs(a - b) <= 2 * ulp(b)) || std::signbit(a) != std::signbit(b);
        }
    bad += !std::isnan(f64::atan2(NAN, 1.0)) + !std::isnan(f64::atan2(1.0, NAN));
    std::printf("rcp %.3f\nrsqrt %.3f\nsqrt %.3f\nlog %.3f\natan2 %.3f\nspecial %d\n", rcp, rsq, sq, lg, at, bad);
    return 0;
}
