// Largest errors of the kick angles' sines and cosines (angles.cuh) on the host
// against 80-bit libm, per decade of |p|: "decade err_pi err_full err_short".
#include "angles.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

using namespace ifdm;

static double err[3];

static void one(double p) {
    const long double S = sinl((long double)p), C = cosl((long double)p);
    double s[3], c[3];
    sincos_pi(p, s[0], c[0]);
    sincos_series<true>(p, s[1], c[1]);
    sincos_series<false>(p, s[2], c[2]);
    for (int i = 0; i < 3; ++i) err[i] = std::max({err[i], (double)fabsl(s[i] - S), (double)fabsl(c[i] - C)});
}

int main() {
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> u(0.1, 1.0);
    for (int dec = -12; dec <= 9; ++dec) {
        err[0] = err[1] = err[2] = 0.0;
        const double top = std::pow(10.0, dec);
        for (int i = 0; i < 200000; ++i) one((i & 1 ? -top : top) * u(rng));
        // the ends of the quadrants and octants, and their neighbours
        for (int k = 0; k < 4000; ++k) {
            const double q = k * 0.78539816339744830962 * std::max(1.0, std::floor(top / 3000.0));
            if (std::fabs(q) > top) break;
            for (double p : {q, std::nextafter(q, 1e300), std::nextafter(q, -1e300)}) one(p), one(-p);
        }
        std::printf("%d %.3e %.3e %.3e\n", dec, err[0], err[1], err[2]);
    }
    return 0;
}
