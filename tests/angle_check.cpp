// Compares the scatter term's angle_quick with atan2 in double on the host:
// angle_check SEED COUNT.  Prints the largest relative error of angles below pi / 4, the
// largest error of those to pi / 2 and of those to pi, and whether the axes are exact.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "scatter_term.cuh"

using namespace smb;

int main(int argc, char** argv) {
    if (argc < 3) return 2;
    std::mt19937_64 gen(std::strtoull(argv[1], nullptr, 10));
    const long n = std::atol(argv[2]);
    auto U = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
    double low = 0.0, mid = 0.0, high = 0.0;
    for (long i = 0; i < n; ++i) {
        const double r = std::exp(U(-3, 5)), angle = i & 1 ? U(0, M_PI) : M_PI * std::pow(U(0, 1), 4);
        const float s = (float)(r * std::sin(angle)), c = (float)(r * std::cos(angle));
        if (!(s >= 0.0f)) continue;
        const double f = std::atan2((double)s, (double)c), e = std::fabs(angle_quick(s, c) - f);
        if (f < M_PI / 4) low = std::fmax(low, f > 0 ? e / f : e);
        else if (f < M_PI / 2) mid = std::fmax(mid, e);
        else high = std::fmax(high, e);
    }
    // the axes and the diagonals
    bool axes = angle_quick(0.0f, 0.0f) == 0.0f && angle_quick(0.0f, 2.0f) == 0.0f;
    const float h = 1.57079632679489662f;
    axes = axes && angle_quick(3.0f, 0.0f) == h && angle_quick(0.0f, -2.0f) == 2 * h;
    std::printf("%.4g %.4g %.4g %d\n", low, mid, high, (int)axes);
    return 0;
}
