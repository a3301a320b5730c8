// Compares the scatter term's tabulated window probability with the double-precision one
// on the host: window_probability_check SEED COUNT WIDTH.  Windows (z1, z2) of width
// WIDTH to 2 WIDTH about and beside zero, every eighth with an end on zero.  Prints the
// largest |error| / p of the windows that hold zero, and the largest (|error| - 3e-9) /
// erfc(|z|) of the others, z their end nearer to zero.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "scatter_term.cuh"

using namespace smb;

int main(int argc, char** argv) {
    if (argc < 4) return 2;
    std::mt19937_64 gen(std::strtoull(argv[1], nullptr, 10));
    const long n = std::atol(argv[2]);
    const float width = (float)std::atof(argv[3]);
    std::vector<float4> table(kWindowNodes);
    build_window_table(table.data());
    auto U = [&](float a, float b) { return std::uniform_real_distribution<float>(a, b)(gen); };
    double across = 0.0, beside = 0.0;
    for (long i = 0; i < n; ++i) {
        const float w = width * U(1, 2);
        float z1 = i & 1 ? -w * U(0, 1) : U(-4, 3.9f);
        if (i % 8 == 0) z1 = i % 16 ? 0.0f : -w;
        const float z2 = z1 + w;
        const double p = window_probability(table.data(), z1, z2);
        if (z1 <= 0.0f && z2 >= 0.0f) {
            const double f = 0.5 * (std::erf((double)z2) - std::erf((double)z1));
            if (f > 0) across = std::fmax(across, std::fabs(p - f) / f);
        } else {
            const double a = z1 > 0 ? z1 : -z2, b = z1 > 0 ? z2 : -z1, f = 0.5 * (std::erfc(a) - std::erfc(b));
            beside = std::fmax(beside, (std::fabs(p - f) - 3e-9) / std::erfc(a));
        }
    }
    const float inf = INFINITY;
    if (std::fabs(window_probability(table.data(), -inf, inf) - 1.0) > 1.2e-7 || window_probability(table.data(), 9.0f, inf) != 0.0f) across = inf;
    // a window whose ends are exchanged: minus the window, as from the functions themselves
    if (std::fabs(window_probability(table.data(), 0.5f, -0.25f) - 0.5 * (std::erfc(0.5) - std::erfc(-0.25))) > 1e-6) across = inf;
    std::printf("%.4g %.4g\n", across, beside);
    return 0;
}
