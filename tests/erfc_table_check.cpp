// Compares the scatter term's tabulated erfc with the double-precision function on the
// host: erfc_table_check SEED COUNT LOW HIGH.  Prints the largest value of
// |error| / (1.25e-7 erfc + 3e-9) over COUNT arguments in [LOW, HIGH], every eighth
// next to a node or midway between two.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "scatter_term.cuh"

using namespace smb;

int main(int argc, char** argv) {
    if (argc < 5) return 2;
    std::mt19937_64 gen(std::strtoull(argv[1], nullptr, 10));
    const long n = std::atol(argv[2]);
    const float lo = (float)std::atof(argv[3]), hi = (float)std::atof(argv[4]);
    std::vector<float4> table(kErfcNodes);
    build_erfc_table(table.data());
    auto U = [&](float a, float b) { return std::uniform_real_distribution<float>(a, b)(gen); };
    double worst = 0.0;
    for (long i = 0; i < n; ++i) {
        float z = U(lo, hi);
        if (i % 8 == 0) z = std::nearbyint(z * 128.0f) / 128.0f + U(-1e-6f, 1e-6f);
        const double f = std::erfc((double)z);
        worst = std::fmax(worst, std::fabs(erfc_at(table.data(), z) - f) / (1.25e-7 * f + 3e-9));
    }
    for (float z : {-INFINITY, INFINITY})
        if (erfc_at(table.data(), z) != std::erfc(z)) worst = INFINITY;
    std::printf("%.4f\n", worst);
    return 0;
}
