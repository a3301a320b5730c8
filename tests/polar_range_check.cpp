// Compares the quick polar range with the reference-order one on the host:
// polar_range_check SEED COUNT DISTANCE.  Units of random size at about DISTANCE from
// the scatter point, seen along random directions, every fourth nearly at a whole
// number of steps.  Prints "<ranges> <other step counts> <largest difference of the
// lowest angle> <largest error of angle_quick>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "scatter_term.cuh"

using namespace smb;

int main(int argc, char** argv) {
    if (argc < 4) return 2;
    std::mt19937_64 gen(std::strtoull(argv[1], nullptr, 10));
    const long n = std::atol(argv[2]);
    const float dist = (float)std::atof(argv[3]);
    auto U = [&](float a, float b) { return std::uniform_real_distribution<float>(a, b)(gen); };
    auto unit = [&] {
        float x, y, z, s;
        do {
            x = U(-1, 1), y = U(-1, 1), z = U(-1, 1);
            s = x * x + y * y + z * z;
        } while (s > 1.0f || s < 0.01f);
        s = 1.0f / std::sqrt(s);
        return float3{x * s, y * s, z * s};
    };
    long other = 0;
    double lo_diff = 0.0, angle_err = 0.0;
    for (long i = 0; i < n; ++i) {
        const float3 u = unit();
        const float len = U(1, 80);
        const float3 c = unit();
        float3 near{}, far{};
        float cmax = -2, cmin = 2;
        const float hx = U(0.4f, 1.2f), hy = U(1, 3), hz = U(0.4f, 1.2f);
        for (int k = 0; k < 8; ++k) {
            float3 e{c.x * dist + (k & 1 ? hx : -hx), c.y * dist + (k & 2 ? hy : -hy), c.z * dist + (k & 4 ? hz : -hz)};
            const float s = 1.0f / std::sqrt(e.x * e.x + e.y * e.y + e.z * e.z);
            e = float3{e.x * s, e.y * s, e.z * s};
            const float d = u.x * e.x + u.y * e.y + u.z * e.z;
            if (d > cmax) cmax = d, near = e;
            if (d < cmin) cmin = d, far = e;
        }
        if (i % 4 == 0) {   // the farthest corner a whole number of steps from the nearest, to 1e-7 rad
            double a = std::acos((double)cmax) + 0.01 * (int)U(1, 30) + U(-1e-7f, 1e-7f);
            float3 w{u.y * near.z - u.z * near.y, u.z * near.x - u.x * near.z, u.x * near.y - u.y * near.x};
            const float s = 1.0f / std::sqrt(w.x * w.x + w.y * w.y + w.z * w.z + 1e-30f);
            w = float3{w.x * s, w.y * s, w.z * s};
            const float3 v{w.y * u.z - w.z * u.y, w.z * u.x - w.x * u.z, w.x * u.y - w.y * u.x};   // in the plane, normal to u
            const float ca = (float)std::cos(a), sa = (float)std::sin(a);
            far = float3{u.x * ca + v.x * sa, u.y * ca + v.y * sa, u.z * ca + v.z * sa};
        }
        const bool zero = i % 5 == 0;
        const PolarRange q = polar_range<true>(u.x * len, u.y * len, u.z * len, near, far, zero);
        const PolarRange r = polar_range<false>(u.x * len, u.y * len, u.z * len, near, far, zero);
        other += q.n != r.n;
        lo_diff = std::fmax(lo_diff, std::fabs((double)q.lo - r.lo));
        const float s = U(0, 1), k = U(-1, 1);
        angle_err = std::fmax(angle_err, std::fabs((double)angle_quick(s, k) - std::atan2((double)s, (double)k)));
    }
    std::printf("%ld %ld %.3g %.3g\n", n, other, lo_diff, angle_err);
    return 0;
}
