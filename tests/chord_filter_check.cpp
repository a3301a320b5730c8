// Compares the tracer's chord_quick, chord_filter and hole_filter with the reference-order
// chord_through and chord_hole on the host: chord_filter_check SEED COUNT RANGE.
// Prints "<wrong calls> <clear hits> <clear misses> <unclear> <largest value error>
// <holes called missed> <holes called crossed> <of them with another value>
// <crossed boxes with another chord_value> <flattened segments>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "tracer.cuh"

using namespace smb;

int main(int argc, char** argv) {
    if (argc < 4) return 2;
    std::mt19937_64 gen(std::strtoull(argv[1], nullptr, 10));
    const long n = std::atol(argv[2]);
    const float range = (float)std::atof(argv[3]), delta = 1.5e-6f * range;
    auto U = [&](float a, float b) { return std::uniform_real_distribution<float>(a, b)(gen); };
    auto side = [&](float h) { return U(0, 1) < 0.5f ? -h : h; };
    const float lat = 0.35f * range;   // image and detector half width; depth up to half the range
    long wrong = 0, hits = 0, misses = 0, unclear = 0, hole_misses = 0, hole_hits = 0, hole_other = 0, other = 0, flat = 0;
    double worst = 0.0;
    for (long i = 0; i < n; ++i) {
        const float hx = U(0.3f, 2), hy = U(0.3f, 4), hz = U(0.3f, 2), near = 3 * delta;
        const float ky = U(0.25f, 0.45f) * range;
        float px = U(-lat, lat), py = U(-0.2f, 0.1f) * range, pz = U(-lat, lat);
        float qx = U(-lat, lat), qy = ky + U(-hy, 3 * hy), qz = U(-lat, lat);
        // the box: around the ray, or with an edge or a corner within a few margins of it
        const float depth = ky + (i % 4 < 2 ? side(hy) : U(-hy, hy)), l = (depth - py) / (qy - py);
        float kx = px + (qx - px) * l, kz = pz + (qz - pz) * l;
        if (i & 1) {
            kx += U(-1.5f, 1.5f) * hx;
            kz += U(-1.5f, 1.5f) * hz;
        } else {
            kx += side(hx) + U(-near, near);
            kz += U(0, 1) < 0.3f ? U(-hz, hz) : side(hz) + U(-near, near);
        }
        if (i % 7 == 0) {          // the segment ends at the box's faces
            qx = kx + U(-1.2f, 1.2f) * hx;
            qz = kz + U(-1.2f, 1.2f) * hz;
            qy = ky + side(hy) + U(-0.003f, 0.003f);
        }
        if (i % 11 == 0) px = qx + U(-0.004f, 0.004f);       // nearly parallel to a face
        if (i % 13 == 0) {         // ... or starts there
            px = kx + side(hx) + U(-0.002f, 0.002f);
            py = ky - hy + U(-0.003f, 0.003f);
            pz = kz + U(-1, 1) * hz;
        }
        if (i % 17 == 0) qx = px + U(-0.003f, 0.003f);       // below the degenerate extent, or nearly
        if (i % 34 == 0) qz = pz;
        if (i % 51 == 0) qy = py;
        const float dx = qx - px, dy = qy - py, dz = qz - pz, len = std::sqrt(dx * dx + dy * dy + dz * dz);
        const ChordRay r = make_chord_ray(px, py, pz, dx, dy, dz, len, delta);
        const Box3 box{-hx, -hy, -hz, hx, hy, hz};
        float chord = 0, quick = 0, value = 0, ref;
        int f, fq;
        if (i % 3) {
            f = r.ok ? chord_filter(r, kx, ky, kz, hx, hy, hz, delta, &chord) : -1;
            fq = r.ok ? chord_quick(r, kx, ky, kz, hx, hy, hz, &quick) : -1;
            value = chord_value(px - kx, py - ky, pz - kz, qx - kx, qy - ky, qz - kz, hx, hy, hz, r.ix, r.iy, r.iz,
                                1 / len);
            ref = chord_through(px - kx, py - ky, pz - kz, qx - kx, qy - ky, qz - kz, box);
        } else {
            const float a = U(-0.5f, 0.5f), c = std::cos(a), s = std::sin(a), ax = px - kx, az = pz - kz;
            const ChordRay k = make_chord_ray(fmaf(ax, c, -az * s), py - ky, fmaf(ax, s, az * c), fmaf(dx, c, -dz * s), dy,
                                              fmaf(dx, s, dz * c), len, 2 * delta);
            f = k.ok ? chord_filter(k, 0, 0, 0, hx, hy, hz, 2 * delta, &chord) : -1;
            fq = k.ok ? chord_quick(k, 0, 0, 0, hx, hy, hz, &quick) : -1;
            value = chord_value(ax * c - az * s, py - ky, ax * s + az * c, (qx - kx) * c - (qz - kz) * s, qy - ky,
                                (qx - kx) * s + (qz - kz) * c, hx, hy, hz, k.ix, k.iy, k.iz, 1 / len);
            ref = chord_through(ax * c - az * s, py - ky, ax * s + az * c, (qx - kx) * c - (qz - kz) * s, qy - ky,
                                (qx - kx) * s + (qz - kz) * c, box);
        }
        ChordRay e = r;
        if (i % 3 && !r.ok && flatten(&e, dx, dy, dz)) {
            float c;
            wrong += chord_filter(e, kx, ky, kz, hx, hy, hz, delta, &c) == 0 && ref != 0;
            ++flat;
        }
        if (fq >= 0) wrong += (fq != 0) != (ref != 0) || (f >= 0 && f != fq) || (fq == 1 && f == 1 && quick != chord);
        if (f < 0) ++unclear;
        else if (f == 0) { ++misses; wrong += ref != 0; }
        else {
            ++hits;
            wrong += ref == 0 || std::fabs(value - ref) > 1e-6f * len;
            other += value != ref;
            worst = std::fmax(worst, std::fabs((double)chord - ref) / (delta * len * std::fmax(r.ax, std::fmax(r.ay, r.az))));
        }
        // a hole of radius hx between ky - hy and ky + hy; every other one has its wall near the ray
        if (py < ky - hy && dy > 0) {
            float hxc = kx, hzc = kz;
            if (i % 5 < 3) {
                const float a = U(0, 6.2831853f), g = hx + U(-near, near), m = (ky + U(-hy, hy) - py) / dy;
                const float m1 = i % 5 == 0 ? (ky - hy - py) / dy : m;
                hxc = px + dx * m1 + g * std::cos(a);
                hzc = pz + dz * m1 + g * std::sin(a);
            }
            float hc = 0;
            const int hf = hole_filter(px, py, pz, dx, dy, dz, r.iy, len, hxc, ky - hy, ky + hy, hzc, hx, delta, &hc);
            const float hr = chord_hole(px, py, pz, qx, qy, qz, hxc, ky - hy, ky + hy, hzc, hx);
            hole_misses += hf == 0;
            hole_hits += hf == 1;
            hole_other += hf == 1 && hc != hr;
            wrong += (hf == 0 && hr != 0) || (hf == 1 && (hr == 0 || std::fabs(hc - hr) > 2e-6f * len));
        }
    }
    std::printf("%ld %ld %ld %ld %.3g %ld %ld %ld %ld %ld\n", wrong, hits, misses, unclear, worst, hole_misses, hole_hits, hole_other, other, flat);
    return 0;
}
