// One term of the primary-Compton scatter sysmat, host- and device-callable:
// the kernels in scatter_kernel.cu evaluate it on the GPU, and host-side
// checks run the same arithmetic on the CPU.  See scatter_kernel.cu for the
// physics and the reference lines each step follows.
#pragma once

#include <cmath>
#include <cstring>

#include "scatter.h"
#include "tracer.cuh"

namespace smb {

constexpr float kDelta = 0.01f;   // the reference's DeltaTheta, as a float
constexpr float kNodesPerRad = (float)kKnNodes / 3.14159265358979323846f;

// Fast quotient, root and reciprocal root for values (never for a decision the
// reference takes): about 2 ulp, against ~10 instructions for the IEEE forms this
// translation unit is compiled with.
SM_HD float sm_rsqrt(float x) { return fast_rsqrt(x); }

SM_HD float sm_fdiv(float a, float b) {
#ifdef __CUDA_ARCH__
    float r;
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
#else
    return a / b;
#endif
}

SM_HD float sm_fsqrt(float x) { return x > 1e-37f ? x * sm_rsqrt(x) : 0.0f; }

SM_HD int sm_rint(float x) {
#ifdef __CUDA_ARCH__
    return __float2int_rn(x);
#else
    return (int)std::nearbyint(x);
#endif
}

// ---- Klein-Nishina rectangle sum in closed form ---------------------------------------
// sum_{i=0}^{n} g(a + i delta) delta = [F(b) - F(a)] + delta/2 (g(a) + g(b))
//   + delta^2/12 (g'(b) - g'(a)) + O(delta^4 g'''),  b = a + n delta.
struct KnEval {
    float f_hi, f_lo, part, g, dg;
};

SM_HD KnEval kn_at(const KnNode* kn, float theta) {
    int j = sm_rint(theta * kNodesPerRad);
    j = j < 0 ? 0 : (j > kKnNodes ? kKnNodes : j);
    const KnNode n = kn[j];
    const float t = theta - n.theta;
    KnEval e;
    e.f_hi = n.f_hi;
    e.f_lo = n.f_lo;
    e.part = t * fmaf(t, fmaf(t, fmaf(t, fmaf(t, n.c4 * 0.2f, n.c3 * 0.25f), n.c2 * (1.0f / 3.0f)), n.c1 * 0.5f), n.c0);
    e.g = fmaf(t, fmaf(t, fmaf(t, fmaf(t, n.c4, n.c3), n.c2), n.c1), n.c0);
    e.dg = fmaf(t, fmaf(t, fmaf(t, 4.0f * n.c4, 3.0f * n.c3), 2.0f * n.c2), n.c1);
    return e;
}

SM_HD float kn_rect_sum(const KnNode* kn, float a, int n) {
    const float b = a + (float)n * kDelta;     // the reference's last sample, theta_low + n * DeltaTheta
    const KnEval A = kn_at(kn, a), B = kn_at(kn, b);
    const float integral = ((B.f_hi - A.f_hi) + (B.f_lo - A.f_lo)) + (B.part - A.part);
    return integral + 0.5f * kDelta * (A.g + B.g) + (kDelta * kDelta / 12.0f) * (B.dg - A.dg);
}

// ---- window probability ------------------------------------------------------------------
// erfc and erf from cubic Taylor pieces at the nodes j / 64, built in double: one 16-byte load
// and six steps each.  The fourth derivative, below 4.4, leaves 7e-10 of a piece (of erf
// 2e-9 of the value), and the ends cut off 2e-9.  The cubic coefficient moves a piece by less
// than 2e-7, so eight bits of it do: the low half of its word holds, as the upper half of
// a float, what rounding took off the node's value, and the error is that of the result.
// erfc has the nodes of [-4.25, 4.25]; erf, which is odd, those of [0, 4.25] after them, times a
// factor that makes its slope at zero, which scales every small value, a float; half
// the factor's inverse is one too (both to 3e-14).
constexpr int kErfcPerUnit = 64, kErfcHalf = 272, kErfcNodes = 2 * kErfcHalf + 1;
constexpr int kWindowNodes = kErfcNodes + kErfcHalf + 1;
constexpr float kErfSlope = 0x1.4ec864p+0f, kErfHalf = 0x1.b9c698p-2f;   // the slope, 1 / (slope sqrt(pi))

inline float4 taylor_node(double value, double d1, double d2, double d3) {
    const float x = (float)value, rest = (float)(value - (double)x), w = (float)d3;
    unsigned wb, rb;
    std::memcpy(&wb, &w, 4);
    std::memcpy(&rb, &rest, 4);
    wb = (wb & 0xffff0000u) | rb >> 16;
    float packed;
    std::memcpy(&packed, &wb, 4);
    return float4{x, (float)d1, (float)d2, packed};
}

inline void build_erfc_table(float4* out) {
    for (int j = 0; j < kErfcNodes; ++j) {
        const double z = (double)(j - kErfcHalf) / kErfcPerUnit, d = -2.0 / std::sqrt(M_PI) * std::exp(-z * z);
        out[j] = taylor_node(std::erfc(z), d, -z * d, (4.0 * z * z - 2.0) * d / 6.0);
    }
    out[0] = float4{2.0f, 0.0f, 0.0f, 0.0f};
    out[kErfcNodes - 1] = float4{0.0f, 0.0f, 0.0f, 0.0f};
}

inline void build_window_table(float4* out) {
    build_erfc_table(out);
    for (int j = 0; j <= kErfcHalf; ++j) {
        const double z = (double)j / kErfcPerUnit, d = kErfSlope * std::exp(-z * z);
        out[kErfcNodes + j] = taylor_node(0.5 * std::sqrt(M_PI) * kErfSlope * std::erf(z), d, -z * d, (4.0 * z * z - 2.0) * d / 6.0);
    }
    out[kWindowNodes - 1] = taylor_node(0.5 * std::sqrt(M_PI) * kErfSlope, 0.0, 0.0, 0.0);
}

constexpr float kErfcEnd = (float)kErfcHalf / (float)kErfcPerUnit;

// The function whose node at zero is *centre, nodes to either side as far as z reaches, as the
// node's value (x) and what is added to it (y).
SM_HD float2 taylor_at(const float4* centre, float z) {
    // adding 1.5 2^23 rounds to a whole number, whose low bits are the sum's
    const float magic = 12582912.0f, y = fmaf(z, (float)kErfcPerUnit, magic), k = y - magic;
#ifdef __CUDA_ARCH__
    const float4 n = __ldg(centre + (__float_as_int(y) - 0x4b400000));
    const float rest = __int_as_float(__float_as_int(n.w) << 16);
#else
    const float4 n = centre[(int)k];
    unsigned b;
    std::memcpy(&b, &n.w, 4);
    b <<= 16;
    float rest;
    std::memcpy(&rest, &b, 4);
#endif
    const float t = fmaf(k, -1.0f / kErfcPerUnit, z);
    return float2{n.x, fmaf(t, n.y, fmaf(t * t, fmaf(t, n.w, n.z), rest))};
}

SM_HD float erfc_at(const float4* nodes, float z) {
    const float2 v = taylor_at(nodes + kErfcHalf, fminf(fmaxf(z, -kErfcEnd), kErfcEnd));
    return v.x + v.y;
}

// 0.5 (erf(z2) - erf(z1)) from the table of build_window_table, without a difference of
// rounded numbers: through erf of both distances where zero lies between the ends, else through
// erfc of them, and always with the nodes' values apart from what is added to them.
// On the GPU against double, windows of +-10 % down to +-0.05 % of the energy at 10 %
// resolution: 4e-8 in the mean square and 2.8e-7 at most; erff and erfcf give 7e-8 and 3e-7
// for the widest, 4e-6 and 2e-5 for the narrowest.
SM_HD float window_probability(const float4* nodes, float z1, float z2) {
    const bool across = (z1 < 0.0f) != (z2 < 0.0f);
    const float4* centre = nodes + (across ? kErfcNodes : kErfcHalf);
    const float2 a = taylor_at(centre, fminf(fabsf(z1), kErfcEnd)), b = taylor_at(centre, fminf(fabsf(z2), kErfcEnd));
    const float sign = across ? 1.0f : -1.0f, half = across ? kErfHalf : 0.5f;
    const float p = fmaf(half, fmaf(sign, b.x, a.x), half * fmaf(sign, b.y, a.y));   // large and small parts apart
    return copysignf(p, z2 - z1);   // left of zero p is the difference the other way round
}

// angle between u and e (atan2 of |u x e| and u . e: accurate at every angle)
SM_HD void angle_parts(float ux, float uy, float uz, const float3& e, float* sine, float* cosine) {
    const float cx = uy * e.z - uz * e.y, cy = uz * e.x - ux * e.z, cz = ux * e.y - uy * e.x;
    *sine = sm_fsqrt(fmaf(cx, cx, fmaf(cy, cy, cz * cz)));
    *cosine = fmaf(ux, e.x, fmaf(uy, e.y, uz * e.z));
}

// atan2(s, c) for s >= 0: atan(t) = t + t x q(x), x = t^2, of the smaller quotient t <= 1.
// q fits the relative error of the whole in the least-maximum sense (Lawson's reweighted
// least squares on 4001 Chebyshev points; each coefficient rounded to a float in turn, from
// the highest, and the rest fitted again): 2.3e-8 with the coefficients as written.  The
// quotient is corrected once and pi / 2 and pi are carried to more than 24 bits, so the
// rest is rounding.  (Not FINE, for a decision with a margin: without these two, to 3e-7.)
// On the GPU 2.3e-8 rad in the mean square for angles to 0.8, 7.3e-8 to pi; atan2f, which
// it stands for, 2.6e-8 and 1.13e-7.
template <bool FINE = true>
SM_HD float angle_quick(float s, float c) {
    const float a = fabsf(c), lo = fminf(s, a), hi = fmaxf(s, a);
    const float t = !(hi > 0.0f) ? 0.0f : (FINE ? near_div(lo, hi, fast_rcp(hi)) : sm_fdiv(lo, hi)), x = t * t;
    float q = 0.00292069255f;
    q = fmaf(q, x, -0.0163679291f);
    q = fmaf(q, x, 0.0432118624f);
    q = fmaf(q, x, -0.0755221471f);
    q = fmaf(q, x, 0.106660053f);
    q = fmaf(q, x, -0.142110556f);
    q = fmaf(q, x, 0.199937731f);
    q = fmaf(q, x, -0.333331525f);
    float p = fmaf(t * x, q, t);
    const bool steep = s > a, back = c < 0.0f;
    const float turn = steep ? 1.57079632679489662f : (back ? 3.14159265358979324f : 0.0f);
    if (steep != back) p = -p;
    return turn + (FINE ? fmaf(turn, -2.78275e-8f, p) : p);   // pi's float is above pi by 2.78275e-8 of it
}

// Polar range of the unit seen from S along u: the lowest angle and the reference's
// number of 0.01 rad steps above it, (int)((hi - lo) / 0.01f).  The step count comes
// from the quick angles except within 2e-4 of a whole step (their error is below 1e-4
// of one), where the reference's own expression decides.
struct PolarRange {
    float lo;
    int n;
};

template <bool QUICK>
SM_HD PolarRange polar_range(float ux, float uy, float uz, const float3& near, const float3& far, bool from_zero) {
    float sn, cn, sf, cf;
    angle_parts(ux, uy, uz, near, &sn, &cn);
    angle_parts(ux, uy, uz, far, &sf, &cf);
    PolarRange r;
    float steps = 0.0f;
    if (QUICK) {
        r.lo = from_zero ? 0.0f : angle_quick(sn, cn);
        steps = (angle_quick<false>(sf, cf) - r.lo) * 100.0f;
        r.n = (int)steps;
    }
    if (!QUICK || fabsf(steps - rintf(steps)) < 2e-4f) {
        r.lo = from_zero ? 0.0f : atan2f(sn, cn);
        r.n = (int)((atan2f(sf, cf) - r.lo) / kDelta);
    }
    return r;
}

// Per-lane constants of the detecting crystal.
struct Det {
    float x, y, z, cm, sm;       // centre (world, y with Image[11]); cos(-rot), sin(-rot)
    float hw, ht, hh;            // half sizes
    float r_unit;                // bounding radius of the unit (scatter.cu:1243)
    float mu_pe, mu_c, res, lo, hi;
    float c_cut;                 // cos(theta) at or below which the 2-sigma window cut rejects, less a margin
    bool on;
};

// The lower window cut as a bound on cos(theta): E' (1 + k sqrt(E'/E0)) <= lo
// (scatter.cu:1231) rejects every E' up to the root E*, i.e. every cos(theta)
// up to 1 - (E0/E* - 1)/alpha.  Returns that cosine less a margin of 2e-3
// (far above the rounding of the per-term test), -2 when nothing is cut and
// 2 when everything is.  The upper cut is left to the per-term test.
SM_HD float window_cos_cut(float e0, float alpha, float res, float lo) {
    const float k = 2.0f * res / 2.35482f;
    auto lhs = [&](float E) { return E * (1.0f + k * sqrtf(E / e0)) - lo; };
    float a = e0 / (1.0f + 2.0f * alpha), b = e0;   // E' over theta in [pi, 0]
    if (lhs(b) <= 0.0f) return 2.0f;
    if (lhs(a) > 0.0f) return -2.0f;
    for (int it = 0; it < 40; ++it) {
        const float m = 0.5f * (a + b);
        if (lhs(m) <= 0.0f) a = m;
        else b = m;
    }
    return 1.0f - (e0 / a - 1.0f) / alpha - 2e-3f;
}

// Per-(detector, scatter point) constants.
struct Src {
    float sx, sy, sz;            // scatter point, world
    float ssx, ssy, ssz;         // ... in the detecting crystal's frame
    float bx, by, bz, bb, L;     // D - S, |D - S|^2, |D - S|
    float phi_k;                 // R_unit / (2 L)
    float c_len;                 // below this cos(theta) the line I -> S misses the unit's bounding sphere
    float e[8][3];               // unit vectors from S to the unit's corners (detector frame)
    float4 pr;                   // pair data
    SM_HD float3 corner(int i) const { return make_float3(e[i][0], e[i][1], e[i][2]); }
    // corner(i) of an index known at run time only, without indexing the registers
    SM_HD float3 pick(int i) const {
        float3 v = corner(0);
#pragma unroll
        for (int k = 1; k < 8; ++k)
            if (i == k) v = corner(k);
        return v;
    }
};

// S, its detector-frame image and D - S: what the column cull needs.
SM_HD void make_src_basic(const Det& D, float4 S, Src& C) {
    C.sx = S.x;
    C.sy = S.y;
    C.sz = S.z;
    C.ssx = (S.x - D.x) * D.cm - (S.z - D.z) * D.sm;
    C.ssy = S.y - D.y;
    C.ssz = (S.x - D.x) * D.sm + (S.z - D.z) * D.cm;
    C.bx = D.x - S.x;
    C.by = D.y - S.y;
    C.bz = D.z - S.z;
    C.bb = fmaf(C.bx, C.bx, fmaf(C.by, C.by, C.bz * C.bz));
    C.L = sqrtf(C.bb);
}

// The rest of the per-(lane, scatter point) constants.
SM_HD void make_src_rest(const Det& D, float4 pr, Src& C) {
    C.phi_k = D.r_unit / 2.0f / C.L;
    const float q = D.r_unit / C.L;
    C.c_len = q < 1.0f ? sqrtf(1.0f - q * q) - 1e-3f : -2.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float ex = ((i & 1) ? D.hw : -D.hw) - C.ssx;
        const float ey = ((i & 2) ? D.ht : -D.ht) - C.ssy;
        const float ez = ((i & 4) ? D.hh : -D.hh) - C.ssz;
        const float inv = sm_rsqrt(fmaf(ex, ex, fmaf(ey, ey, ez * ez)));
        C.e[i][0] = ex * inv;
        C.e[i][1] = ey * inv;
        C.e[i][2] = ez * inv;
    }
    C.pr = pr;
}

// Largest cos(theta) over the voxel column I0 + t e, t in [0, T] (|e| = 1):
// with w = S - I = w_perp + u e, u = (w0 . e) - t, cos = (B + u beta) / sqrt(A + u^2)
// (A = |w_perp|^2, B = w_perp . b^, beta = e . b^) is stationary only at u = beta A / B.
SM_HD float column_max_cos(const Src& C, float i0x, float i0y, float i0z, float ex, float ey, float ez, float T) {
    const float wx = C.sx - i0x, wy = C.sy - i0y, wz = C.sz - i0z;
    const float inv_l = sm_rsqrt(C.bb);
    const float bx = C.bx * inv_l, by = C.by * inv_l, bz = C.bz * inv_l;
    const float p = fmaf(wx, ex, fmaf(wy, ey, wz * ez));
    const float px = wx - p * ex, py = wy - p * ey, pz = wz - p * ez;
    const float A = fmaf(px, px, fmaf(py, py, pz * pz));
    const float B = fmaf(px, bx, fmaf(py, by, pz * bz));
    const float beta = fmaf(ex, bx, fmaf(ey, by, ez * bz));
    auto f = [&](float u) { return (B + u * beta) * sm_rsqrt(A + u * u); };
    float m = fmaxf(f(p), f(p - T));
    if (B != 0.0f) {
        const float us = beta * A / B;
        if (us > p - T && us < p) m = fmaxf(m, f(us));
    }
    return m;
}

// One term without its weight W.  I: voxel (world); Is: voxel in the detector
// frame.  SrcT: Src, or a view of one kept in shared memory (same members).
// QUICK: the window probability from a table and the polar range from quick
// angles (a seventh less work, errors no larger); the transfer matrices, which are
// rounded to bf16 and compared with the exact columns at a thousandth of their
// size, keep the other form.
template <bool QUICK, class SrcT>
SM_HD float scatter_term(const ScatterParams& P, const Det& D, const SrcT& C, const KnNode* kn, const float4* window_nodes,
                                              float inv_norm, float ix, float iy, float iz, float isx, float isy,
                                              float isz) {
    // scatter angle at S between I -> S and S -> D (scatter.cu:1225)
    const float ax = C.sx - ix, ay = C.sy - iy, az = C.sz - iz;
    const float aa = fmaf(ax, ax, fmaf(ay, ay, az * az));
    const float inv_ab = sm_rsqrt(aa * C.bb);
    float c = fmaf(ax, C.bx, fmaf(ay, C.by, az * C.bz)) * inv_ab;
    c = fminf(1.0f, fmaxf(-1.0f, c));
    const float r = fmaf(P.alpha, 1.0f - c, 1.0f);       // E0 / E'
    const float E = sm_fdiv(P.e0, r);
    const float res_e = D.res * sm_rsqrt(r);                // res sqrt(E'/E0)
    const float k2 = res_e * (2.0f / 2.35482f);
    if ((E * (1.0f + k2) <= D.lo) || (E * (1.0f - k2) >= D.hi)) return 0.0f;   // 2-sigma window cut (:1231)
    const float inv_s2 = sm_fdiv(2.35482f / 1.41421356237309515f, res_e * E);   // 1 / (sigma sqrt 2)
    // 0.5 (erf(z2) - erf(z1)), through erfc when both limits lie on one side of E'
    const float z1 = (D.lo - E) * inv_s2, z2 = (D.hi - E) * inv_s2;
    float p_win;
    if (QUICK) p_win = window_probability(window_nodes, z1, z2);
    else if (z1 > 0.0f) p_win = 0.5f * (erfcf(z1) - erfcf(z2));
    else if (z2 < 0.0f) p_win = 0.5f * (erfcf(-z2) - erfcf(-z1));
    else p_win = 0.5f * (erff(z2) - erff(z1));
    // azimuth range (:1244-1252)
    const float cx = ay * C.bz - az * C.by, cy = az * C.bx - ax * C.bz, cz = ax * C.by - ay * C.bx;
    const float sn = sm_fsqrt(fmaf(cx, cx, fmaf(cy, cy, cz * cz))) * inv_ab;
    float phi_frac = 1.0f;
    if (!(C.L * sn * 2.0f <= D.r_unit)) phi_frac = 4.0f * asinf(fminf(sm_fdiv(C.phi_k, sn), 1.0f)) * 0.159154943091895336f;
    // polar range over the unit's corners (:1272-1298)
    const float ux = C.ssx - isx, uy = C.ssy - isy, uz = C.ssz - isz;
    // u . e_i orders the corners by angle (u is not normalised: the scale is common)
    float cmax = 0.0f, cmin = 0.0f;
    int near = 0, far = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float3 e = C.corner(i);
        const float ci = fmaf(ux, e.x, fmaf(uy, e.y, uz * e.z));
        if (i == 0 || ci > cmax) { cmax = ci; near = i; }
        if (i == 0 || ci < cmin) { cmin = ci; far = i; }
    }
    // the line from the voxel through S continues into the unit: theta_min = 0 (:1264-1266, :1293-1296);
    // it cannot unless it passes the unit's bounding sphere (cos(theta) >= c_len)
    bool through = false;
    if (c >= C.c_len) {
        // the segment reaches 1000 mm beyond S: chord_quick with the margin of its range
        // (its end point rounds within it too), else the reference's own points and chord
        const float dsq = fmaf(ux, ux, fmaf(uy, uy, uz * uz)), inv = sm_rsqrt(dsq);
        const float len = fmaf(dsq, inv, 1000.0f), k = len * inv;
        const ChordRay cr = make_chord_ray(isx, isy, isz, ux * k, uy * k, uz * k, len, 3e-6f * len);
        float chord;
        int f = cr.ok ? chord_quick(cr, 0.0f, 0.0f, 0.0f, D.hw, D.ht, D.hh, &chord) : -1;
        if (f < 0) {
            const float dis = sqrtf(dsq);
            const float xt = C.ssx + 1000.0f * (C.ssx - isx) / dis;
            const float yt = C.ssy + 1000.0f * (C.ssy - isy) / dis;
            const float zt = C.ssz + 1000.0f * (C.ssz - isz) / dis;
            const Box3 ub{-D.hw, -D.ht, -D.hh, D.hw, D.ht, D.hh};
            f = chord_through(isx, isy, isz, xt, yt, zt, ub) > 0.001f;
        }
        through = f != 0;
    }
    const PolarRange th = polar_range<QUICK>(ux, uy, uz, C.pick(near), C.pick(far), through);
    const float ratio = kn_rect_sum(kn, th.lo, th.n) * inv_norm;
    // attenuation and absorption at E' (:1309-1392)
    const float r3 = r * r * r;
    const float mu_pe = D.mu_pe * r3, mu_c = D.mu_c * r, mu = mu_pe + mu_c;
    const float att = fmaf(C.pr.x, r3, fmaf(C.pr.y, r, C.pr.z * mu));
    const float absorb = -expm1f(-C.pr.w * mu) * sm_fdiv(mu_pe, mu);
    return phi_frac * ratio * p_win * expf(-att) * absorb;
}

}  // namespace smb
