// Device ray primitives of the photoelectric tracer.
//
// Every hit/miss decision here is taken in IEEE single precision with the same
// operations, in the same order, as the reference primitives
// (PEGen_RayTracing_CircularHole/PESysMatGen.cu:19-373).  The translation unit
// is compiled with -fmad=false -prec-div=true -prec-sqrt=true, so no multiply
// and add are fused behind our back: the lists of holes and crystals a ray
// hits are the reference's, bit for bit.  Where a value (not a decision) has
// a better-conditioned form, the better form is used and says so.
#pragma once

#include <cmath>

#include <cuda_runtime.h>

// Host and device: the kernels use these, and host-side checks of the
// kernels' arithmetic call the same code.
#ifndef SM_HD
#define SM_HD __host__ __device__ __forceinline__
#endif

namespace smb {

struct Vec3 {
    float x, y, z;
};

struct Box3 {
    float x1, y1, z1, x2, y2, z2;
};

// The hardware's approximate reciprocal and reciprocal square root.  Subnormal operands
// count as zero: nothing here divides by or takes the root of one (lengths are at least a
// rounding of the coordinates, or exactly zero), and the forms that keep subnormals spend
// three more instructions on rescaling.
SM_HD float fast_rcp(float d) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
#else
    return 1.0f / d;
#endif
}

SM_HD float fast_rsqrt(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / std::sqrt(x);
#endif
}

// Entry/exit parameters of one slab for a segment parameterised by length
// t_total (PESysMatGen.cu:57-64 and every slab of :19-151).
SM_HD void slab_pair(float a_in, float a_out, float lo, float hi, float t_total, float& t_lo,
                                          float& t_hi) {
    float inv = t_total / (a_out - a_in);
    if (inv < 0.0f) {
        t_lo = (hi - a_in) * inv;
        t_hi = (lo - a_in) * inv;
    } else {
        t_hi = (hi - a_in) * inv;
        t_lo = (lo - a_in) * inv;
    }
}

// Intersection of two slabs; false when they are disjoint.
SM_HD bool slab_2d(float a_in, float a_out, float a_lo, float a_hi, float b_in, float b_out,
                                        float b_lo, float b_hi, float t_total, float& tmin, float& tmax) {
    float ta0, ta1, tb0, tb1;
    slab_pair(a_in, a_out, a_lo, a_hi, t_total, ta0, ta1);
    slab_pair(b_in, b_out, b_lo, b_hi, t_total, tb0, tb1);
    if ((ta0 > tb1) || (tb0 > ta1)) return false;
    tmin = (tb0 > ta0) ? tb0 : ta0;
    tmax = (tb1 < ta1) ? tb1 : ta1;
    return true;
}

// Slab entry/exit of the segment a -> b (after its degenerate cases).
// Returns 0 for "no overlap", 1 for an overlap [tmin, tmax] of a segment of
// length t_total; the axis-degenerate answers (a full box side) come back as
// code 2 with the length in tmax.
SM_HD int slab_segment(float xi, float yi, float zi, float xo, float yo, float zo, const Box3& b,
                                            bool inside_variant, float& tmin, float& tmax, float& t_total) {
    const float eps = 0.001f;
    bool cx = fabsf(xo - xi) < eps, cy = fabsf(yo - yi) < eps, cz = fabsf(zo - zi) < eps;
    if (cx & cy & cz) return 0;
    if (cx & cy) {  // along z
        if ((xi >= b.x1 & xi <= b.x2) & (yi >= b.y1 & yi <= b.y2)) {
            if (!inside_variant) {
                if ((zi <= b.z1 & zo >= b.z2) || (zo <= b.z1 & zi >= b.z2)) { tmax = fabsf(b.z2 - b.z1); return 2; }
            } else {
                if (zi < zo) { tmax = zo - b.z1; return 2; }
                if (zi > zo) { tmax = b.z2 - zo; return 2; }
            }
        }
        return 0;
    }
    if (cz & cy) {  // along x
        if ((zi >= b.z1 & zi <= b.z2) & (yi >= b.y1 & yi <= b.y2)) {
            if (!inside_variant) {
                if ((xi <= b.x1 & xo >= b.x2) || (xo <= b.x1 & xi >= b.x2)) { tmax = fabsf(b.x2 - b.x1); return 2; }
            } else {
                if (xi < xo) { tmax = xo - b.x1; return 2; }
                if (xi > xo) { tmax = b.x2 - xo; return 2; }
            }
        }
        return 0;
    }
    if (cx & cz) {  // along y
        if ((xi >= b.x1 & xi <= b.x2) & (zi >= b.z1 & zi <= b.z2)) {
            if (!inside_variant) {
                if ((yi <= b.y1 & yo >= b.y2) || (yo <= b.y1 & yi >= b.y2)) { tmax = fabsf(b.y2 - b.y1); return 2; }
            } else {
                if (yi < yo) { tmax = yo - b.y1; return 2; }
                if (yi > yo) { tmax = b.y2 - yo; return 2; }
            }
        }
        return 0;
    }
    if (cx) {  // plane x = const: slabs y, z
        if (xi >= b.x2 || xi <= b.x1) return 0;
        t_total = sqrtf((yo - yi) * (yo - yi) + (zo - zi) * (zo - zi));
        return slab_2d(yi, yo, b.y1, b.y2, zi, zo, b.z1, b.z2, t_total, tmin, tmax) ? 1 : 0;
    }
    if (cy) {  // plane y = const: slabs x, z
        if (yi >= b.y2 || yi <= b.y1) return 0;
        t_total = sqrtf((xo - xi) * (xo - xi) + (zo - zi) * (zo - zi));
        return slab_2d(xi, xo, b.x1, b.x2, zi, zo, b.z1, b.z2, t_total, tmin, tmax) ? 1 : 0;
    }
    if (cz) {  // plane z = const: slabs x, y
        if (zi >= b.z2 || zi <= b.z1) return 0;
        t_total = sqrtf((xo - xi) * (xo - xi) + (yo - yi) * (yo - yi));
        return slab_2d(xi, xo, b.x1, b.x2, yi, yo, b.y1, b.y2, t_total, tmin, tmax) ? 1 : 0;
    }
    t_total = sqrtf((xo - xi) * (xo - xi) + (yo - yi) * (yo - yi) + (zo - zi) * (zo - zi));
    if (!slab_2d(xi, xo, b.x1, b.x2, yi, yo, b.y1, b.y2, t_total, tmin, tmax)) return 0;
    float tz0, tz1;
    slab_pair(zi, zo, b.z1, b.z2, t_total, tz0, tz1);
    if ((tmin > tz1) || (tz0 > tmax)) return 0;
    if (tz0 > tmin) tmin = tz0;
    if (tz1 < tmax) tmax = tz1;
    return 1;
}

// Chord of segment a -> b through box, counted only if the segment enters and
// leaves strictly inside (PESysMatGen.cu:19-151).
SM_HD float chord_through(float xi, float yi, float zi, float xo, float yo, float zo,
                                               const Box3& b) {
    const float eps = 0.001f;
    float tmin = 0.0f, tmax = 0.0f, t_total = 0.0f;
    int code = slab_segment(xi, yi, zi, xo, yo, zo, b, false, tmin, tmax, t_total);
    if (code == 0) return 0.0f;
    if (code == 2) return tmax;
    if ((tmax - tmin) < eps) return 0.0f;
    if (tmin >= t_total || tmax >= t_total) return 0.0f;
    if (tmin <= eps || tmax <= eps) return 0.0f;
    return tmax - tmin;
}

// Chord from the box entry to the end of the segment inside the box
// (PESysMatGen.cu:153-307).
SM_HD float chord_to_end(float xi, float yi, float zi, float xo, float yo, float zo,
                                              const Box3& b) {
    const float eps = 0.001f;
    if (fabsf(yo - yi) < 0.001f) return 0.0f;
    float tmin = 0.0f, tmax = 0.0f, t_total = 0.0f;
    int code = slab_segment(xi, yi, zi, xo, yo, zo, b, true, tmin, tmax, t_total);
    if (code == 0) return 0.0f;
    if (code == 2) return tmax;
    if ((tmax - tmin) < eps) return 0.0f;
    if (tmin >= t_total) return 0.0f;
    if (tmax <= eps) return 0.0f;
    if ((tmax >= t_total) && (tmin > eps)) return t_total - tmin;
    if ((tmin <= eps) && (tmax <= t_total)) return tmax;
    if ((tmin <= eps) && (tmax >= t_total)) return t_total;
    return tmax - tmin;
}

// Chord through a hole: cylinder of radius R, axis parallel to y at (xc, zc),
// between the planes y1 < y2 (PESysMatGen.cu:309-373).  Decisions in single
// precision as the reference; for rays that enter or leave through the wall
// the value t2 - t1 comes from a double-precision discriminant when it is
// small relative to its terms (near-tangent rays), where the single-precision
// difference (kx^2+kz^2)R^2 - (kx z - kz x)^2 cancels.
SM_HD float chord_hole(float xi, float yi, float zi, float xo, float yo, float zo, float xc,
                                            float y1, float y2, float zc, float R) {
    if (fabsf(y1 - y2) < 0.001f) return 0.0f;
    float t_total = sqrtf((xo - xi) * (xo - xi) + (yo - yi) * (yo - yi) + (zo - zi) * (zo - zi));
    float kx = (xo - xi) / t_total, ky = (yo - yi) / t_total, kz = (zo - zi) / t_total;
    float x_a = xi + kx / ky * (y1 - yi), x_b = xi + kx / ky * (y2 - yi);
    float z_a = zi + kz / ky * (y1 - yi), z_b = zi + kz / ky * (y2 - yi);
    float t_a = (y1 - yi) / ky, t_b = (y2 - yi) / ky;
    bool in_a = (x_a - xc) * (x_a - xc) + (z_a - zc) * (z_a - zc) <= R * R;
    bool in_b = (x_b - xc) * (x_b - xc) + (z_b - zc) * (z_b - zc) <= R * R;
    const float tiny = 0.0001f;
    if (in_a && in_b) {
        if (t_a <= tiny || t_b <= tiny) return 0.0f;
        if (t_a >= t_total || t_b >= t_total) return 0.0f;
        return fabsf(t_b - t_a);
    }
    float px = xi - xc, pz = zi - zc;
    float kk = kx * kx + kz * kz;
    float cross = kx * pz - kz * px;
    float disc = kk * R * R - cross * cross;
    if (disc <= 0.00001f) return 0.0f;
    float sq = sqrtf(disc);
    float t1 = (-(kx * px + kz * pz) - sq) / kk;
    float t2 = (-(kx * px + kz * pz) + sq) / kk;
    if (!in_a && !in_b) {
        if (!((t1 >= t_a) && (t2 <= t_b))) return 0.0f;
        if (t2 <= tiny || t1 <= tiny) return 0.0f;
        if (t2 >= t_total || t1 >= t_total) return 0.0f;
    } else if (in_a) {  // enters through the y1 cap, leaves through the wall
        if (t2 <= tiny || t_a <= tiny) return 0.0f;
        if (t2 >= t_total || t_a >= t_total) return 0.0f;
    } else {            // enters through the wall, leaves through the y2 cap
        if (t_b <= tiny || t1 <= tiny) return 0.0f;
        if (t_b >= t_total || t1 >= t_total) return 0.0f;
    }
    // Value (the decision above is unchanged): near-tangent rays get the wall
    // roots from a double-precision discriminant.
    double r1 = t1, r2 = t2;
    if (disc < 0.01f * (kk * R * R)) {
        double kxd = kx, kzd = kz, pxd = px, pzd = pz, Rd = R;
        double kkd = kxd * kxd + kzd * kzd;
        double cr = kxd * pzd - kzd * pxd;
        double dd = kkd * Rd * Rd - cr * cr;
        double s = sqrt(dd > 0.0 ? dd : 0.0);
        double bd = kxd * pxd + kzd * pzd;
        r1 = (-bd - s) / kkd;
        r2 = (-bd + s) / kkd;
    }
    if (!in_a && !in_b) return (float)(r2 - r1);
    if (in_a) return (float)(r2 - (double)t_a);
    return (float)((double)t_b - r1);
}

// ---- chord_through decided without its divisions and square root -----------------
// A segment a -> b prepared once for many boxes: its start, the reciprocal of
// its extent on each axis and their magnitudes, its length.
struct ChordRay {
    float px, py, pz;
    float ix, iy, iz, ax, ay, az;
    float len;
    float margin;   // largest of delta |1/d_i|; infinite unless ok: then nothing is clear to chord_quick
    float eps;      // the reference's 0.001 in units of the segment
    bool ok;        // no axis is near the reference's degenerate extent (0.001)
};

// 1 / d to about one unit in the last place.
SM_HD float chord_rcp(float d) {
    const float r = fast_rcp(d);
    return fmaf(r, fmaf(-d, r, 1.0f), r);
}

SM_HD ChordRay make_chord_ray(float px, float py, float pz, float dx, float dy, float dz, float len,
                             float delta) {
    ChordRay c;
    c.px = px; c.py = py; c.pz = pz;
    c.ix = chord_rcp(dx); c.iy = chord_rcp(dy); c.iz = chord_rcp(dz);
    c.ax = fabsf(c.ix); c.ay = fabsf(c.iy); c.az = fabsf(c.iz);
    c.len = len;
    c.ok = fminf(fminf(fabsf(dx), fabsf(dy)), fabsf(dz)) > 0.002f;
    c.margin = c.ok ? delta * fmaxf(fmaxf(c.ax, c.ay), c.az) : INFINITY;
    c.eps = 0.001f * chord_rcp(len);
    return c;
}

// A segment with one axis below the reference's degenerate extent, which it leaves out
// of the slabs: there the segment stays inside the slab or misses the box.  Makes r fit
// for chord_filter's "no chord" call (a steep reciprocal says the same); false when an
// axis is too near the limit to tell, or two are below it (the reference then counts a
// segment that starts on the box too).
SM_HD bool flatten(ChordRay* r, float dx, float dy, float dz) {
    const float d[3] = {fabsf(dx), fabsf(dy), fabsf(dz)};
    float* inv[3] = {&r->ix, &r->iy, &r->iz};
    float* mag[3] = {&r->ax, &r->ay, &r->az};
    int flat = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (d[a] < 0.0009f) {
            *inv[a] = *mag[a] = 1e9f;
            ++flat;
        } else if (!(d[a] > 0.002f)) return false;
    }
    return flat == 1;
}

// chord_through of the box of half sizes (hx, hy, hz) about (cx, cy, cz), when
// the answer is clear: 1 (the chord, in `chord`), 0 (no chord) or -1 (too
// close to call: chord_through decides).  In units of the segment, axis i of
// the box grown or shrunk by delta is crossed between t_i -+ (h_i +- delta) |1/d_i|;
// `grown` bounds the reference's tmin from below and its tmax from above,
// `shrunk` the other way round, so a condition that both satisfy is the
// reference's.  delta covers the rounding of either form: the boxes' corners
// in the segment's frame (2 units of 2^-24 of the coordinate range S), and the
// slab parameters along the segment (10 units of its length <= S), together
// below 8e-7 S; pe_plan passes 1.5e-6 S.
SM_HD int chord_filter(const ChordRay& r, float cx, float cy, float cz, float hx, float hy, float hz, float delta,
                       float* chord) {
    const float eps = 0.001f;
    const float tx = (cx - r.px) * r.ix, ty = (cy - r.py) * r.iy, tz = (cz - r.pz) * r.iz;
    const float gx = hx + delta, gy = hy + delta, gz = hz + delta;
    const float sx = hx - delta, sy = hy - delta, sz = hz - delta;
    const float lo_g = fmaxf(fmaxf(fmaf(-gx, r.ax, tx), fmaf(-gy, r.ay, ty)), fmaf(-gz, r.az, tz));
    const float hi_g = fminf(fminf(fmaf(gx, r.ax, tx), fmaf(gy, r.ay, ty)), fmaf(gz, r.az, tz));
    const float lo_s = fmaxf(fmaxf(fmaf(-sx, r.ax, tx), fmaf(-sy, r.ay, ty)), fmaf(-sz, r.az, tz));
    const float hi_s = fminf(fminf(fmaf(sx, r.ax, tx), fmaf(sy, r.ay, ty)), fmaf(sz, r.az, tz));
    if ((hi_g - lo_g) * r.len < eps || hi_s > 1.0f || lo_s * r.len < eps) return 0;
    if ((hi_s - lo_s) * r.len > eps && hi_g < 1.0f && lo_g * r.len > eps) {
        const float lo = fmaxf(fmaxf(fmaf(-hx, r.ax, tx), fmaf(-hy, r.ay, ty)), fmaf(-hz, r.az, tz));
        const float hi = fminf(fminf(fmaf(hx, r.ax, tx), fmaf(hy, r.ay, ty)), fmaf(hz, r.az, tz));
        *chord = (hi - lo) * r.len;
        return 1;
    }
    return -1;
}

// The same call with one margin for all axes (the largest of delta |1/d_i|): a
// third of the work, unclear more often for rays nearly parallel to a face.
SM_HD int chord_quick(const ChordRay& r, float cx, float cy, float cz, float hx, float hy, float hz, float* chord) {
    const float tx = (cx - r.px) * r.ix, ty = (cy - r.py) * r.iy, tz = (cz - r.pz) * r.iz;
    const float lo = fmaxf(fmaxf(fmaf(-hx, r.ax, tx), fmaf(-hy, r.ay, ty)), fmaf(-hz, r.az, tz));
    const float hi = fminf(fminf(fmaf(hx, r.ax, tx), fmaf(hy, r.ay, ty)), fmaf(hz, r.az, tz));
    const float w = hi - lo, m = r.margin;
    *chord = w * r.len;
    if (w < r.eps - 2.0f * m || hi > 1.0f + m || lo < r.eps - m) return 0;
    if (w > r.eps + 2.0f * m && hi < 1.0f - m && lo > r.eps + m) return 1;
    return -1;
}

// a / b with rb ~ 1 / b, and sqrt(x), each with one residual correction (Markstein,
// IBM J. Res. Dev. 34 (1990) 111): the correctly rounded result but for about one
// operand in 2^20, without the range checks of the IEEE forms.  For values only.
SM_HD float near_div(float a, float b, float rb) {
    const float q = a * rb;
    return fmaf(fmaf(-q, b, a), rb, q);
}

SM_HD float near_root(float x, float r) {   // r ~ 1 / sqrt(x)
    const float s = x * r;
    return fmaf(fmaf(-s, s, x), 0.5f * r, s);
}

SM_HD float near_sqrt(float x) { return near_root(x, fast_rsqrt(x)); }

// chord_through's own value, operation for operation, for a segment a -> b that a
// filter called a clear chord of the box of half sizes h about the origin; ix, iy,
// iz and inv_len: the reciprocals of its extents and length, to a few units of 2^-24.
SM_HD float chord_value(float xi, float yi, float zi, float xo, float yo, float zo, float hx, float hy, float hz,
                        float ix, float iy, float iz, float inv_len) {
    const float dx = xo - xi, dy = yo - yi, dz = zo - zi;
    const float t = near_root(dx * dx + dy * dy + dz * dz, inv_len);
    const float qx = near_div(t, dx, ix), qy = near_div(t, dy, iy), qz = near_div(t, dz, iz);
    const float x1 = (-hx - xi) * qx, x2 = (hx - xi) * qx, y1 = (-hy - yi) * qy, y2 = (hy - yi) * qy;
    const float z1 = (-hz - zi) * qz, z2 = (hz - zi) * qz;
    return fminf(fminf(fmaxf(x1, x2), fmaxf(y1, y2)), fmaxf(z1, z2)) -
           fmaxf(fmaxf(fminf(x1, x2), fminf(y1, y2)), fminf(z1, z2));
}

// chord_hole of a hole cylinder for a segment that runs towards larger y and
// starts before the hole, when the answer is clear: 1 (the chord), 0 (none) or -1
// (chord_hole decides).  Between the depth planes y1 and y2 the segment moves
// laterally from w (relative to the axis) by e.  Clear calls stay `margin` away
// from the wall at both planes (the reference's points there round by a few
// units of 2^-24 of the coordinates), clear of its end-point tests, above twice
// its floor of the discriminant, and where it takes its roots in single precision
// and a miss is far from a tangent.  The chord is then chord_hole's, operation for
// operation: through tungsten an entry follows it times 3.5 / mm, so another
// form's rounding of 4e-6 mm would show as 1.4e-5 of the entry.
SM_HD int hole_filter(float px, float py, float pz, float dx, float dy, float dz, float inv_dy, float len, float xc,
                      float y1, float y2, float zc, float R, float margin, float* chord) {
    const float l1 = (y1 - py) * inv_dy, l2 = (y2 - py) * inv_dy, dl = l2 - l1;
    const float wx = fmaf(dx, l1, px) - xc, wz = fmaf(dz, l1, pz) - zc;   // from the axis, at the y1 plane
    const float ex = dx * dl, ez = dz * dl;
    const float vx = wx + ex, vz = wz + ez;                               // ... at the y2 plane
    const float ww = fmaf(wx, wx, wz * wz), vv = fmaf(vx, vx, vz * vz);
    const float far2 = (R + margin) * (R + margin), near2 = (R - margin) * (R - margin);
    const float ee = fmaf(ex, ex, ez * ez), we = fmaf(wx, ex, wz * ez);
    const float cr = fmaf(wx, ez, -wz * ex);
    const bool between = we < 0.0f && we > -ee;                           // the nearest point lies between the planes
    if (between ? cr * cr > far2 * ee : fminf(ww, vv) > far2) return 0;
    const bool in_a = ww < near2, in_b = vv < near2;
    if (!(in_a || ww > far2) || !(in_b || vv > far2) || !(R > margin) || !(l1 * len > 0.001f && l2 < 0.9999f) ||
        !(y2 - y1 > 0.01f))
        return -1;
    const float t = near_sqrt(dx * dx + dy * dy + dz * dz), rt = chord_rcp(t);
    const float ky = near_div(dy, t, rt), rk = chord_rcp(ky);
    const float t_a = near_div(y1 - py, ky, rk), t_b = near_div(y2 - py, ky, rk);
    if (in_a && in_b) {
        *chord = fabsf(t_b - t_a);
        return 1;
    }
    const float kx = near_div(dx, t, rt), kz = near_div(dz, t, rt);
    const float qx = px - xc, qz = pz - zc;
    const float kk = kx * kx + kz * kz;
    const float cross = kx * qz - kz * qx;
    const float full = kk * R * R, disc = full - cross * cross;
    if (!(disc > 0.05f * full) || !(disc > 2e-5f)) return -1;
    const float sq = near_sqrt(disc), rkk = chord_rcp(kk), b = -(kx * qx + kz * qz);
    const float t1 = near_div(b - sq, kk, rkk), t2 = near_div(b + sq, kk, rkk);
    *chord = in_a ? t2 - t_a : (in_b ? t_b - t1 : t2 - t1);
    return 1;
}

}  // namespace smb
