// Primary-Compton scatter kernels for sm_100a (see scatter.h for the split).
//
// Physics per (detector d, voxel I, scatter point S), as the reference's
// crystalScatterSysMatCuda / collimatorScatterSysMatCuda
// (ScatterGen_RayTracing_CircularHole/scatter.cu:1077-1437, :1544-1936):
//   W(S, I) * RangePhi / 2pi * KNfraction(theta_min, theta_max) * P_window(E')
//     * exp(-sum_k mu_k(E') L_k - mu_d(E') L_self) * (1 - exp(-mu_d(E') L_abs)) mu_pe,d(E') / mu_d(E')
// with E' = E0 / (1 + alpha (1 - cos theta)), theta the angle at S between
// I -> S and S -> D, mu_pe(E') = mu_pe (E0/E')^3, mu_c(E') = mu_c E0/E'.
// W is PE[s, I] mu_c,d / mu_pe,d (crystal scatter) or the virtual solid angle
// of the hole times mu_c / mu_t of plate 0 (collimator scatter).
//
// Differences in arithmetic (not in the quantities): the cosine and sine of
// the scatter angle come from a dot and a cross product instead of
// cos(acos(.)), the polar range from atan2 of the extreme unit-box corners
// instead of eight acos, and the reference's 0.01 rad rectangle sum of the
// Klein-Nishina integrand (up to 315 terms) from a closed form: the
// Euler-Maclaurin formula with the exact integral (a Taylor table of
// g = KN sin theta, built in double on the host) and its first two
// correction terms, whose remainder is below 1e-10.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "scatter.h"
#include "scatter_term.cuh"
#include "tracer.cuh"

namespace smb {
namespace {


// ---- bitmaps (scatter.cu:1440-1540, :1939-2009) ------------------------------
// Single-precision expressions in the reference's order; this translation
// unit is compiled without fused multiply-add, so every bit matches.
__device__ __forceinline__ float dist3(float x1, float y1, float z1, float x2, float y2, float z2) {
    return sqrtf((x1 - x2) * (x1 - x2) + (y1 - y2) * (y1 - y2) + (z1 - z2) * (z1 - z2));
}

__device__ __noinline__ bool crystal_bit(const float4* cr, int i, int j, int k) {
    const float4 a = cr[i], b = cr[j], c = cr[k];
    const float Lij = dist3(a.x, a.y, a.z, b.x, b.y, b.z);
    const float crit_ij = a.w / Lij, crit_ji = b.w / Lij;
    const float ex_ij = (a.x - b.x) / Lij, ey_ij = (a.y - b.y) / Lij, ez_ij = (a.z - b.z) / Lij;
    const float ex_ji = (b.x - a.x) / Lij, ey_ji = (b.y - a.y) / Lij, ez_ji = (b.z - a.z) / Lij;
    const float Lik = dist3(c.x, c.y, c.z, a.x, a.y, a.z);
    const float crit_ki = c.w / Lik;
    const float Ljk = dist3(c.x, c.y, c.z, b.x, b.y, b.z);
    const float crit_kj = c.w / Ljk;
    const float ex_ki = (c.x - a.x) / Lik, ey_ki = (c.y - a.y) / Lik, ez_ki = (c.z - a.z) / Lik;
    const float ex_kj = (c.x - b.x) / Ljk, ey_kj = (c.y - b.y) / Ljk, ez_kj = (c.z - b.z) / Ljk;
    if (dist3(ex_ki, ey_ki, ez_ki, ex_ji, ey_ji, ez_ji) <= crit_ki + crit_ji) return true;
    return dist3(ex_kj, ey_kj, ez_kj, ex_ij, ey_ij, ez_ij) <= crit_kj + crit_ij;
}

__device__ __noinline__ bool collimator_bit(const float4* cr, const float4* hr, int i, int j, int k) {
    const float4 h = hr[i], b = cr[j], c = cr[k];
    const float Lij = dist3(h.x, h.y, h.z, b.x, b.y, b.z);
    const float crit_ji = b.w / Lij;
    const float ex_ji = (b.x - h.x) / Lij, ey_ji = (b.y - h.y) / Lij, ez_ji = (b.z - h.z) / Lij;
    const float Lik = dist3(c.x, c.y, c.z, h.x, h.y, h.z);
    const float crit_ki = c.w / Lik;
    const float ex_ki = (c.x - h.x) / Lik, ey_ki = (c.y - h.y) / Lik, ez_ki = (c.z - h.z) / Lik;
    return dist3(ex_ki, ey_ki, ez_ki, ex_ji, ey_ji, ez_ji) <= crit_ki + crit_ji;
}

// Pair index (i <= j) -> i: the largest i with i*N - i*(i-1)/2 <= pair.
__device__ __forceinline__ int pair_row(long long pair, int N) {
    const double b = 2.0 * N + 1.0;
    int i = (int)((b - sqrt(b * b - 8.0 * (double)pair)) * 0.5);
    if (i < 0) i = 0;
    auto start = [N](long long r) { return r * N - r * (r - 1) / 2; };
    while (i > 0 && start(i) > pair) --i;
    while (i + 1 < N && start(i + 1) <= pair) ++i;
    return i;
}

// The cone test |u_k - u_axis| <= R_k / |k - a| + c (u_k, u_axis unit vectors from a) by
// squares with one reciprocal square root: 1 yes, 0 no, -1 too close to call.  The
// squared distance 2 - 2 cos is good to 2e-6 and the right side to 1e-6 of itself, the
// band is five times that and more.
__device__ __forceinline__ int cone_quick(const float4& k, float ax, float ay, float az, float ux, float uy, float uz,
                                          float c) {
    const float dx = k.x - ax, dy = k.y - ay, dz = k.z - az;
    const float inv = fast_rsqrt(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
    const float cosine = fmaf(dx, ux, fmaf(dy, uy, dz * uz)) * inv;
    const float rhs = fmaf(k.w, inv, c), r2 = rhs * rhs;
    const float diff = fmaf(-2.0f, cosine, 2.0f) - r2, band = fmaf(1e-4f, r2, 1e-5f);
    return diff < -band ? 1 : (diff > band ? 0 : -1);
}

// The line between crystal (or hole) a and crystal b as the bitmaps' cone tests see it.
struct PairAxis {
    float4 a, b;
    float ux, uy, uz;            // unit vector a -> b
    float ca, cb;                // R_b / |ab|, R_a / |ab|
};

__device__ __forceinline__ PairAxis pair_axis(const float4& a, const float4& b) {
    PairAxis p;
    p.a = a;
    p.b = b;
    p.ux = b.x - a.x;
    p.uy = b.y - a.y;
    p.uz = b.z - a.z;
    const float inv = fast_rsqrt(fmaf(p.ux, p.ux, fmaf(p.uy, p.uy, p.uz * p.uz)));
    p.ux *= inv;
    p.uy *= inv;
    p.uz *= inv;
    p.ca = b.w * inv;
    p.cb = a.w * inv;
    return p;
}

// The bitmap's bit of (i, j, k), i < j crystals or i hole, j crystal; p = pair_axis of i and j.
template <int KIND>
__device__ __forceinline__ bool pair_bit(const ScatterTables& T, const PairAxis& p, int i, int j, int k) {
    const float4 c = T.crystal_raw[k];
    int f = cone_quick(c, p.a.x, p.a.y, p.a.z, p.ux, p.uy, p.uz, p.ca);                   // seen from i
    if (KIND == kScatterCrystal) {
        if (f != 1) {
            const int g = cone_quick(c, p.b.x, p.b.y, p.b.z, -p.ux, -p.uy, -p.uz, p.cb);   // seen from j
            f = g == 1 ? 1 : (f | g);                                                     // -1 when either is unclear
        }
        return f < 0 ? crystal_bit(T.crystal_raw, i, j, k) : f == 1;
    }
    return f < 0 ? collimator_bit(T.crystal_raw, T.hole_raw, i, j, k) : f == 1;
}

// Bitmap words: lane = bit, so a warp's loads of the crystals k are consecutive; each
// lane keeps the word of its own turn and 32 words are stored together.  A bit is
// decided by cone_quick and, when that cannot call, by the reference's expression
// (about 500 instructions: every bit took it before, 59.5 ms for 2048 crystals).
// Crystal pairs: bit = (i N - i (i + 1) / 2 + j) N + k, i <= j; set for i < j, k != i, j.
// Collimator: bit = i N^2 + j N + k for layer-0 hole i, crystals j, k.
template <int KIND>
__global__ void __launch_bounds__(256) bitmap_kernel(uint32_t* __restrict__ words, long long n_words, ScatterTables T) {
    const int N = T.n_crystals, lane = threadIdx.x & 31;
    const long long total = KIND == kScatterCrystal ? ((long long)N * (N + 1) / 2) * N : (long long)T.n_holes0 * N * N;
    const long long n_groups = (n_words + 31) / 32;
    long long pair = -1;
    int i = 0, j = 0;
    PairAxis axis{};
    for (long long g = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; g < n_groups;
         g += ((long long)gridDim.x * blockDim.x) >> 5) {
        long long next = g * 1024 + lane;              // this lane's bit of the group's first word
        long long at = next / N;
        int k = (int)(next - at * N);
        uint32_t mine = 0u;
        for (int w = 0; w < 32; ++w, next += 32, k += 32) {
            while (k >= N) {
                k -= N;
                ++at;
            }
            bool set = false;
            if (next < total) {
                if (at != pair) {
                    pair = at;
                    if (KIND == kScatterCrystal) {
                        i = pair_row(pair, N);
                        j = (int)(pair - ((long long)i * N - (long long)i * (i - 1) / 2)) + i;
                    } else {
                        i = (int)(pair / N);
                        j = (int)(pair - (long long)i * N);
                    }
                    axis = pair_axis(KIND == kScatterCrystal ? T.crystal_raw[i] : T.hole_raw[i], T.crystal_raw[j]);
                }
                if (KIND != kScatterCrystal || (i < j && k != i && k != j)) set = pair_bit<KIND>(T, axis, i, j, k);
            }
            const uint32_t word = __ballot_sync(0xffffffffu, set);
            if (w == lane) mine = word;
        }
        if (g * 32 + lane < n_words) words[g * 32 + lane] = mine;
    }
}

// ---- per (scatter point, detector) ---------------------------------------------
// sum_k L_k mu_pe_k, sum_k L_k mu_c_k over the crystals k the bitmap flags for
// the pair (scatter.cu:1309-1367, :1832-1889), the path inside the detecting
// crystal before its unit (:1371-1382), and the absorption chord (:1385-1392).
// The detector unit is the whole crystal (the reference's divide = 1), whose
// centre is the crystal centre.
// A warp takes 32 neighbouring detectors and one scatter point S.  The crystals their
// segments can meet are those whose box meets the hull of S and the detectors' box B, the
// union of the boxes S + l (B - S), l in [0, 1]: every face gives a bound on l, and the
// test is whether the bounds leave any (lane = crystal, 32 at a time, boxes grown by
// 0.01 mm).  The survivors, some dozens of thousands, are walked by all lanes, each with
// its own segment: chord_quick drops the uncrossed ones, crossed ones take
// chord_through's value if the bitmap flags them - read from a given bitmap, or decided
// here for the crossed crystal alone, without building the N^3 / 2 bits (walking the
// flagged crystals of a computed bitmap took 24.7 ms for 2048 x 2048 pairs).
template <int KIND>
__global__ void __launch_bounds__(128) scatter_pair_kernel(const __grid_constant__ DevGeometry G,
                                                           const __grid_constant__ ScatterTables T,
                                                           const uint32_t* __restrict__ bitmap,
                                                           const int* __restrict__ perm, int r0, int r1,
                                                           float4* __restrict__ pair, int n_sources) {
    const int N = T.n_crystals;
    const int r = r0 + blockIdx.x * blockDim.x + threadIdx.x;
    const int d = perm[min(r, r1 - 1)];
    const long long ld = r1 - r0;
    const float4 Dp = G.c.pos[d], Dsz = G.c.size[d], Dr = G.c.rot[d];
    const int lane = threadIdx.x & 31;
    Box3 B{Dp.x, Dp.y, Dp.z, Dp.x, Dp.y, Dp.z};          // of the warp's detector centres
    for (int o = 16; o > 0; o >>= 1) {
        B.x1 = fminf(B.x1, __shfl_xor_sync(0xffffffffu, B.x1, o));
        B.y1 = fminf(B.y1, __shfl_xor_sync(0xffffffffu, B.y1, o));
        B.z1 = fminf(B.z1, __shfl_xor_sync(0xffffffffu, B.z1, o));
        B.x2 = fmaxf(B.x2, __shfl_xor_sync(0xffffffffu, B.x2, o));
        B.y2 = fmaxf(B.y2, __shfl_xor_sync(0xffffffffu, B.y2, o));
        B.z2 = fmaxf(B.z2, __shfl_xor_sync(0xffffffffu, B.z2, o));
    }
    for (int q = blockIdx.y; q < n_sources; q += gridDim.y) {
        float4 S;
        int s;
        if (KIND == kScatterCrystal) {
            S = T.crystal_src[q];
            s = q / T.n_points;
        } else {
            S = T.hole_src[q];
            s = q;
        }
        const bool on = r < r1 && !(KIND == kScatterCrystal && s == d);
        long long base;
        if (KIND == kScatterCrystal) {
            const int lo = s < d ? s : d, hi = s < d ? d : s;
            base = ((long long)lo * N - (long long)lo * (lo + 1) / 2 + hi) * N;
        } else {
            base = ((long long)s * N + d) * N;
        }
        const float dx = Dp.x - S.x, dy = Dp.y - S.y, dz = Dp.z - S.z;
        const float len2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz)), inv_len = fast_rsqrt(len2);
        ChordRay cr = make_chord_ray(S.x, S.y, S.z, dx, dy, dz, len2 * inv_len, T.chord_delta);
        const bool flat = !cr.ok && flatten(&cr, dx, dy, dz);   // source and detector in one layer, row or column
        PairAxis axis{};
        int pi = s, pj = d;
        if (!bitmap) {
            if (KIND == kScatterCrystal) {
                pi = min(s, d);
                pj = max(s, d);
            }
            axis = pair_axis(KIND == kScatterCrystal ? T.crystal_raw[pi] : T.hole_raw[pi], T.crystal_raw[pj]);
        }
        // bounds on l: l * face >= gap (face > 0: from below, < 0: from above)
        const float face[6] = {B.x2 - S.x, B.y2 - S.y, B.z2 - S.z, S.x - B.x1, S.y - B.y1, S.z - B.z1};
        float inv_face[6];
#pragma unroll
        for (int a = 0; a < 6; ++a) inv_face[a] = fabsf(face[a]) > 1e-4f ? fast_rcp(face[a]) : 0.0f;
        float a_pe = 0.0f, a_c = 0.0f;
        for (int k0 = 0; k0 < N; k0 += 32) {
            bool meets = false;
            if (k0 + lane < N) {
                const float4 lo = __ldg(G.c.lo + k0 + lane), hi = __ldg(G.c.hi + k0 + lane);
                const float m = 0.01f;
                const float gap[6] = {lo.x - m - S.x, lo.y - m - S.y, lo.z - m - S.z, S.x - hi.x - m, S.y - hi.y - m, S.z - hi.z - m};
                float from = 0.0f, to = 1.0f;
                bool empty = false;
#pragma unroll
                for (int a = 0; a < 6; ++a) {
                    const float l = gap[a] * inv_face[a];
                    if (face[a] > 1e-4f) from = fmaxf(from, l);
                    else if (face[a] < -1e-4f) to = fminf(to, l);
                    else empty |= gap[a] > 1e-4f;
                }
                meets = !empty && from <= to;
            }
            uint32_t any = __ballot_sync(0xffffffffu, meets);
            if (!any) continue;
            // which of them this lane's pair counts
            uint32_t bits = on ? 0xffffffffu : 0u;
            if (on && bitmap) {
                const long long bit = base + k0, w = bit >> 5;
                const int sh = (int)(bit & 31);
                const uint32_t lo = __ldg(bitmap + w), hi = sh && (w << 5) + 32 < base + N ? __ldg(bitmap + w + 1) : 0u;
                bits = __funnelshift_r(lo, hi, sh);
            }
            if ((d & ~31) == k0) bits &= ~(1u << (d & 31));
            if (KIND == kScatterCrystal && (s & ~31) == k0) bits &= ~(1u << (s & 31));
            while (any) {
                const int b = __ffs(any) - 1, k = k0 + b;
                any &= any - 1u;
                const float4 kp = __ldg(G.c.pos + k), ks = __ldg(G.c.size + k), kr = __ldg(G.c.rot + k);
                if (!(bits >> b & 1u)) continue;
                const float hx = 0.5f * ks.x, hy = 0.5f * ks.y, hz = 0.5f * ks.z;
                const float xa = (S.x - kp.x) * kr.x - (S.z - kp.z) * kr.y;
                const float ya = S.y - kp.y;
                const float za = (S.x - kp.x) * kr.y + (S.z - kp.z) * kr.x;
                const float xb = (Dp.x - kp.x) * kr.x - (Dp.z - kp.z) * kr.y;
                const float yb = Dp.y - kp.y;
                const float zb = (Dp.x - kp.x) * kr.y + (Dp.z - kp.z) * kr.x;
                ChordRay c = cr;
                c.px = xa;
                c.py = ya;
                c.pz = za;
                if (kr.x != 1.0f || kr.y != 0.0f)
                    c = make_chord_ray(xa, ya, za, fmaf(dx, kr.x, -dz * kr.y), dy, fmaf(dx, kr.y, dz * kr.x), cr.len,
                                       2.0f * T.chord_delta);
                float chord;
                int f = -1;
                if (c.ok && cr.ok) f = chord_quick(c, 0.0f, 0.0f, 0.0f, hx, hy, hz, &chord);
                else if (flat && kr.x == 1.0f && kr.y == 0.0f)
                    f = chord_filter(c, 0.0f, 0.0f, 0.0f, hx, hy, hz, T.chord_delta, &chord) == 0 ? 0 : -1;
                if (f == 0) continue;
                const float len = f > 0 ? chord_value(xa, ya, za, xb, yb, zb, hx, hy, hz, c.ix, c.iy, c.iz, inv_len)
                                        : chord_through(xa, ya, za, xb, yb, zb, Box3{-hx, -hy, -hz, hx, hy, hz});
                if (len == 0.0f || (!bitmap && !pair_bit<KIND>(T, axis, pi, pj, k))) continue;
                const float4 kph = __ldg(G.c.phys + k);
                a_pe += len * kph.x;
                a_c += len * kph.y;
            }
        }
        float4 out = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (on) {
            // scatter point in the detecting crystal's frame
            const float xs = (S.x - Dp.x) * Dr.x - (S.z - Dp.z) * Dr.y;
            const float ys = S.y - Dp.y;
            const float zs = (S.x - Dp.x) * Dr.y + (S.z - Dp.z) * Dr.x;
            const Box3 cb{-Dsz.x / 2.0f, -Dsz.y / 2.0f, -Dsz.z / 2.0f, Dsz.x / 2.0f, Dsz.y / 2.0f, Dsz.z / 2.0f};
            const Box3 ub{-0.5f * Dsz.x, -0.5f * Dsz.y, -0.5f * Dsz.z, 0.5f * Dsz.x, 0.5f * Dsz.y, 0.5f * Dsz.z};
            const float l1 = chord_to_end(xs, ys, zs, 0.0f, 0.0f, 0.0f, cb);
            const float l2 = chord_to_end(xs, ys, zs, 0.0f, 0.0f, 0.0f, ub);
            const float L = dist3(S.x, S.y, S.z, Dp.x, Dp.y, Dp.z);
            const float xt = 0.0f + 1000.0f * (0.0f - xs) / L;
            const float yt = 0.0f + 1000.0f * (0.0f - ys) / L;
            const float zt = 0.0f + 1000.0f * (0.0f - zs) / L;
            const float labs = chord_through(xs, ys, zs, xt, yt, zt, ub);
            out = make_float4(a_pe, a_c, l1 - l2, labs);
        }
        if (r < r1) pair[(long long)q * ld + (r - r0)] = out;
    }
}

// Column xx (0..7) of brick b: its (x, z), first y and whether it exists.
struct BrickCol {
    int x, z, y0, ci;            // ci: index in the column list (column mode)
    bool valid;
};

__device__ __forceinline__ BrickCol brick_column(const ScatterParams& P, int b, int xx) {
    BrickCol c;
    if (P.cols) {
        const int cg = b % P.bricks_x, by = b / P.bricks_x;
        c.ci = cg * kScBrickX + xx;
        c.valid = c.ci < P.n_cols;
        const int2 xz = c.valid ? P.cols[c.ci] : make_int2(0, 0);
        c.x = xz.x;
        c.z = xz.y;
        c.y0 = by * kScBrickY;
    } else {
        const int bx = b % P.bricks_x, by = (b / P.bricks_x) % P.bricks_y, bz = b / (P.bricks_x * P.bricks_y);
        c.x = bx * kScBrickX + xx;
        c.z = bz;
        c.y0 = by * kScBrickY;
        c.ci = 0;
        c.valid = c.x < P.nx;
    }
    return c;
}

// ---- sources with PE != 0 per voxel brick -----------------------------------------
__global__ void brick_sources_kernel(ScatterParams P, int N, uint32_t* __restrict__ out) {
    const int b = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = blockIdx.y * kScWarps + warp;
    if (s >= N) return;
    const BrickCol bc = brick_column(P, b, lane & 7);
    bool any = false;
    for (int it = 0; it < kScBrickY / 4; ++it) {
        const int y = bc.y0 + it * 4 + (lane >> 3);
        if (bc.valid && y < P.ny) {
            const long long v = (long long)bc.x + (long long)P.nx * (y + (long long)P.ny * bc.z);
            any |= __ldg(P.pe + (long long)s * P.ld_pe + v) != 0.0f;
        }
    }
    if (__any_sync(0xffffffffu, any) && lane == 0) atomicOr(out + (long long)b * P.src_words + (s >> 5), 1u << (s & 31));
}

// Detecting crystal d: geometry, energy window, switch (scatter.cu:1189-1205);
// returns the per-detector factor of the kind (mu_c / mu_pe / points, or plate mu_c / mu_t).
template <int KIND>
__device__ __forceinline__ float setup_det(const ScatterParams& P, const DevGeometry& G, const ScatterTables& T, int d,
                                           Det& D) {
    const float4 pos = G.c.pos[d], sz = G.c.size[d], rt = G.c.rot[d], ph = G.c.phys[d];
    D.x = pos.x; D.y = pos.y; D.z = pos.z; D.cm = rt.x; D.sm = rt.y;
    D.hw = 0.5f * sz.x; D.ht = 0.5f * sz.y; D.hh = 0.5f * sz.z;
    D.r_unit = sqrtf(sz.x * sz.x / 1.0f / 1.0f + sz.z * sz.z / 1.0f / 1.0f + sz.y * sz.y / 1.0f / 1.0f) / 2.0f;
    D.mu_pe = ph.x; D.mu_c = ph.y; D.res = ph.z;
    if (P.same_window > 0) { D.lo = P.win_lo; D.hi = P.win_hi; }
    else {
        D.lo = (1.0f - D.res / 2.0f) * P.e0;
        D.hi = (1.0f + D.res / 2.0f) * P.e0;
    }
    D.on = P.use_compton == 1 && pos.w > 0.01f;   // (scatter.cu:1203-1205)
    D.c_cut = window_cos_cut(P.e0, P.alpha, D.res, D.lo);
    return KIND == kScatterCrystal ? D.mu_c / D.mu_pe / (float)T.n_points : P.plate_c_over_t;
}

// Voxel centre (world) of fractional voxel indices: FOV shift and image rotation (scatter.cu:1172-1184).
__device__ __forceinline__ float3 voxel_world(const ScatterParams& P, float x, float y, float z) {
    float xi = (x - (float)P.nx / 2.0f + 0.5f) * P.vx;
    float yi = (y - (float)P.ny / 2.0f + 0.5f) * P.vy;
    float zi = (z - (float)P.nz / 2.0f + 0.5f) * P.vz;
    xi = xi + P.shx;
    yi = yi + P.shy;
    zi = zi + P.shz;
    return make_float3(xi * P.cos_a - yi * P.sin_a, xi * P.sin_a + yi * P.cos_a, zi);
}

// ---- transfer of arrival points per source ------------------------------------------
// K[a][r][s] = scale_d * sum_p term(vbar[a][s], s_p, d) for d = perm[r] and anchor a:
// the crystal-scatter sysmat entry per unit PE of source s with every photon
// arriving from vbar[a][s] (fractional voxel indices; w <= 0: source unused).
// Thread = rank (coalesced pair reads), grid.y = source; the source point and
// its pair sums are set up once for all anchors.
constexpr int kMaxAnchorsPerPass = 8;

template <typename KT>
__global__ void scatter_transfer_kernel(ScatterParams P, DevGeometry G, ScatterTables T, const float4* __restrict__ vbar,
                                        int n_anchors, KT* __restrict__ K, long long ldk, long long anchor_stride) {
    __shared__ KnNode kn[kKnNodes + 1];
    for (int i = threadIdx.x; i < kKnNodes + 1; i += blockDim.x) kn[i] = T.kn[i];
    __syncthreads();
    const int rank = P.rank0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (rank >= P.rank1) return;
    const int d = P.perm[rank];
    Det D;
    const float scale = setup_det<kScatterCrystal>(P, G, T, d, D);
    for (int s = blockIdx.y; s < T.n_crystals; s += gridDim.y) {
        for (int a0 = 0; a0 < n_anchors; a0 += kMaxAnchorsPerPass) {
            const int na = min(kMaxAnchorsPerPass, n_anchors - a0);
            float acc[kMaxAnchorsPerPass];
            float3 I[kMaxAnchorsPerPass], Is[kMaxAnchorsPerPass];
            bool use[kMaxAnchorsPerPass];
#pragma unroll
            for (int j = 0; j < kMaxAnchorsPerPass; ++j) {
                acc[j] = 0.0f;
                use[j] = false;
                if (j < na) {
                    const float4 vb = vbar[(long long)(a0 + j) * T.n_crystals + s];
                    use[j] = D.on && s != d && vb.w > 0.0f;
                    I[j] = voxel_world(P, vb.x, vb.y, vb.z);
                    Is[j] = make_float3((I[j].x - D.x) * D.cm - (I[j].z - D.z) * D.sm, I[j].y - D.y,
                                        (I[j].x - D.x) * D.sm + (I[j].z - D.z) * D.cm);
                }
            }
            bool any = false;
#pragma unroll
            for (int j = 0; j < kMaxAnchorsPerPass; ++j) any |= use[j];
            if (any) {
                for (int p = 0; p < T.n_points; ++p) {
                    const int q = s * T.n_points + p;
                    Src C;
                    make_src_basic(D, T.crystal_src[q], C);
                    make_src_rest(D, P.pair[(long long)q * P.pair_ld + (P.pair_col ? P.pair_col[rank] : rank - P.pair_r0)], C);
#pragma unroll
                    for (int j = 0; j < kMaxAnchorsPerPass; ++j)
                        if (use[j])
                            acc[j] += scatter_term<false>(P, D, C, kn, nullptr, T.kn_inv_norm, I[j].x, I[j].y, I[j].z, Is[j].x, Is[j].y,
                                                   Is[j].z);
                }
            }
#pragma unroll
            for (int j = 0; j < kMaxAnchorsPerPass; ++j)
                if (j < na) K[(long long)(a0 + j) * anchor_stride + (long long)(rank - P.rank0) * ldk + s] = (KT)(acc[j] * scale);
        }
    }
}

// Same values as scatter_transfer_kernel, arranged for memory traffic: a CTA
// takes 16 detectors (ranks) x 8 sources, stages the pair sums of that tile
// once in shared memory (instead of reading them again for every pass of 8
// anchors), and each detector's 8 consecutive sources are stored together
// (a run of 16 or 32 bytes instead of one sector per lane).  Up to 16 scatter
// points per crystal.
constexpr int kTrRanks = 16, kTrSrcs = 8, kTrMaxPoints = 16;

struct __align__(16) TrSmem {
    KnNode kn[kKnNodes + 1];
    float4 pr[kTrMaxPoints][kTrRanks][kTrSrcs];   // pair sums of the tile: [point][detector][source]
};

template <typename KT>
__global__ void __launch_bounds__(kTrRanks * kTrSrcs) scatter_transfer_tiled_kernel(
    ScatterParams P, DevGeometry G, ScatterTables T, const float4* __restrict__ vbar, int n_anchors,
    KT* __restrict__ K, long long ldk, long long anchor_stride) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TrSmem& S = *reinterpret_cast<TrSmem*>(smem_raw);
    KnNode* kn = S.kn;
    auto& pr = S.pr;
    const int tid = threadIdx.x, rl = tid / kTrSrcs, sl = tid % kTrSrcs;
    const int r0 = P.rank0 + blockIdx.x * kTrRanks, s0 = blockIdx.y * kTrSrcs;
    const int np = T.n_points;
    for (int i = tid; i < kKnNodes + 1; i += blockDim.x) kn[i] = T.kn[i];
    for (int i = tid; i < np * kTrSrcs * kTrRanks; i += blockDim.x) {
        const int r = i % kTrRanks, ss = (i / kTrRanks) % kTrSrcs, p = i / (kTrRanks * kTrSrcs);
        const int rank = r0 + r, src = s0 + ss;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (rank < P.rank1 && src < T.n_crystals) {
            const long long col = P.pair_col ? (long long)P.pair_col[rank] : (long long)(rank - P.pair_r0);
            v = P.pair[(long long)(src * np + p) * P.pair_ld + col];
        }
        pr[p][r][ss] = v;
    }
    __syncthreads();
    const int rank = r0 + rl, s = s0 + sl;
    if (rank >= P.rank1 || s >= T.n_crystals) return;
    const int d = P.perm[rank];
    Det D;
    const float scale = setup_det<kScatterCrystal>(P, G, T, d, D);
    for (int a0 = 0; a0 < n_anchors; a0 += kMaxAnchorsPerPass) {
        const int na = min(kMaxAnchorsPerPass, n_anchors - a0);
        float acc[kMaxAnchorsPerPass];
        float3 I[kMaxAnchorsPerPass], Is[kMaxAnchorsPerPass];
        bool use[kMaxAnchorsPerPass];
#pragma unroll
        for (int j = 0; j < kMaxAnchorsPerPass; ++j) {
            acc[j] = 0.0f;
            use[j] = false;
            if (j < na) {
                const float4 vb = vbar[(long long)(a0 + j) * T.n_crystals + s];
                use[j] = D.on && s != d && vb.w > 0.0f;
                I[j] = voxel_world(P, vb.x, vb.y, vb.z);
                Is[j] = make_float3((I[j].x - D.x) * D.cm - (I[j].z - D.z) * D.sm, I[j].y - D.y,
                                    (I[j].x - D.x) * D.sm + (I[j].z - D.z) * D.cm);
            }
        }
        bool any = false;
#pragma unroll
        for (int j = 0; j < kMaxAnchorsPerPass; ++j) any |= use[j];
        if (any) {
            for (int p = 0; p < np; ++p) {
                Src C;
                make_src_basic(D, T.crystal_src[s * np + p], C);
                make_src_rest(D, pr[p][rl][sl], C);
#pragma unroll
                for (int j = 0; j < kMaxAnchorsPerPass; ++j)
                    if (use[j])
                        acc[j] += scatter_term<false>(P, D, C, kn, nullptr, T.kn_inv_norm, I[j].x, I[j].y, I[j].z, Is[j].x, Is[j].y,
                                               Is[j].z);
            }
        }
#pragma unroll
        for (int j = 0; j < kMaxAnchorsPerPass; ++j)
            if (j < na) K[(long long)(a0 + j) * anchor_stride + (long long)(rank - P.rank0) * ldk + s] = (KT)(acc[j] * scale);
    }
}

// ---- exact scatter of a detector tile and a voxel brick -----------------------------------
// CTA = 32 detectors x C columns (C = 4, 2 or 1) of 32 voxels along y, 8 warps; 8 / C
// warps share a column and take every (8 / C)-th detector.  Only a few per cent of the
// (detector, voxel, scatter point) terms pass the energy window, scattered over lanes, and
// a term costs some 350 instructions: each warp lists the pairs that can pass and evaluates
// full warps of them.  Per batch of NQ scatter points:
//  1. the CTA stages, per (point, detector), everything the terms need of it (Src: offsets,
//     corner directions, the pair sums), once for all columns, culls the detectors whose
//     window no voxel of a column reaches, and stages the points' weights (PE of the
//     source, or the hole's solid angle) per voxel; the loads of the next batch are issued
//     before the terms of this one;
//  2. each warp tests its voxels (lane = voxel) for every remaining detector with the
//     cosine alone against the detector's threshold (margin 2e-3, far above the test's
//     rounding) and appends the passing (point, detector, voxel) to its queue;
//  3. whenever 32 entries wait, one term per lane; the sums are doubles in shared memory,
//     every cell owned by one warp and added to in (source, point) order, so the split
//     into columns, rows lists and bricks changes no bit.
// What bounds it: instruction issue (FP32 and transcendental; 66 % of the slots taken, the
// rest fixed latencies), 2 CTAs of 8 warps per SM by registers and shared memory alike.
// 2048 detectors x 16384 voxels x 2048 points, the whole call with its pairs: 297 ms with
// the terms evaluated where their lane is the detector (17 of 32 lanes at work), 140 ms in
// this form.
template <int C>
struct ScShape {
    static constexpr int NQ = 8;                       // points per batch (shared memory: 5 KB each)
    static constexpr int W = kScWarps / C;             // warps per column
    static constexpr int PER = NQ * 32 * C / kScThreads;   // staged weights per thread
};

template <int C>
struct __align__(16) ScSmem {
    KnNode kn[kKnNodes + 1];
    double acc[C][kScTileD][kScBrickY];                // cell (d, y) at [d][y ^ d]: no bank conflicts either way
    float4 vox[C][kScBrickY];                          // voxel centres (world); w < 0 marks outside the grid
    float wgt[ScShape<C>::NQ][C][kScBrickY];           // weight of the point for the voxel
    float4 src[ScShape<C>::NQ];                        // scatter points
    float4 b[ScShape<C>::NQ][kScTileD];                // D - S, and c_cut |D - S| (1e30: detector off)
    float4 pr[ScShape<C>::NQ][kScTileD];               // pair sums
    float4 e[ScShape<C>::NQ][8][kScTileD];             // corner directions; w: |D-S|^2, |D-S|, phi_k, c_len, S in D's frame
    float4 det[4][kScTileD];                           // Det's fields
    float scale[kScTileD];                             // per detector: mu_c / mu_pe / points, or plate mu_c / mu_t
    int d[kScTileD];
    unsigned todo[ScShape<C>::NQ][C];                  // per (point, column): detectors that pass the column's cull
    unsigned short queue[kScWarps][96];                // point << 10 | detector << 5 | voxel
};

template <int C>
constexpr bool two_ctas() { return 2 * (sizeof(ScSmem<C>) + 1024) <= 228 * 1024; }
static_assert(two_ctas<4>() && two_ctas<2>() && two_ctas<1>(), "two CTAs per SM");

// scatter_term's view of a staged (point, detector).
struct SrcView {
    const float4* e;             // [8] corner directions, stride kScTileD
    float sx, sy, sz, ssx, ssy, ssz, bx, by, bz, bb, L, phi_k, c_len;
    float4 pr;
    __device__ __forceinline__ float3 corner(int i) const {
        const float4 v = e[i * kScTileD];
        return make_float3(v.x, v.y, v.z);
    }
    __device__ __forceinline__ float3 pick(int i) const { return corner(i); }
};

template <int KIND, int C>
__global__ void __launch_bounds__(kScThreads, 2) scatter_main_kernel(const __grid_constant__ ScatterParams P,
                                                                    const __grid_constant__ DevGeometry G,
                                                                    const __grid_constant__ ScatterTables T) {
    using Shape = ScShape<C>;
    constexpr int NQ = Shape::NQ, W = Shape::W, PER = Shape::PER, PARTS = kScBrickX / C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ScSmem<C>& S = *reinterpret_cast<ScSmem<C>*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = blockIdx.x % PARTS, b = (blockIdx.x / PARTS) % P.n_bricks, dt = blockIdx.x / (PARTS * P.n_bricks);
    const int c0 = part * C;                                 // first column of the brick
    const int y0 = brick_column(P, b, 0).y0;

    for (int i = tid; i < kKnNodes + 1; i += kScThreads) S.kn[i] = T.kn[i];
    for (int i = tid; i < C * kScBrickY * kScTileD; i += kScThreads) (&S.acc[0][0][0])[i] = 0.0;
    for (int i = tid; i < C * kScBrickY; i += kScThreads) {
        const BrickCol bc = brick_column(P, b, c0 + i % C);
        const int y = y0 + i / C;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        if (bc.valid && y < P.ny) {
            const float3 w = voxel_world(P, (float)bc.x, (float)y, (float)bc.z);
            v = make_float4(w.x, w.y, w.z, 1.0f);
        }
        S.vox[i % C][i / C] = v;
    }
    const int n_det = min(kScTileD, P.rank1 - (P.rank0 + dt * kScTileD));
    if (warp == 0) {
        const int rank = P.rank0 + dt * kScTileD + lane;
        Det D{};
        D.on = false;
        float scale = 0.0f;
        int d = -1;
        if (lane < n_det) {
            d = P.perm[rank];
            scale = setup_det<KIND>(P, G, T, d, D);
        }
        S.det[0][lane] = make_float4(D.x, D.y, D.z, D.cm);
        S.det[1][lane] = make_float4(D.sm, D.hw, D.ht, D.hh);
        S.det[2][lane] = make_float4(D.r_unit, D.mu_pe, D.mu_c, D.res);
        S.det[3][lane] = make_float4(D.lo, D.hi, D.on ? D.c_cut : 2.0f, 0.0f);
        S.scale[lane] = scale;
        S.d[lane] = d;
    }
    __syncthreads();

    // this warp's column: I0 + t e, t in [0, col_t] (image y axis, rotated); lane = voxel
    const int col = warp / W, sub = warp % W;
    const float4 I = S.vox[col][lane];
    const float col_ex = -P.sin_a, col_ey = P.cos_a;
    const float col_t = (float)(min(kScBrickY, P.ny - y0) - 1) * P.vy;
    const float c_cut = S.det[3][lane].z;                    // lane = detector
    const unsigned mine = (W == 2 ? 0x55555555u : (W == 4 ? 0x11111111u : 0x01010101u)) << sub;

    // This thread's place in the staged weights: one voxel of the tile, points first, first + step, ...
    constexpr int kPlaces = 32 * C, kStep = kScThreads / kPlaces;
    const int w_first = tid / kPlaces, w_col = tid % C, w_y = tid % kPlaces / C;
    long long w_at = -1;
    if (KIND == kScatterCrystal) {
        const BrickCol bc = brick_column(P, b, c0 + w_col);
        if (bc.valid && y0 + w_y < P.ny) w_at = bc.x + (long long)P.nx * (y0 + w_y + (long long)P.ny * bc.z);
    }
    const unsigned below = (1u << lane) - 1u;
    unsigned short* const waiting = S.queue[warp];
    long long pair_at = 0;                                   // this lane's pair column
    if (lane < n_det) {
        const int rank = P.rank0 + dt * kScTileD + lane;
        pair_at = P.pair_col ? P.pair_col[rank] : rank - P.pair_r0;
    }

    // The scatter points in order: sources with PE != 0 in the brick and their points, or the holes.
    const uint32_t* srcw = KIND == kScatterCrystal ? P.brick_sources + (long long)b * P.src_words : nullptr;
    int wd = -1, next_p = T.n_points, next_s = -1;
    uint32_t bits = 0u;
    // Loads of a batch: weights (crystal kind) and this thread's pair sums.  q: points, -1 past
    // the last; s: their sources.
    int q[NQ], s[NQ];
    float pe[PER];
    float4 pr;
    auto fetch = [&] {
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            q[k] = s[k] = -1;
            if (KIND != kScatterCrystal) {
                if (next_s + 1 < T.n_holes0) q[k] = ++next_s;
                continue;
            }
            if (next_p >= T.n_points) {
                while (!bits && wd + 1 < P.src_words) bits = srcw[++wd];
                if (!bits) continue;
                next_s = (wd << 5) + __ffs(bits) - 1;
                bits &= bits - 1u;
                next_p = 0;
            }
            q[k] = next_s * T.n_points + next_p++;
            s[k] = next_s;
        }
        if (KIND == kScatterCrystal) {
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                int sk = -1;
#pragma unroll
                for (int j = 0; j < NQ; ++j) sk = w_first + i * kStep == j ? s[j] : sk;
                pe[i] = sk >= 0 && w_at >= 0 ? __ldg(P.pe + (long long)sk * P.ld_pe + w_at) : 0.0f;
            }
        }
        pr = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (warp < NQ && lane < n_det) {
            int qk = -1;
#pragma unroll
            for (int j = 0; j < NQ; ++j) qk = warp == j ? q[j] : qk;
            if (qk >= 0) pr = __ldg(P.pair + (long long)qk * P.pair_ld + pair_at);
        }
    };
    fetch();
    while (q[0] >= 0) {
        __syncthreads();                                     // the previous batch's terms are done
        int n_q = 0;
#pragma unroll
        for (int k = 0; k < NQ; ++k) n_q += q[k] >= 0;
        if (KIND == kScatterCrystal) {
#pragma unroll
            for (int i = 0; i < PER; ++i) S.wgt[w_first + i * kStep][w_col][w_y] = pe[i];
        }
        if (warp < n_q) {
            int qk = q[0], sk = s[0];
#pragma unroll
            for (int j = 1; j < NQ; ++j) {
                qk = warp == j ? q[j] : qk;
                sk = warp == j ? s[j] : sk;
            }
            const float4 pt = KIND == kScatterCrystal ? T.crystal_src[qk] : T.hole_src[qk];
            if (lane == 0) S.src[warp] = pt;
            Det D;
            const float4 d0 = S.det[0][lane], d1 = S.det[1][lane];
            D.x = d0.x; D.y = d0.y; D.z = d0.z; D.cm = d0.w; D.sm = d1.x; D.hw = d1.y; D.ht = d1.z; D.hh = d1.w;
            D.r_unit = S.det[2][lane].x;
            const bool on = c_cut < 2.0f && !(KIND == kScatterCrystal && sk == S.d[lane]);
            Src c;
            make_src_basic(D, pt, c);
            S.b[warp][lane] = make_float4(c.bx, c.by, c.bz, on ? c_cut * c.L : 1e30f);
            // detectors whose window no voxel of a column passes sit that column out
            for (int xx = 0; xx < C; ++xx) {
                const float4 v0 = S.vox[xx][0];
                const unsigned m = __ballot_sync(0xffffffffu, on && column_max_cos(c, v0.x, v0.y, v0.z, col_ex, col_ey, 0.0f, col_t) > c_cut);
                if (lane == 0) S.todo[warp][xx] = m;
            }
            if (on) {
                make_src_rest(D, pr, c);
                const float more[8] = {c.bb, c.L, c.phi_k, c.c_len, c.ssx, c.ssy, c.ssz, 0.0f};
#pragma unroll
                for (int i = 0; i < 8; ++i) S.e[warp][i][lane] = make_float4(c.e[i][0], c.e[i][1], c.e[i][2], more[i]);
                S.pr[warp][lane] = pr;
            }
        }
        __syncthreads();
        fetch();                                             // next batch, in flight during the terms

        int count = 0;                                       // queue length
        int k = 0;                                           // point of the batch
        unsigned todo = 0u;                                  // its detectors still to test
        float ux = 0.0f, uy = 0.0f, uz = 0.0f;               // direction voxel -> point, NaN where the voxel has no term
        auto open_point = [&] {
            // weights and directions of the voxels (lane)
            const float4 pt = S.src[k];
            float w;
            bool live;
            if (KIND == kScatterCrystal) {
                w = S.wgt[k][col][lane];
                live = w != 0.0f;
            } else {
                // virtual solid angle of the hole seen from the voxel (scatter.cu:1707-1713)
                const float vr = 0.1f;
                const float dx = I.x - pt.x, dy = I.y - pt.y, dz = I.z - pt.z;
                const float L2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                const float Lih = sqrtf(L2);
                w = (vr * vr * 3.14159265358979323846f + pt.w * vr) / (4.0f * 3.14159265358979323846f * L2) *
                    fabsf(pt.y - I.y) / Lih;
                S.wgt[k][col][lane] = w;                     // (the column's warps write the same values)
                live = I.w >= 0.0f;
            }
            todo = __any_sync(0xffffffffu, live) ? S.todo[k][col] & mine : 0u;
            ux = pt.x - I.x; uy = pt.y - I.y; uz = pt.z - I.z;
            const float inv = live ? fast_rsqrt(fmaf(ux, ux, fmaf(uy, uy, uz * uz))) : __int_as_float(0x7fffffff);
            ux *= inv; uy *= inv; uz *= inv;
        };
        open_point();
        for (;;) {
            // fill the queue to a full warp of terms
            while (count < 32) {
                if (!todo) {
                    if (++k >= n_q) break;
                    open_point();
                    continue;
                }
                // two detectors at a time (the second may be the first again: then it passes nothing)
                const int d0 = __ffs(todo) - 1;
                todo &= todo - 1u;
                const bool both = todo != 0u;
                const int d1 = both ? __ffs(todo) - 1 : d0;
                todo &= todo - 1u;
                const float4 b0 = S.b[k][d0], b1 = S.b[k][d1];
                const bool p0 = fmaf(ux, b0.x, fmaf(uy, b0.y, uz * b0.z)) > b0.w;
                const bool p1 = both && fmaf(ux, b1.x, fmaf(uy, b1.y, uz * b1.z)) > b1.w;
                const unsigned m0 = __ballot_sync(0xffffffffu, p0), m1 = __ballot_sync(0xffffffffu, p1);
                if (p0) waiting[count + __popc(m0 & below)] = (unsigned short)(k << 10 | d0 << 5 | lane);
                count += __popc(m0);
                if (p1) waiting[count + __popc(m1 & below)] = (unsigned short)(k << 10 | d1 << 5 | lane);
                count += __popc(m1);
            }
            if (count == 0) break;
            __syncwarp();
            const int n = min(count, 32);
            const unsigned item = waiting[lane < n ? lane : 0];
            const int slot = item >> 10, dl = item >> 5 & 31, j = item & 31;
            double add = 0.0;
            if (lane < n) {
                Det D;
                const float4 d0 = S.det[0][dl], d1 = S.det[1][dl], d2 = S.det[2][dl], d3 = S.det[3][dl];
                D.x = d0.x; D.y = d0.y; D.z = d0.z; D.cm = d0.w;
                D.sm = d1.x; D.hw = d1.y; D.ht = d1.z; D.hh = d1.w;
                D.r_unit = d2.x; D.mu_pe = d2.y; D.mu_c = d2.z; D.res = d2.w;
                D.lo = d3.x; D.hi = d3.y;
                SrcView c;
                c.e = &S.e[slot][0][dl];
                const float4 pt = S.src[slot], bd = S.b[slot][dl];
                c.sx = pt.x; c.sy = pt.y; c.sz = pt.z;
                c.bx = bd.x; c.by = bd.y; c.bz = bd.z;
                c.bb = c.e[0].w; c.L = c.e[kScTileD].w; c.phi_k = c.e[2 * kScTileD].w; c.c_len = c.e[3 * kScTileD].w;
                c.ssx = c.e[4 * kScTileD].w; c.ssy = c.e[5 * kScTileD].w; c.ssz = c.e[6 * kScTileD].w;
                c.pr = S.pr[slot][dl];
                const float4 V = S.vox[col][j];
                const float isx = (V.x - D.x) * D.cm - (V.z - D.z) * D.sm;
                const float isy = V.y - D.y;
                const float isz = (V.x - D.x) * D.sm + (V.z - D.z) * D.cm;
                const float t = scatter_term<true>(P, D, c, S.kn, T.window, T.kn_inv_norm, V.x, V.y, V.z, isx, isy, isz);
                add = (double)(S.wgt[slot][col][j] * t);
            }
            // a cell may wait for several points: one point at a time
            const int last = __shfl_sync(0xffffffffu, slot, n - 1);
            for (int p = __shfl_sync(0xffffffffu, slot, 0); p <= last; ++p) {
                if (lane < n && slot == p) S.acc[col][dl][j ^ dl] += add;
                __syncwarp();
            }
            // the rest of the queue moves up
            const unsigned short rest = waiting[32 + lane], more = waiting[64 + lane];
            __syncwarp();
            if (lane < count - n) waiting[lane] = rest;
            if (lane + 32 < count - n) waiting[32 + lane] = more;
            count -= n;
        }
    }
    __syncthreads();

    // write the tile: (detector, y, C columns) with the column fastest
    for (int i = tid; i < n_det * kScBrickY * C; i += kScThreads) {
        const int xx = i % C, yy = i / C % kScBrickY, dl = i / (C * kScBrickY);
        const BrickCol oc = brick_column(P, b, c0 + xx);
        const int yv = y0 + yy;
        if (!oc.valid || yv >= P.ny) continue;
        const int rk = P.rank0 + dt * kScTileD + dl;
        const long long ocol = P.cols ? (long long)oc.ci * P.ny + yv
                                      : (long long)oc.x + (long long)P.nx * (yv + (long long)P.ny * oc.z);
        const long long orow = P.slot ? (long long)P.slot[rk] : (long long)(S.d[dl] - P.dst_row0);
        float* out = P.dst + orow * P.ld + ocol;
        const float v = (float)S.acc[xx][dl][yy ^ dl] * S.scale[dl];
        *out = P.accumulate ? *out + v : v;
    }
}

template <int KIND, int C>
cudaError_t launch_main(const ScatterParams& P, const DevGeometry& G, const ScatterTables& T, long long tiles,
                        cudaStream_t s) {
    const long long blocks = tiles * (kScBrickX / C);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const cudaError_t e = cudaFuncSetAttribute(scatter_main_kernel<KIND, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(ScSmem<C>));
    if (e != cudaSuccess) return e;
    scatter_main_kernel<KIND, C><<<(unsigned)blocks, kScThreads, sizeof(ScSmem<C>), s>>>(P, G, T);
    return cudaGetLastError();
}

}  // namespace

int64_t crystal_bitmap_words(int n) {
    const int64_t bits = ((int64_t)n * (n + 1) / 2) * n;
    return (bits + 31) / 32;
}

int64_t collimator_bitmap_words(int n, int h0) {
    const int64_t bits = (int64_t)h0 * n * n;
    return (bits + 31) / 32;
}

cudaError_t launch_bitmap_crystal(uint32_t* words, int64_t n_words, const ScatterTables& T, cudaStream_t s) {
    if (n_words <= 0) return cudaSuccess;
    const long long blocks = std::min<long long>((n_words + 255) / 256, 148LL * 64);   // a warp per 32 words
    bitmap_kernel<kScatterCrystal><<<(unsigned)blocks, 256, 0, s>>>(words, n_words, T);
    return cudaGetLastError();
}

cudaError_t launch_bitmap_collimator(uint32_t* words, int64_t n_words, const ScatterTables& T, cudaStream_t s) {
    if (n_words <= 0) return cudaSuccess;
    const long long blocks = std::min<long long>((n_words + 255) / 256, 148LL * 64);
    bitmap_kernel<kScatterCollimator><<<(unsigned)blocks, 256, 0, s>>>(words, n_words, T);
    return cudaGetLastError();
}

cudaError_t launch_scatter_pairs(int kind, const DevGeometry& G, const ScatterTables& T, const uint32_t* bitmap,
                                 const int* perm, int r0, int r1, float4* pair, cudaStream_t s) {
    const int n_src = kind == kScatterCrystal ? T.n_crystals * T.n_points : T.n_holes0;
    if (r1 <= r0 || n_src <= 0) return cudaSuccess;
    dim3 grid((r1 - r0 + 127) / 128, std::min(n_src, 65535));
    if (kind == kScatterCrystal)
        scatter_pair_kernel<kScatterCrystal><<<grid, 128, 0, s>>>(G, T, bitmap, perm, r0, r1, pair, n_src);
    else
        scatter_pair_kernel<kScatterCollimator><<<grid, 128, 0, s>>>(G, T, bitmap, perm, r0, r1, pair, n_src);
    return cudaGetLastError();
}

cudaError_t launch_brick_sources(const ScatterParams& P, const ScatterTables& T, uint32_t* brick_sources,
                                 cudaStream_t s) {
    dim3 grid(P.n_bricks, (T.n_crystals + kScWarps - 1) / kScWarps);
    brick_sources_kernel<<<grid, kScThreads, 0, s>>>(P, T.n_crystals, brick_sources);
    return cudaGetLastError();
}

cudaError_t launch_scatter_transfer(const ScatterParams& P, const DevGeometry& G, const ScatterTables& T,
                                    const float4* vbar, int n_anchors, void* K, bool k_bf16, long long ldk,
                                    long long anchor_stride, cudaStream_t s) {
    if (P.rank1 <= P.rank0 || T.n_crystals <= 0 || n_anchors <= 0) return cudaSuccess;
    if (T.n_points <= kTrMaxPoints && (T.n_crystals + kTrSrcs - 1) / kTrSrcs <= 65535) {
        dim3 tg((P.rank1 - P.rank0 + kTrRanks - 1) / kTrRanks, (T.n_crystals + kTrSrcs - 1) / kTrSrcs);
        const int smem = (int)sizeof(TrSmem);
        cudaError_t e;
        if (k_bf16) {
            e = cudaFuncSetAttribute(scatter_transfer_tiled_kernel<__nv_bfloat16>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return e;
            scatter_transfer_tiled_kernel<__nv_bfloat16><<<tg, kTrRanks * kTrSrcs, smem, s>>>(
                P, G, T, vbar, n_anchors, static_cast<__nv_bfloat16*>(K), ldk, anchor_stride);
        } else {
            e = cudaFuncSetAttribute(scatter_transfer_tiled_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     smem);
            if (e != cudaSuccess) return e;
            scatter_transfer_tiled_kernel<float><<<tg, kTrRanks * kTrSrcs, smem, s>>>(
                P, G, T, vbar, n_anchors, static_cast<float*>(K), ldk, anchor_stride);
        }
        return cudaGetLastError();
    }
    dim3 grid((P.rank1 - P.rank0 + 127) / 128, std::min(T.n_crystals, 65535));
    if (k_bf16)
        scatter_transfer_kernel<__nv_bfloat16><<<grid, 128, 0, s>>>(P, G, T, vbar, n_anchors,
                                                                   static_cast<__nv_bfloat16*>(K), ldk, anchor_stride);
    else
        scatter_transfer_kernel<float><<<grid, 128, 0, s>>>(P, G, T, vbar, n_anchors, static_cast<float*>(K), ldk,
                                                            anchor_stride);
    return cudaGetLastError();
}

cudaError_t launch_scatter_main(const ScatterParams& P, const DevGeometry& G, const ScatterTables& T,
                                cudaStream_t s) {
    const long long tiles = (long long)((P.rank1 - P.rank0 + kScTileD - 1) / kScTileD) * P.n_bricks;
    if (tiles <= 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // Columns per CTA: fewer repeat the staging and the culls (by 1.12 and 1.37 of a
    // column's time at 2048 crystals), more leave the last wave of CTAs (2 per SM) emptier.
    // The cheaper of those that fill two waves, else one column.  (Eight columns: no faster
    // anywhere, 142.7 against 142.2 ms for 2048 crystals, 29.0 against 25.4 ms for 576.)
    const long long slots = 2LL * sms;
    int c = 1;
    double best = 0.0;
    for (int n : {4, 2, 1}) {
        const long long blocks = tiles * (kScBrickX / n);
        if (blocks < 2 * slots) continue;
        const double waves = (double)((blocks + slots - 1) / slots);
        const double cost = waves * n * (n == 4 ? 1.0 : (n == 2 ? 1.12 : 1.37));
        if (best == 0.0 || cost < best) {
            best = cost;
            c = n;
        }
    }
    if (P.kind == kScatterCrystal) {
        if (c == 4) return launch_main<kScatterCrystal, 4>(P, G, T, tiles, s);
        if (c == 2) return launch_main<kScatterCrystal, 2>(P, G, T, tiles, s);
        return launch_main<kScatterCrystal, 1>(P, G, T, tiles, s);
    }
    if (c == 4) return launch_main<kScatterCollimator, 4>(P, G, T, tiles, s);
    if (c == 2) return launch_main<kScatterCollimator, 2>(P, G, T, tiles, s);
    return launch_main<kScatterCollimator, 1>(P, G, T, tiles, s);
}

}  // namespace smb
