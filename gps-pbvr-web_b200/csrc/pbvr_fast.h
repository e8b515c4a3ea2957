// Fast decisions of the PBVR methods, shared by the particle kernel (with the GPU's approximate
// functions) and the CPU check of the error bounds (the same arithmetic with every approximation
// pushed to the edge of its assumed error).
//
// Most particles of a close view are never written: in the near orbit of a 560k-splat scene at
// 1280x720, 99 % of them fall off screen, behind the near plane or out of the radial keep test, and
// all that matters for them is whether they count as points. pbvr_decide answers that from
// approximate maths and a bound on |approximate - exact f32 value|; where a bound straddles a
// threshold it answers "undecided" and the caller runs the exact path from the particle's own
// stream, so the answers are the exact path's.
//
// Error model. Every standard normal is within kEN of the exact path's and at most kRMax in size
// (pairs with x = -2 log u1 < kXMin are left undecided; u1 = 0 gives NaN, which decides nothing).
// The camera-space position is linear in the normals, c(u) = C + M u, with C and M folded per
// splat in 64 bits; its bound against the exact path's f32 chain (world position, translation,
// rotation) is a per-splat constant that counts every rounding at the magnitude it happens at.
// The image position's bound e then is one fused expression in 1/z and the position's size, and
// the radial keep test is decided on the interval of y that e leaves: eol(y) = -log(1 - y) / y
// grows with y, so a draw above it at the upper end is surely rejected, one below it at the lower
// end surely kept, however wide the interval is. kU is one rounding, 2^-24; the constants of the
// approximations are checked on the GPU over every input they can get (gpsb_debug_fast_bounds);
// the exact maths' own errors are those of fmath.h.
//
// Measured (B200, 560k splats, PBVR Extinction C3+R, 1280x720) against an error bound propagated
// step by step from the magnitudes of the absolute coordinates, with every on-screen particle on the
// exact path and 4096-particle tiles per block: near view 79.9 -> 45.8 ms for 4 ensembles, mid 33.6
// -> 18.5 ms for 8, far 18.2 -> 11.8 ms for 64.
#pragma once
#include <math.h>
#include <stdint.h>

#include "fmath.h"

namespace gxf {

constexpr float kU = 6.0e-8f;
constexpr float kLogAbs = 3.5e-7f, kLogRel = 3.5e-7f;  // |ln2 lg2(v) - log v| <= kLogAbs + kLogRel |log v|, v in [kUMin, 1)
constexpr float kSinCos = 1e-6f;                    // sin and cos of t = RN(2 pi u), u = k 2^-24
constexpr float kXMin = 1e-3f;                      // smallest x = -2 log u1 the bounds cover
constexpr float kErMax = 2.5e-6f;                   // |r - r_exact| for x >= kXMin (r = x rsqrt(x))
constexpr float kRMax = 5.77f;                      // largest r (u1 >= kUMin)
constexpr float kEN = kErMax * (1.0f + 2.0f * kSinCos) + kRMax * (kSinCos + 2.01f * kU) + 1e-7f;  // one normal
constexpr float kLn2 = 0.693147182f;
constexpr float kHalfLog2e = 0.72134752f;

enum : uint32_t { kRadial = 1u, kJitter = 4u };  // FLAG_RADIAL, FLAG_JITTER

// Constants of a frame.
struct Frame {
    float kcx, kcy;    // principal point minus the frame's centre
    float hw, hh;      // half the frame
    float c0;          // constant part of the position bound (sums at the frame's size, jitter)
    float k3;          // the projection is at most this much larger than the jittered position
    float near_z, sd;  // sd: jitter scale, 0 without jitter
};

GX_HD Frame make_frame(uint32_t W, uint32_t H, float cx, float cy, float near_z, float sd, uint32_t flags) {
    Frame F;
    F.kcx = (float)((double)cx - 0.5 * (double)W);
    F.kcy = (float)((double)cy - 0.5 * (double)H);
    F.hw = 0.5f * (float)W;
    F.hh = 0.5f * (float)H;
    F.near_z = near_z;
    F.sd = (flags & kJitter) ? sd : 0.0f;
    const float kc = fmaxf(fabsf(F.kcx), fabsf(F.kcy)), j = fabsf(F.sd);
    F.k3 = 1.01f * (kc + j * (kRMax + kEN));
    // two sums of the exact path at the frame's size, the principal point's roundings, four
    // roundings of the projection, the jitter's normal and its product's roundings
    F.c0 = 1.05f * (kU * (1.5f * fmaxf((float)W, (float)H) + 4.0f * kc + 4.0f * F.k3) + j * (kEN + 6.0f * kU * kRMax));
    if (W > (1u << 20) || H > (1u << 20)) F.c0 = INFINITY;  // kCellBias holds grids below 2^22: settle nothing
    return F;
}

// The fast record of a splat, 24 floats: q[0..3] X (scaled by fx), q[4..7] Y (by fy), q[8..11] Z: the
// constant and the factors of (ux, uy, uz); q[12..14] the conic a, 2b, c; q[15] the bound factor of
// the squared distance; q[16..17] mean minus the frame's centre; q[18] log2 of the clamped opacity;
// q[19] eol(o) 2^-24; q[20..21] e1, e2 of the position bound; q[22] zmin, q[23] zbehind.
GX_HD void make_record(const Frame& F, const float* rot0, const float* rot1, const float* rot2, const float* pos, float fx,
                       float fy, const float* g, float k00, float k10, float k11, float k20, float k21, float k22, float a,
                       float b, float c, float mx, float my, float oo, float h, float* q) {
    const double U = 6.0e-8, gm = (double)kRMax + (double)kEN;
    const double s[3] = {fabs((double)k00), fabs((double)k10) + fabs((double)k11),
                         fabs((double)k20) + fabs((double)k21) + fabs((double)k22)};
    const float* rot[3] = {rot0, rot1, rot2};
    double E[3], top = 0.0;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const double f = r == 0 ? (double)fx : r == 1 ? (double)fy : 1.0;
        const double r0 = rot[r][0], r1 = rot[r][1], r2 = rot[r][2];
        double C = 0.0, w = 0.0, d = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double p = (double)g[i] - (double)pos[i], ri = rot[r][i], ai = fabs(ri);
            C += ri * p;
            // exact path: the normals, the sum for the world position, the translation
            w += ai * ((double)kEN * s[i] + U * (fabs((double)g[i]) + fabs(p) + 8.0 * s[i] * gm));
            d += ai * (fabs(p) + s[i] * gm);  // terms of the rotation's dot product, 3 roundings of their sum
        }
        const double m0 = r0 * k00 + r1 * k10 + r2 * k20, m1 = r1 * k11 + r2 * k21, m2 = r2 * k22;
        const double size = fabs(C) + (fabs(m0) + fabs(m1) + fabs(m2)) * gm;
        E[r] = 1.05 * fabs(f) * (w + 3.5 * U * d + 5.0 * U * size);  // + this path: the constants and 3 fused sums
        q[4 * r] = (float)(f * C);
        q[4 * r + 1] = (float)(f * m0);
        q[4 * r + 2] = (float)(f * m1);
        q[4 * r + 3] = (float)(f * m2);
        top = fmax(top, fabs(f) * size);
    }
    const double K = fabs((double)a) + 2.0 * fabs((double)b) + fabs((double)c);
    q[12] = a;
    q[13] = 2.0f * b;
    q[14] = c;
    q[15] = (float)(2.0 * K * 0.72134752 * 1.03);
    q[16] = (float)((double)mx - (double)F.hw);
    q[17] = (float)((double)my - (double)F.hh);
    q[18] = gx::log(oo) * 1.44269502f;
    q[19] = h * (1.0f / 16777216.0f);
    // 1 / (z - eZ) <= 1.0323 / z for z > 32 eZ
    q[20] = (float)(1.09 * (fmax(E[0], E[1]) + (double)F.k3 * E[2]));
    q[21] = (float)(1.09 * E[2]);
    const double zn = fmax(fmax((double)F.near_z + E[2], 32.0 * E[2]), 1e-6), zb = (double)F.near_z - E[2];
    q[22] = (float)(zn + fabs(zn) * 2.4e-7);
    q[23] = (float)(zb - fabs(zb) * 2.4e-7);
    // no decision where the splat's numbers leave the range the bounds hold in
    if (!(top < 1e30) || !(K < 1e30) || !(fabs((double)mx) < 1e30) || !(fabs((double)my) < 1e30) || !(E[2] < 1e30) ||
        !(E[0] < 1e30) || !(E[1] < 1e30) || !(oo > 0.0f) || !(h > 0.0f && h < 1e30f)) {
        q[22] = INFINITY;
        q[23] = -INFINITY;
    }
}

// One Box-Muller pair from the stream, drawn in the order of the exact path (cosine part, sine part).
template <class A>
GX_HD bool pair(A& ap, uint32_t& st, float& c, float& s) {
    st = gx::pcg(st);
    const float u1 = (float)(st >> 8u) * (1.0f / 16777216.0f);
    st = gx::pcg(st);
    const float t = (float)(st >> 8u) * (gxc::kTwoPi * (1.0f / 16777216.0f));  // = RN(2 pi u2)
    float x;
    const float r = ap.radius(u1, x);
    c = r * ap.cos(t);
    s = r * ap.sin(t);
    return x >= kXMin;
}

struct Point {
    float x, y;  // image position from the frame's centre
    float z, e;  // depth and the position's bound
};

// 0 not a point, 1 a point off screen, 2 undecided, 3 a point on screen or within e of its edge (at P).
// vc: the ViewConditioned draw against `keep` comes first (exact), and where ap.every(dropped) says so
// (every lane of a warp) nothing else is computed, as from far away almost no particle is kept: 560k splats,
// 1280x720, 4 ensembles, distance 60 (0.3 % kept) 12.7 -> 6.8 ms (the exact path of each lane, left at its draw,
// takes 10.4), 20: 13.4 -> 9.5, 7: 13.9 -> 13.3, 2.5: 10.6 both, with 2x2 subpixels 11.2 -> 11.4. Otherwise
// straight-line code: the lanes of a warp rarely agree on an early exit.
template <class A>
GX_HD uint32_t decide(A& ap, const Frame& F, uint32_t flags, bool vc, float keep, uint32_t st, const float* q, Point& P) {
    bool drop = false;
    if (vc) {
        uint32_t s = gx::pcg(gx::pcg(gx::pcg(gx::pcg(st))));  // past the two pairs
        drop = gx::next_u(&s) >= keep;
        if (ap.every(drop)) return 0u;
    }
    float uz, uy, ux, jy;
    bool ok = pair(ap, st, uz, uy);
    ok &= pair(ap, st, ux, jy);  // jy is the pair's spare, used by the jitter
    if (vc) st = gx::pcg(st);
    const float X = gx::fma_(q[3], uz, gx::fma_(q[2], uy, gx::fma_(q[1], ux, q[0])));
    const float Y = gx::fma_(q[7], uz, gx::fma_(q[6], uy, gx::fma_(q[5], ux, q[4])));
    const float Z = gx::fma_(q[11], uz, gx::fma_(q[10], uy, gx::fma_(q[9], ux, q[8])));
    const bool behind = Z <= q[23];
    bool sure = Z > q[22];
    const float iz = ap.rcp(Z);
    float sx = gx::fma_(X, iz, F.kcx), sy = gx::fma_(Y, iz, F.kcy);
    if (flags & kJitter) {
        float jx, js;
        sure &= pair(ap, st, jx, js);
        sx = gx::fma_(F.sd, jx, sx);
        sy = gx::fma_(F.sd, jy, sy);
    }
    // |position - exact position| <= (eXY + |projection| eZ) / (z - eZ) + roundings in both paths at
    // the position's size (10 kU) and the frame's (c0)
    const float T = fmaxf(fabsf(sx), fabsf(sy));
    const float e = gx::fma_(T, gx::fma_(iz, q[21], 6.5e-7f), gx::fma_(iz, q[20], F.c0));
    const bool off = fabsf(sx) > F.hw + e || fabsf(sy) > F.hh + e;
    uint32_t res = off ? 1u : 3u;
    if (flags & kRadial) {
        const float dx = sx - q[16], dy = sy - q[17];
        const float r2 = gx::fma_(dx, gx::fma_(q[13], dy, q[12] * dx), dy * (q[14] * dy));
        // |r2 - exact r2| <= 2 K (D + e) (e + 10 kU D), in powers of two of exp(-r2 / 2); the constant
        // covers the errors of both exponentials, log2 o and the roundings of this form
        const float D = fmaxf(fabsf(dx), fabsf(dy));
        const float ce = gx::fma_((D + e) * q[15], gx::fma_(D, 6e-7f, e), 1.3e-5f);
        const float t = gx::fma_(r2, -kHalfLog2e, q[18]);
        const float yh = ap.ex2(fminf(t + ce, q[18] + 1.3e-5f)), yl = ap.ex2(t - ce);
        // -log(1 - y) at both ends, the exact path's rounding of 1 - y included; ur y against it, within
        // 9e-7 and a relative 1.5e-6 (both logarithms' errors, the divisions by y and by eol(o))
        const float lh = ap.lg2((1.0f - 2.0f * kU) - yh), ll = ap.lg2((1.0f + 2.0f * kU) - yl);
        st = gx::pcg(st);
        const float ur = (float)(st >> 8u) * q[19];
        bool reject = gx::fma_(lh, kLn2 * 1.0000015f, ur * yh) >= 9e-7f;
        bool kept = gx::fma_(ll, kLn2 * 0.9999985f, ur * yl) < -9e-7f;
        // the exact path may sit at a smaller y, where the same error weighs more: at most 9e-7 / 1e-4
        // of 1, as it takes 1 + y / 2 below y = 1e-4; there only draws next to 1 are open
        reject = reject && ur >= 1.0096f;
        if (yh < 9.9e-5f) {
            reject = ur >= 1.0001f;
            kept = ur < 0.9999f;
        }
        res = reject ? 0u : (kept ? res : 2u);
    }
    res = sure ? res : 2u;
    res = behind || drop ? 0u : res;
    P.x = sx;
    P.y = sy;
    P.z = Z;
    P.e = e;
    return ok || drop ? res : 2u;
}

// Subpixel of a point that decide() left on screen: true when its bound settles it; on = within the
// frame, (cx, cy) its grid coordinates. Half a subpixel minus the bound (c0 again for the grid sum).
constexpr float kCellBias = 12582912.0f;  // 1.5 * 2^23: adding it rounds to the nearest whole number
GX_HD bool settle(const Frame& F, uint32_t side, uint32_t W, uint32_t H, const Point& P, uint32_t& cx, uint32_t& cy, bool& on) {
    const float s = (float)side;
    const float hx = gx::fma_(P.x, s, F.hw * s - 0.5f), hy = gx::fma_(P.y, s, F.hh * s - 0.5f);
    const float bx = hx + kCellBias, by = hy + kCellBias;
    const float lim = 0.5f - 2e-6f - (P.e + F.c0) * (s * 1.02f);
    cx = gx::f2b(bx) - 0x4B400000u;
    cy = gx::f2b(by) - 0x4B400000u;
    on = cx < W * side && cy < H * side;
    return fabsf(hx - (bx - kCellBias)) < lim && fabsf(hy - (by - kCellBias)) < lim;
}

}  // namespace gxf
