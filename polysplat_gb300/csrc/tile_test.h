// The exact ellipse / tile-box test of the key emission, and the candidate
// tiles of a row that a Gaussian's sweep has to test.  One header for the
// kernels and for the host check of the candidates against the test
// (tests/test_tile_candidates.py), which is built with -ffp-contract=off.
#pragma once

#include <stdint.h>

#include <cmath>

#ifdef __CUDACC__
#define GSR_TT_FN __device__ __forceinline__
#define GSR_TT_MUL(a, b) __fmul_rn(a, b)
#define GSR_TT_SUB(a, b) __fsub_rn(a, b)
#define GSR_TT_FMA(a, b, c) __fmaf_rn(a, b, c)
// fast math: within 2 ulp of the quotient, which a host check can stand in for
#define GSR_TT_DIV(a, b) ((a) / (b))
#else
#define GSR_TT_FN inline
#define GSR_TT_MUL(a, b) ((a) * (b))
#define GSR_TT_SUB(a, b) ((a) - (b))
#define GSR_TT_FMA(a, b, c) std::fma(a, b, c)
#ifndef GSR_TT_DIV
#define GSR_TT_DIV(a, b) ((a) / (b))
#endif
struct int2 { int x, y; };
struct float2 { float x, y; };
struct float3 { float x, y, z; };
#endif

namespace gsr {

// Ellipse / tile-box tests (preprocess.cu:257-311).
//
// The arithmetic is written with explicit rounding intrinsics, one per
// operation of the reference's expressions, fused where those expressions
// contract under fast math (x * y + z -> fma(x, y, z); x * x - y * z ->
// fma(x, x, -(y * z))).  Left to the compiler, the fusion of the same
// expression can differ between the kernels that inline it, and a tile on
// the ellipse's edge then passes in one kernel and fails in another: the
// depth-first pipeline counts a Gaussian's tiles in one kernel and emits
// them in another, so the two must agree bit for bit.
//
// The test takes the box's vertical and horizontal edge nearer the centre and
// asks whether the ellipse's quadratic reaches <= 0 on it.  What depends on the
// edge alone (an Edge) is formed once per tile column or row, so that a 2x2
// group of tiles needs four of them and not eight, without branches between
// them: 613 -> 461 us for the large-Gaussian sweep of 8 served views.
struct Edge {
    float two_a, b, delta;
};

// The edge at offset `off` from the centre: a, cross, c the conic with the
// edge's own direction first.
GSR_TT_FN Edge edge_at(float along, float cross, float across, float off, float w)
{
    Edge e;
    e.two_a = GSR_TT_MUL(2.0f, along);
    e.b = GSR_TT_MUL(GSR_TT_MUL(-2.0f, cross), off);
    const float c = GSR_TT_FMA(GSR_TT_MUL(across, off), off, -w);
    e.delta = GSR_TT_FMA(e.b, e.b, -GSR_TT_MUL(GSR_TT_MUL(4.0f, along), c));
    return e;
}

// ... reaches <= 0 between l - d and r - d (dl, dr) along the edge
GSR_TT_FN bool edge_hit(const Edge& e, float dl, float dr)
{
    const float t1 = GSR_TT_FMA(dl, e.two_a, e.b);
    const float t2 = GSR_TT_FMA(dr, e.two_a, e.b);
    return (e.delta >= 0.0f) & ((t1 <= 0.0f) | (GSR_TT_MUL(t1, t1) <= e.delta)) &
           ((t2 >= 0.0f) | (GSR_TT_MUL(t2, t2) <= e.delta));
}

// One tile column or row: its pixels [lo, hi], their offsets from the centre,
// the offset of the nearer edge, and whether it holds the centre.
struct Slab {
    float dl, dr, off;
    bool centre;
};

GSR_TT_FN Slab slab_of(int lo, int hi, float c)
{
    Slab s;
    s.dl = GSR_TT_SUB((float)lo, c);
    s.dr = GSR_TT_SUB((float)hi, c);
    s.off = GSR_TT_SUB(c, c * 2.0f < (float)(lo + hi) ? (float)lo : (float)hi);
    s.centre = (c >= (float)lo) & (c <= (float)hi);
    return s;
}

GSR_TT_FN bool tile_hit(int x, int y, int bx, int by, float2 ctr, float3 con, float power)
{
    const Slab col = slab_of(x * bx, x * bx + bx - 1, ctr.x), row = slab_of(y * by, y * by + by - 1, ctr.y);
    const float w = GSR_TT_MUL(2.0f, power);
    if (col.centre && row.centre) return true;
    if (!(power > 0.0f)) return false;
    if (edge_hit(edge_at(con.z, con.y, con.x, col.off, w), row.dl, row.dr)) return true;
    return edge_hit(edge_at(con.x, con.y, con.z, row.off, w), col.dl, col.dr);
}

// Tiles of quad (qx, qy) that lie in the Gaussian's rectangle [rmin, rmax)
// and pass tile_hit: bit (x & 1) | (y & 1) << 1 per hit tile.  These are
// exactly the tiles the per-tile emission would give keys.
GSR_TT_FN uint32_t quad_mask(int qx, int qy, int2 rmin, int2 rmax, int bx, int by, float2 ctr, float3 con, float power)
{
    const float w = GSR_TT_MUL(2.0f, power);
    const int x0 = 2 * qx * bx, y0 = 2 * qy * by;
    const Slab col[2] = {slab_of(x0, x0 + bx - 1, ctr.x), slab_of(x0 + bx, x0 + 2 * bx - 1, ctr.x)};
    const Slab row[2] = {slab_of(y0, y0 + by - 1, ctr.y), slab_of(y0 + by, y0 + 2 * by - 1, ctr.y)};
    uint32_t m = 0u;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < 2; k++) {  // one column's and one row's edge at a time
        const Edge ce = edge_at(con.z, con.y, con.x, col[k].off, w);
        m |= (edge_hit(ce, row[0].dl, row[0].dr) ? 1u << k : 0u) | (edge_hit(ce, row[1].dl, row[1].dr) ? 4u << k : 0u);
        const Edge re = edge_at(con.x, con.y, con.z, row[k].off, w);
        m |= (edge_hit(re, col[0].dl, col[0].dr) ? 1u << 2 * k : 0u) |
             (edge_hit(re, col[1].dl, col[1].dr) ? 2u << 2 * k : 0u);
    }
    m = power > 0.0f ? m : 0u;
    m |= ((col[0].centre ? 5u : 0u) | (col[1].centre ? 10u : 0u)) & ((row[0].centre ? 3u : 0u) | (row[1].centre ? 12u : 0u));
    // tiles of the rectangle
    m &= (2 * qx >= rmin.x && 2 * qx < rmax.x ? 5u : 0u) | (2 * qx + 1 >= rmin.x && 2 * qx + 1 < rmax.x ? 10u : 0u);
    m &= (2 * qy >= rmin.y && 2 * qy < rmax.y ? 3u : 0u) | (2 * qy + 1 >= rmin.y && 2 * qy + 1 < rmax.y ? 12u : 0u);
    return m;
}

// ---------------------------------------------------------------------------
// Which tiles can pass the test.
//
// kBandEllipse: a well-conditioned ellipse A dx^2 + 2B dx dy + C dy^2 <= w (w =
// 2 power).  In exact arithmetic the test only accepts tiles whose box meets
// the ellipse.  In float it can also accept a tile just outside.  On a box
// edge at offset dx from the centre, the test accepts a point of the edge
// where the computed quadratic is <= 0; the computed discriminant errs by a
// few 2^-24 of its terms' size, (B^2 + AC) dx^2 + C w, so every accepted point
// satisfies Q <= w (1 + k u (1 + kappa)), with u = 2^-24, kappa = 2AC / det >=
// (B^2 + AC) / det and k about 10 (the same holds for the horizontal edge).
// The candidates are therefore the exact row extents of the ellipse inflated
// to w (1 + tau), tau = 64 u (1 + kappa), plus half a pixel and a relative 1e-5
// for the rounding of the band arithmetic itself and of pixel coordinates.
// det = AC - B^2 is formed with a single rounding (Kahan's fused difference of
// products), and the half-width at height dy as sqrt(det (dymax - dy) (dymax +
// dy)) / A, which does not cancel near the top and bottom, so every extent
// carries a few ulp of relative error.
//
// kBandNeedle: A and C of one sign, with AC - B^2 below 1e-6 AC, or negative,
// or the ellipse beyond the above's range (FP32 covariances whose determinant
// cancelled, to a few ulp or to below zero).  The float discriminant says
// little there, but an accepted edge still lies near the conic's axis.  Write
// D(t, a) = max(a, 0) w + e |a| w + t^2 (max(0, -det) + e (AC + B^2)) with e =
// 16 u: the computed discriminant is at most 4 D (each of its operations errs
// by u of terms that sum to at most (AC + B^2) t^2 + |a| w, four of them in
// all).  With a > 0 the test accepts the row's pixels [l, r] on a vertical edge
// at offset dx = cx - ex only if t1 <= 2 sqrt(D) and t2 >= -2 sqrt(D) up to
// their rounding, that is if (B / C) dx lies within E = sqrt(D(dx, C)) / |C| +
// 4u (|l - cy| + |B dx / C|) of [l - cy, r - cy]; with a < 0 the inequalities
// turn round and ask that [l - cy, r - cy] lie within E of it, which implies
// the same.  So ex lies in an interval; and a horizontal edge at offset dy is
// accepted only if the tile's columns meet cx + (B / A) dy -+ E' with the same
// form.  E is taken at the rectangle's largest |dx|.  The row's
// candidates are the hull of both intervals and of the centre's tile, widened
// by a pixel and a relative 1e-5.  One clustered 3 M-Gaussian 1080p frame
// holds about 3200 rectangles of 8000 tiles each that are no well-conditioned
// ellipse; sweeping all their tiles was two thirds of the emission's tests, and
// the 40% of them with negative A and C hit a tile in four of them.
//
// kBandCentre: a NaN in the conic makes every discriminant NaN, as do a conic
// of infinities alone (a determinant of zero; inf - inf) with A and C of one
// sign, and without power > 0 no edge is tested: only the tile holding the
// centre can pass.
//
// kBandFull: everything else (A and C of different signs, zero, infinite):
// every tile.
enum : int { kBandFull = 0, kBandEllipse = 1, kBandNeedle = 2, kBandCentre = 3 };

struct Band {
    int kind;
    float B, inv_a, inv_c, det, dymax, dxmax, dyr, cx, cy, m;
    float e_h0, e_h1, e_v;  // needle: E' = sqrt(e_h0 + e_h1 dy^2) / A + ..., E at the largest |dx|
};

GSR_TT_FN Band make_band(float3 q, float power, float2 c, int x_lo, int x_hi, int bx)
{
    Band b;
    const float A = q.x, B = q.y, C = q.z, w = 2.0f * power;
    const float u = 5.9604645e-8f;
    const float bb = B * B;
    const float det = GSR_TT_FMA(A, C, -bb) + GSR_TT_FMA(-B, B, bb);
    const float kappa = GSR_TT_DIV(2.0f * (A * C), det);
    const float wb = w * (1.0f + 64.0f * u * (1.0f + kappa));  // inflated for the test's rounding
    b.B = B;
    b.inv_a = GSR_TT_DIV(1.0f, A);
    b.inv_c = GSR_TT_DIV(1.0f, C);
    b.det = det;
    b.dymax = sqrtf(GSR_TT_DIV(wb * A, det));
    b.dxmax = sqrtf(GSR_TT_DIV(wb * C, det));
    b.dyr = -B * sqrtf(GSR_TT_DIV(wb, C * det));  // dy where the ellipse reaches its largest x
    b.cx = c.x;
    b.cy = c.y;
    b.m = 0.5f + 1e-5f * fmaxf(b.dxmax, b.dymax);
    b.e_h0 = b.e_h1 = b.e_v = 0.0f;
    b.kind = kBandFull;
    const bool near = fabsf(c.x) < 1e7f && fabsf(c.y) < 1e7f;
    const bool infinite = fabsf(A) > 3.4028235e38f && fabsf(B) > 3.4028235e38f && fabsf(C) > 3.4028235e38f;
    if (!(A == A) || !(B == B) || !(C == C) || !(power > 0.0f) || (infinite && A * C > 0.0f)) {
        b.kind = kBandCentre;
    } else if (A > 0.0f && C > 0.0f && det > 1e-6f * (A * C) && b.dymax < 1e6f && b.dxmax < 1e6f &&
               fabsf(b.dyr) < 1e6f && near) {
        b.kind = kBandEllipse;
    } else if (near && A * C > 0.0f && fabsf(A) > 1e-15f && fabsf(C) > 1e-15f && fabsf(A) < 1e15f && fabsf(C) < 1e15f &&
               fabsf(B) < 1e15f && w < 1e15f) {
        b.kind = kBandNeedle;
        const float e = 16.0f * u;
        const float grow = fmaxf(0.0f, -det) + e * GSR_TT_FMA(A, C, bb);
        const float dxm = fmaxf(fabsf(c.x - (float)(x_lo * bx)), fabsf(c.x - (float)(x_hi * bx)));
        b.e_h0 = (fmaxf(A, 0.0f) + e * fabsf(A)) * w;
        b.e_h1 = grow;
        b.e_v = (sqrtf((fmaxf(C, 0.0f) + e * fabsf(C)) * w + grow * dxm * dxm) + 4.0f * u * fabsf(B) * dxm) *
                fabsf(b.inv_c);
        b.dxmax = dxm;
    }
    return b;
}

// Candidate tile columns [c_lo, c_hi] of tile row `ty` within [x_lo, x_hi):
// false when the row has none.
GSR_TT_FN bool band_columns(const Band& e, int ty, int by, int bx, int x_lo, int x_hi, int& c_lo, int& c_hi)
{
    float lo, hi;  // pixel range of the candidates
    const float l = (float)(ty * by), r = (float)(ty * by + by - 1);
    if (e.kind == kBandEllipse) {
        const float p = fmaxf(l - e.m - e.cy, -e.dymax);
        const float q = fminf(r + e.m - e.cy, e.dymax);
        if (!(p <= q)) return false;
        auto half = [&](float dy) {
            return sqrtf(e.det * fmaxf(0.0f, e.dymax - dy) * fmaxf(0.0f, e.dymax + dy)) * e.inv_a;
        };
        const float hp = half(p), hq = half(q);
        const float mp = -e.B * p * e.inv_a, mq = -e.B * q * e.inv_a;  // centre line of the ellipse at p, q
        const float xr = (e.dyr >= p && e.dyr <= q) ? e.dxmax : fmaxf(mp + hp, mq + hq);
        const float xl = (-e.dyr >= p && -e.dyr <= q) ? -e.dxmax : fminf(mp - hp, mq - hq);
        lo = e.cx + xl - e.m;
        hi = e.cx + xr + e.m;
    } else {
        const bool row_of_centre = e.cy >= l && e.cy <= r;
        // a pixel on either side, as everywhere: the quotient by a width that is
        // no power of two may fall below a whole number
        lo = row_of_centre ? e.cx - 1.0f : 3e38f;
        hi = row_of_centre ? e.cx + 1.0f : -3e38f;
        if (e.kind == kBandNeedle) {
            const float u = 5.9604645e-8f;
            // horizontal edge: the test's dy, its middle and half-width
            const float dy = e.cy * 2.0f < l + r ? e.cy - l : e.cy - r;
            const float mid = e.B * dy * e.inv_a;
            const float eh = sqrtf(e.e_h0 + e.e_h1 * dy * dy) * fabsf(e.inv_a) + 4.0f * u * (e.dxmax + fabsf(mid));
            const float mh = 1.0f + 1e-5f * (fabsf(e.cx) + fabsf(mid) + eh);
            lo = fminf(lo, e.cx + mid - eh - mh);
            hi = fmaxf(hi, e.cx + mid + eh + mh);
            // vertical edges: (B / C) dx within [v0, v1]
            const float far_y = fmaxf(fabsf(l - e.cy), fabsf(r - e.cy));
            const float ev = e.e_v * 1.00001f + 4.0f * u * far_y + 1e-5f * far_y + 1.0f;
            const float v0 = l - e.cy - ev, v1 = r - e.cy + ev;
            const float slope = e.B * e.inv_c;
            if (fabsf(slope) < 1e-6f) {  // next to an axis: every column, if any
                if (v0 <= 1e-6f * e.dxmax && v1 >= -1e-6f * e.dxmax) {
                    lo = -3e38f;
                    hi = 3e38f;
                }
            } else {
                const float d0 = GSR_TT_DIV(v0, slope), d1 = GSR_TT_DIV(v1, slope);  // dx range, in either order
                const float dmin = fminf(d0, d1), dmax = fmaxf(d0, d1);
                const float mv = 1.0f + 1e-5f * (fabsf(e.cx) + fmaxf(fabsf(dmin), fabsf(dmax)));
                // the edge ex = cx - dx is the tile's first or last column
                lo = fminf(lo, e.cx - dmax - mv - (float)(bx - 1));
                hi = fmaxf(hi, e.cx - dmin + mv + (float)(bx - 1));
            }
        }
    }
    if (!(lo == lo) || !(hi == hi)) {  // no bound: every column
        lo = -3e38f;
        hi = 3e38f;
    }
    c_lo = (int)fmaxf((float)x_lo, fminf(floorf(GSR_TT_DIV(lo, (float)bx)), (float)x_hi));
    c_hi = (int)fminf((float)(x_hi - 1), fmaxf(floorf(GSR_TT_DIV(hi, (float)bx)), -1.0f));
    return c_lo <= c_hi;
}

}  // namespace gsr
