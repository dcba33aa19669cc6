// gs_convert_fast.cuh — the FP32 side of the PLY conversion.
//
// gs_convert.cuh defines what a record holds: values worked out in double and rounded once to
// float (or to 8 bits).  GB300 runs two double operations per clock and SM against 128 float
// ones, so the same values are worked out here as unevaluated sums of two floats (about 2^-45)
// and rounded once; each function says whether rounding is certain, that is, whether every value
// within its error bound rounds the same way.  Where it is not (a value that close to a rounding
// boundary, a special value, a range the bounds do not cover) the caller takes the double path, so
// the two agree bit for bit.  All functions run on the host as well, where they are checked
// against the double path.
#pragma once

#include "gs_convert.cuh"

namespace gs {

// An unevaluated sum hi + lo of two floats.
struct Two {
    float hi, lo;
};

// Exact sum and product of two floats (Knuth; Dekker with an FMA).
GS_HD Two two_sum(float a, float b) {
    const float s = a + b, t = s - a;
    return Two{s, (a - (s - t)) + (b - t)};
}
GS_HD Two two_prod(float a, float b) {
    const float p = a * b;
    return Two{p, fmaf(a, b, -p)};
}

// hi + lo rounded to float in *out; false when a value within err of it could round elsewhere
// (or when anything is NaN).  err also covers the rounding of lo -+ err.
GS_HD bool round_certain(float hi, float lo, float err, float *out) {
    const float a = hi + (lo - err), b = hi + (lo + err);
    *out = a;
    return a == b;
}

// 2^(j/32) as hi + lo, j = 0..31.
#define GS_EXP_TABLE_SIZE 32
#define GS_EXP_TABLE \
    { \
        {0x1p+0f, 0.0f}, {0x1.059b0ep+0f, -0x1.9d4f52p-25f}, {0x1.0b5586p+0f, 0x1.9f3122p-25f}, {0x1.11301ep+0f, -0x1.fdb496p-25f}, \
        {0x1.172b84p+0f, -0x1.c15742p-27f}, {0x1.1d4874p+0f, -0x1.d2e8cap-25f}, {0x1.2387a6p+0f, 0x1.ceac48p-25f}, {0x1.29e9ep+0f, -0x1.5c0424p-25f}, \
        {0x1.306fep+0f, 0x1.4636e2p-25f}, {0x1.371a74p+0f, -0x1.18aac6p-25f}, {0x1.3dea64p+0f, 0x1.824684p-25f}, {0x1.44e086p+0f, 0x1.8624b4p-30f}, \
        {0x1.4bfdaep+0f, -0x1.593abcp-25f}, {0x1.5342b6p+0f, -0x1.2c561p-25f}, {0x1.5ab07ep+0f, -0x1.5bd5ecp-27f}, {0x1.6247ecp+0f, -0x1.f8b55p-25f}, \
        {0x1.6a09e6p+0f, 0x1.9fcef4p-26f}, {0x1.71f75ep+0f, 0x1.1d8beep-25f}, {0x1.7a1148p+0f, -0x1.829fdp-25f}, {0x1.82589ap+0f, -0x1.accc7cp-26f}, \
        {0x1.8ace54p+0f, 0x1.15506ep-27f}, {0x1.93737cp+0f, -0x1.e64744p-25f}, {0x1.9c4918p+0f, 0x1.51f848p-27f}, {0x1.a5503cp+0f, -0x1.b83b54p-25f}, \
        {0x1.ae89fap+0f, -0x1.a94b14p-26f}, {0x1.b7f77p+0f, -0x1.a09438p-25f}, {0x1.c199bep+0f, -0x1.3d56b2p-27f}, {0x1.cb720ep+0f, -0x1.8837ccp-27f}, \
        {0x1.d5818ep+0f, -0x1.822dbcp-27f}, {0x1.dfc974p+0f, -0x1.908c94p-25f}, {0x1.ea4afap+0f, 0x1.52486cp-27f}, {0x1.f50766p+0f, -0x1.246ebp-26f}, \
    }

// exp(x) rounded to float, after P. T. P. Tang, "Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic" (ACM TOMS 15(2), 1989): x = n ln2/32 + r with
// |r| <= ln2/64, exp(x) = 2^(n div 32) 2^((n mod 32)/32) (1 + expm1(r)), every term that reaches
// 2^-45 carried as a pair.  False outside |x| <= 80 or when the rounding is not certain.
GS_HD bool exp_certain(float x, const Two *table, float *out) {
    if (!(fabsf(x) <= 80.0f)) return false;
    const float n = rintf(x * 0x1.715476p+5f);  // 32 / ln2
    const int ni = (int)n;
    // ln2/32 in three parts of 12 bits, whose products with n (12 bits) are exact, and a rest
    Two r = two_sum(x - n * 0x1.62ep-6f, -(n * 0x1.0bep-20f));
    const Two r3 = two_sum(r.hi, -(n * 0x1.be8p-32f));
    const float rl = (r.lo + r3.lo) - n * 0x1.cf79acp-45f;
    const float rh = r3.hi;
    // expm1: r + r^2/2 as pairs, the rest in one float
    const Two sq = two_prod(rh, 0.5f * rh);
    const float q = (rh * rh) * (rh * fmaf(rh, fmaf(rh, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f));
    const Two h = two_sum(rh, sq.hi);
    const float hl = q + (((h.lo + sq.lo) + rl) + rh * rl);
    // table entry times (1 + expm1)
    const Two t = table[ni & 31];
    const Two m = two_prod(t.hi, h.hi);
    const Two v = two_sum(t.hi, m.hi);
    const float vl = v.lo + (fmaf(t.hi, hl, fmaf(t.lo, h.hi, t.lo)) + m.lo);
    float e;
    if (!round_certain(v.hi, vl, 0x1p-40f, &e)) return false;  // v is below 2.04
    const int k = ni >> 5;  // |k| <= 116: the scaling by 2^k is exact
    union {
        uint32_t u;
        float f;
    } s;
    s.u = (uint32_t)(k + 127) << 23;
    *out = e * s.f;
    return true;
}

// q / |q| rounded to float per component (x, y, z, w).  1/sqrt by one third-order step from a
// float estimate y0: with s y0^2 = 1 - e, 1/sqrt(s) = y0 (1 + e/2 + 3e^2/8 + ...), |e| < 2^-20.
template <class Rsqrt>
GS_HD bool unit_quat_certain(const float q[4], Rsqrt estimate, float out[4]) {
    Two s = two_prod(q[0], q[0]);
    bool ok = true;
    for (int k = 0; k < 4; ++k) {
        // products of smaller components lose their low parts
        ok = ok && (q[k] == 0.0f || fabsf(q[k]) >= 0x1p-30f);
        if (k == 0) continue;
        const Two p = two_prod(q[k], q[k]);
        const Two t = two_sum(s.hi, p.hi);
        s = Two{t.hi, t.lo + (s.lo + p.lo)};
    }
    if (!(ok && s.hi >= 0x1p-20f && s.hi <= 0x1p20f)) return false;
    const float y0 = estimate(s.hi);
    const Two yy = two_prod(y0, y0);
    const Two p = two_prod(s.hi, yy.hi);
    const float e = (1.0f - p.hi) - (p.lo + fmaf(s.hi, yy.lo, s.lo * yy.hi));
    if (!(fabsf(e) < 0x1p-20f)) return false;
    const float c = e * fmaf(0.375f, e, 0.5f);
    for (int k = 0; k < 4; ++k) {
        const Two v = two_prod(q[k], y0);
        float r;
        ok = round_certain(v.hi, fmaf(v.hi, c, v.lo), 0x1p-40f * fabsf(v.hi), &r) && ok;
        out[k] = q[k] == 0.0f ? q[k] : r;  // keeps the sign of zero
    }
    return ok;
}

// cov3d_from_rot_scale: R from exact products (error below 5 2^-48), M = R S, and the six sums of
// M M^T.  Adding up the roundings of the low parts bounds the error, with the double path's own and
// the rounding of the test, by 0.99 2^-43 of the sum of the squared scales (largest seen against
// 113-bit arithmetic over 10M random records: 0.30 2^-43).
GS_HD bool cov3d_certain(const float rot[4], const float scale[3], float out[6]) {
    const float x = rot[0], y = rot[1], z = rot[2], w = rot[3];
    bool ok = true;
    for (int k = 0; k < 4; ++k) ok = ok && (rot[k] == 0.0f || fabsf(rot[k]) >= 0x1p-30f) && fabsf(rot[k]) <= 1.0f;
    for (int k = 0; k < 3; ++k) ok = ok && scale[k] >= 0x1p-30f && scale[k] <= 0x1p30f;
    // narrow ranges keep every low part a normal float
    const float smax = fmaxf(scale[0], fmaxf(scale[1], scale[2])), smin = fminf(scale[0], fminf(scale[1], scale[2]));
    if (!(ok && smin >= smax * 0x1p-12f)) return false;
    const Two xx = two_prod(x, x), yy = two_prod(y, y), zz = two_prod(z, z);
    const Two xy = two_prod(x, y), xz = two_prod(x, z), yz = two_prod(y, z);
    const Two wx = two_prod(w, x), wy = two_prod(w, y), wz = two_prod(w, z);
    const Two pairs[9][2] = {{yy, zz}, {xy, wz}, {xz, wy}, {xy, wz}, {xx, zz}, {yz, wx}, {xz, wy}, {yz, wx}, {xx, yy}};
    const float sign[9] = {1, -1, 1, 1, 1, -1, -1, 1, 1};
    Two M[9];
    for (int k = 0; k < 9; ++k) {
        const Two t = two_sum(pairs[k][0].hi, sign[k] * pairs[k][1].hi);
        Two r{2.0f * t.hi, 2.0f * (t.lo + (pairs[k][0].lo + sign[k] * pairs[k][1].lo))};
        if (k % 4 == 0) {
            const Two d = two_sum(1.0f, -r.hi);
            r = Two{d.hi, d.lo - r.lo};
        }
        r = two_sum(r.hi, r.lo);  // |lo| back to half an ulp of hi
        const float s = scale[k % 3];
        const Two m = two_prod(r.hi, s);
        M[k] = Two{m.hi, fmaf(r.lo, s, m.lo)};
    }
    const float err = 0x1p-43f * fmaf(scale[0], scale[0], fmaf(scale[1], scale[1], scale[2] * scale[2]));
    const int A[6] = {0, 0, 0, 1, 1, 2}, B[6] = {0, 1, 2, 1, 2, 2};
    for (int k = 0; k < 6; ++k) {
        float lo = 0.0f;
        Two sum{0.0f, 0.0f};
        for (int c = 0; c < 3; ++c) {
            const Two a = M[A[k] * 3 + c], b = M[B[k] * 3 + c];
            const Two p = two_prod(a.hi, b.hi);
            lo += fmaf(a.lo, b.hi, fmaf(a.hi, b.lo, p.lo));
            if (c == 0) {
                sum = Two{p.hi, 0.0f};
            } else {
                const Two t = two_sum(sum.hi, p.hi);
                sum = Two{t.hi, sum.lo + t.lo};
            }
        }
        ok = round_certain(sum.hi, sum.lo + lo, err, &out[k]) && ok;
    }
    return ok;
}

// 255 v for v clamped to [0, 1], rounded half to even, from a float t = 255 v known to within
// err; false when that does not settle it (a half-way point inside the error, or NaN).
GS_HD bool unorm8_certain(float t, float err, uint32_t *out) {
    t = t > 0.0f ? (t < 255.0f ? t : 255.0f) : (t <= 0.0f ? 0.0f : t);  // NaN stays
    const float r = rintf(t);
    *out = (uint32_t)r;
    return fabsf(t - r) < 0.5f - err;
}

}  // namespace gs
