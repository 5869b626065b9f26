// chromat_ff.cuh -- the bilinear value of the chromatic PSF's zoom in FP32
// arithmetic.  The reference adds three of its four taps in double and rounds
// each sum to float (psf.c:54-136):
//   s = (1-u)(1-t) v00,  s = s + (1-u) t v01,  s = s + u (1-t) v10.
// The FP64 pipe bounded the zoom, so the sums are formed in float-float (pairs
// hi + lo): 1 - u as an exact pair, the products as exact two-products.  A sum is
// within 2^-43.5 of the exact one this way and the reference's own within 2^-50,
// both relative to the size of its terms (a position between -1 and 0 belongs to
// pixel 0, where u < 0 and taps are subtracted); where all values within 2^-42 of
// that size around the pair round to one float, that float is the reference's
// (Ziv's rounding test, "Fast evaluation of elementary mathematical functions with
// correctly rounded last bit", ACM TOMS 17, 1991).  The rest -- a sum beside a
// midpoint, about one pixel in 50,000, terms below 2^-80, whose errors may
// underflow, infinities and NaN -- is left to the double expressions.
// Host-compilable, checked against them on the CPU.
#pragma once
#include "atan_ff.cuh"

namespace atmwfs {

// The reference's expressions; the last tap in float, as there.
AW_HD float chromat_taps_f64(float u, float t, float v00, float v01, float v10, float v11)
{
    const double du = 1.0 - (double)u, dt = 1.0 - (double)t;
    float s = (float)(du * dt * (double)v00);
    s = (float)((double)s + du * (double)t * (double)v01);
    s = (float)((double)s + (double)u * dt * (double)v10);
    return ff_add(s, ff_mul(ff_mul(u, t), v11));
}

// s = float(r + e), m the size of what was added; false: values within 2^-42 m
// of r + e round otherwise.
AW_HD bool chromat_round(float r, float e, float m, float& s)
{
    const float d = ff_mul(m, 0x1p-42f);
    s = ff_add(r, ff_sub(e, d));
    return s == ff_add(r, ff_add(e, d));
}

// s = float(s + (wh + wl) v); m: the smaller of m and the size of the terms.
AW_HD bool chromat_add(float wh, float wl, float v, float& s, float& m)
{
    const float h = ff_mul(wh, v), l = ff_fma(wl, v, ff_fma(wh, v, -h));
    float r, e;
    ff_two_sum(s, h, r, e);
    const float n = ff_add(fabsf(r), fabsf(h));
    m = fminf(m, n);
    return chromat_round(r, ff_add(e, l), n, s);
}

// The bilinear value; false: chromat_taps_f64 has to say.
AW_HD bool chromat_taps(float u, float t, float v00, float v01, float v10, float v11, float& out)
{
    float duh, dul, dth, dtl, s;
    ff_two_sum(1.0f, -u, duh, dul);
    ff_two_sum(1.0f, -t, dth, dtl);
    const float w0 = ff_mul(duh, dth), w1 = ff_mul(duh, t), w2 = ff_mul(u, dth);
    const float w0l = ff_fma(duh, dtl, ff_fma(dul, dth, ff_fma(duh, dth, -w0)));
    const float w1l = ff_fma(dul, t, ff_fma(duh, t, -w1)), w2l = ff_fma(u, dtl, ff_fma(u, dth, -w2));
    const float h = ff_mul(w0, v00);
    float m = fabsf(h);
    bool sure = chromat_round(h, ff_fma(w0l, v00, ff_fma(w0, v00, -h)), m, s);
    sure = chromat_add(w1, w1l, v01, s, m) && sure;
    sure = chromat_add(w2, w2l, v10, s, m) && sure;
    sure = sure && (m >= 0x1p-80f || (v00 == 0.0f && v01 == 0.0f && v10 == 0.0f));
    out = ff_add(s, ff_mul(ff_mul(u, t), v11));
    return sure;
}

}  // namespace atmwfs
