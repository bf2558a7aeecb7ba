// kb_series.cuh -- the Bessel factors of the tap records as power series on float
// pairs: the host's coefficients and the device's evaluation.
#pragma once
#include <cmath>
#include <vector>

#include "cgs_common.cuh"
#include "cgs_types.h"

namespace cgs {

// Float pairs hi + lo (|lo| at most half an ulp of hi): about 46 bits from FP32
// operations, of which the GPU has 64 times as many as FP64 ones.  Knuth's and
// Dekker's error-free sum and product (the product's error from a fused
// multiply-add).
CGS_D float2 pair_sum(float a, float b)
{
    const float h = __fadd_rn(a, b), t = __fsub_rn(h, a);
    return make_float2(h, __fadd_rn(__fsub_rn(a, __fsub_rn(h, t)), __fsub_rn(b, t)));
}
CGS_D float2 pair_norm(float h, float l)   // |h| >= |l|
{
    const float s = __fadd_rn(h, l);
    return make_float2(s, __fsub_rn(l, __fsub_rn(s, h)));
}
CGS_D float2 pair_mul(float2 a, float2 b)
{
    const float p = __fmul_rn(a.x, b.x);
    return pair_norm(p, __fmaf_rn(a.y, b.x, __fmaf_rn(a.x, b.y, __fmaf_rn(a.x, b.x, -p))));
}
CGS_D float2 pair_add(float2 a, float2 b)
{
    const float2 s = pair_sum(a.x, b.x);
    return pair_norm(s.x, __fadd_rn(s.y, __fadd_rn(a.y, b.y)));
}
// 1 - q^2 for 0 <= q <= 1
CGS_D float2 pair_one_minus_sq(float q)
{
    const float p = __fmul_rn(q, q);
    const float2 s = pair_sum(1.f, -p);
    return pair_norm(s.x, __fsub_rn(s.y, __fmaf_rn(q, q, -p)));
}

// True when every value within 2^-41 of the pair's rounds to its hi.  The pairs
// below are within 2^-44 of the FP64 forms they stand for, so then hi is the
// float that the FP64 form rounds to.  A pair that lies closer to the middle
// between two floats (1.1 x 10^-5 of 4 x 10^7 draws) is formed in FP64 instead:
// without that, 1 in 10^6 to 10^7 floats was a neighbour of the FP64 form's.
CGS_D bool pair_rounds(float2 v)
{
    const float e = __fmul_rn(fabsf(v.x), 0x1p-41f);
    return __fadd_rn(v.x, __fadd_rn(v.y, e)) == v.x && __fadd_rn(v.x, __fsub_rn(v.y, e)) == v.x;
}

// The series by Horner's rule.  All terms are positive, so the rounding errors
// stay at a few 2^-46 of the value (2^-44.6 the largest of 2 x 10^7 draws at b =
// 8.9962, 14.9086 and 18.5, products with 1 / C included).
CGS_D float2 kb_series(const KbSeries& c, float2 s)
{
    float t = 0.f;
    for (int k = c.nf - 1; k >= 0; --k) t = __fmaf_rn(t, s.x, c.cf[k]);
    float2 r = make_float2(t, 0.f);
    for (int k = c.nd - 1; k >= 0; --k) r = pair_add(c.cd[k], pair_mul(r, s));
    return r;
}

// Factor of a tap at distance q (in kernel half-widths) along axis a, and the
// magnitude of its derivative with respect to the coordinate
CGS_D float2 kb_value(const KbParams& kb, int a, float q)
{
    return pair_mul(kb_series(kb.i0, pair_one_minus_sq(q)), kb.rC[a]);
}
CGS_D float2 kb_slope(const KbParams& kb, int a, float q)
{
    const float2 f = pair_mul(make_float2(q, 0.f), kb.f0[a]);
    return pair_mul(kb_series(kb.i1, pair_one_minus_sq(q)), f);
}

inline float2 float_pair(double v)
{
    const float h = (float)v;
    return make_float2(h, (float)(v - (double)h));
}

// I0(b sqrt(s)) (order 0) or I1(b sqrt(s)) / sqrt(s) (order 1) as a power
// series in s (Abramowitz and Stegun 9.6.10): c_k = (b/2)^order (b^2/4)^k /
// (k! (k + order)!), all positive.  Terms until their sum at s = 1 no longer
// changes; the tail that makes up less than 2^-30 of it goes to FP32 (its share
// is largest at s = 1).  nd = 0 when the shape needs more than the arrays hold.
inline KbSeries kb_series_of(double b, int order)
{
    std::vector<double> c;
    double t = order ? 0.5 * b : 1.0, sum = 0.0;
    for (int k = 0; k < 200; ++k) {
        c.push_back(t);
        sum += t;
        t *= 0.25 * b * b / ((double)(k + 1) * (double)(k + 1 + order));
        if (t < 1e-18 * sum && 0.25 * b * b < (double)(k + 1) * (double)(k + 1)) break;
    }
    int nd = (int)c.size();
    double tail = 0.0;
    while (nd > 1 && tail + c[nd - 1] < sum * 0x1p-30) tail += c[--nd];
    KbSeries s{};
    const int nf = (int)c.size() - nd;
    if (!(b >= 0.0) || !std::isfinite(sum) || nd > KB_ND || nf > KB_NF) return s;
    s.nd = nd;
    s.nf = nf;
    for (int k = 0; k < nd; ++k) s.cd[k] = float_pair(c[k]);
    for (int k = 0; k < nf; ++k) s.cf[k] = (float)c[nd + k];
    return s;
}

// series and scales of a kernel whose G, w and b are set
inline void kb_scales(KbParams& kb)
{
    for (int a = 0; a < 3; ++a) {
        const float dk = (float)(1.0 / (double)(float)(kb.G[a] - 1));
        const double C = (double)(float)(100.0f * kb.w * dk);
        kb.rC[a] = float_pair(1.0 / C);
        kb.f0[a] = float_pair((double)kb.b * (2.0 / ((double)kb.w * (double)dk)) / C);
    }
}

}  // namespace cgs
