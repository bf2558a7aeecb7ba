// gridding_common.cuh -- tap-record helpers shared by the gridding kernels:
// the packed nearest grid point and the 64-byte record load.
#pragma once
#include "cgs_common.cuh"
#include "cgs_types.h"

namespace cgs {

CGS_D unsigned pack_nearest(int nx, int ny, int nz)
{
    return (unsigned)nx | ((unsigned)ny << 11) | ((unsigned)nz << 22);
}
CGS_D void unpack_nearest(unsigned u, int& nx, int& ny, int& nz)
{
    nx = (int)(u & 2047u);
    ny = (int)((u >> 11) & 2047u);
    nz = (int)(u >> 22);
}


CGS_D void load_record(const TapRecord* __restrict__ rec, long long i, float (&w)[15], int& nx, int& ny,
                       int& nz)
{
    const float4* p = reinterpret_cast<const float4*>(rec + i);
    const float4 a = __ldg(p + 0), b = __ldg(p + 1), c = __ldg(p + 2), d = __ldg(p + 3);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    w[8] = c.x; w[9] = c.y; w[10] = c.z; w[11] = c.w;
    w[12] = d.x; w[13] = d.y; w[14] = d.z;
    unpack_nearest(__float_as_uint(d.w), nx, ny, nz);
}

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

// The series by Horner's rule.  All terms are positive, so the rounding errors
// stay at a few 2^-46 of the value; the tail in plain FP32 adds 2^-30 of an
// FP32 ulp.
CGS_D float2 kb_series(const KbSeries& c, float2 s)
{
    float t = 0.f;
    for (int k = c.nf - 1; k >= 0; --k) t = __fmaf_rn(t, s.x, c.cf[k]);
    float2 r = make_float2(t, 0.f);
    for (int k = c.nd - 1; k >= 0; --k) r = pair_add(c.cd[k], pair_mul(r, s));
    return r;
}

}  // namespace cgs
