// Host build of the tap records' Bessel factors (csrc/kb_series.cuh): the
// device's rounded FP32 operations as plain ones (compiled without contraction).
#include <cmath>
#include <cuda_runtime.h>

static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }

#include "kb_series.cuh"

// slope 0: the factors of taps at distances q[0..n), 1: their derivatives; v: the
// pairs' hi, sure: whether the FP64 form rounds to it.  Returns the FP32-pair
// terms of the series (0: the shape has no series).
extern "C" int kb_factors(float w, float b, int grid, int slope, long n, const float* q, float* v, unsigned char* sure)
{
    cgs::KbParams kb{};
    for (int a = 0; a < 3; ++a) kb.G[a] = grid;
    kb.w = w;
    kb.b = b;
    kb.i0 = cgs::kb_series_of((double)b, 0);
    kb.i1 = cgs::kb_series_of((double)b, 1);
    cgs::kb_scales(kb);
    for (long i = 0; i < n; ++i) {
        const float2 p = slope ? cgs::kb_slope(kb, 0, q[i]) : cgs::kb_value(kb, 0, q[i]);
        v[i] = p.x;
        sure[i] = cgs::pair_rounds(p);
    }
    return slope ? kb.i1.nd : kb.i0.nd;
}
