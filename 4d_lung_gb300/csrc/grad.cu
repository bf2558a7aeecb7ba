// grad.cu -- gradients of the data-consistency loss
//   L = 1/2 sum_c sum_i D_i |(E_c S_c x)_i - y_ci|^2
// with respect to the sample coordinates (and, through the adjoint chain,
// the image).  E_c is the forward operator of nufftFWD (Reco.cpp:521-553);
// the reference has no derivatives, this is the extension that trajectory
// self-calibration needs.
//
// The interpolation weight of a tap is the product of three per-axis KB
// factors, w = fx(kx) fy(ky) fz(kz), so dw/dkx = fx'(kx) fy fz and so on.
// The per-axis derivatives are stored per sample like the tap records
// (15 floats + the packed nearest point), and one gather pass computes the
// predicted samples, their three coordinate derivatives, the residual, the
// loss partials and dL/dk.
#include "launch.h"
#include "gridding_common.cuh"
#include "ptx_async.cuh"

#include <algorithm>

namespace cgs {

// Derivative records: df/dk of the 5 candidate factors per axis, with the
// distance arithmetic of k_tap_records (Reco.cpp:763-771: double k minus
// float index * float dk, distance rounded to float).  For
// f = I0(b s) / C, s = sqrt(1 - q^2), q = 2 |d| / (w dk):
//   df/dk = -(I1(b s) / s) * b * q * sign(d) * 2 / (w dk) / C,
// with I1(b s) / s -> b / 2 as s -> 0; its power series in s^2 (kb_series).
__global__ void k_tap_grad_records(const double* __restrict__ k, const int* __restrict__ sample_idx, long long n,
                                   KbParams kb, TapRecord* __restrict__ out)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long g = sample_idx ? sample_idx[i] : i;
    TapRecord r;
    float* f = reinterpret_cast<float*>(&r);
    const float wHalf = (float)(kb.w / 2.0);
    int nearest[3];
    for (int a = 0; a < 3; ++a) {
        const int N = kb.G[a];
        const double ka = k[3 * g + a];
        const float dk = (float)(1.0 / (double)(float)(N - 1));
        int nr = (int)__dadd_rn(__dmul_rn((double)(N - 1), ka), 0.5);
        nr = nr < 0 ? 0 : (nr > N - 1 ? N - 1 : nr);
        nearest[a] = nr;
        for (int j = 0; j < TAPS_1D; ++j) {
            const int gi = nr - 2 + j;
            float val = 0.f;
            if (gi >= 0 && gi <= N - 1) {
                const double dd = ka - (double)__fmul_rn((float)gi, dk);
                const float d = (float)fabs(dd);
                if (!(d > wHalf * dk)) {
                    const float q = (float)(2.f * d) / (float)(kb.w * dk);
                    float dv = 0.f;
                    bool sure = kb.i1.nd > 0;
                    if (sure) {
                        const float2 p = kb_slope(kb, a, q);
                        dv = -p.x;
                        sure = pair_rounds(p);
                    }
                    if (!sure) {
                        const double s2 = __dadd_rn(1.0, -__dmul_rn((double)q, (double)q));
                        const double s = s2 > 0.0 ? sqrt(s2) : 0.0;
                        const double b = (double)kb.b;
                        const double i1s = s > 1e-12 ? cyl_bessel_i1(b * s) / s : 0.5 * b;
                        const double C = (double)(float)(100.0f * kb.w * dk);
                        dv = (float)(-i1s * b * (double)q * (2.0 / ((double)kb.w * (double)dk)) / C);
                    }
                    val = dd >= 0.0 ? dv : -dv;
                }
            }
            f[a * TAPS_1D + j] = val;
        }
    }
    f[15] = __uint_as_float(pack_nearest(nearest[0], nearest[1], nearest[2]));
    out[i] = r;
}

cudaError_t launch_tap_grad_records(const double* k, const int* sample_idx, long long n, const KbParams& kb,
                                    TapRecord* out, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_tap_grad_records<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(k, sample_idx, n, kb, out);
    return cudaGetLastError();
}

// One thread per sample of one bin; coils in chunks of CC.  Writes
//   rv[i][c]     = D_i r_ci          (the adjoint chain's samples), if rv
//   grad_k[g][a] = sum_c D_i Re(conj(r_ci) dy_ci/dk_a), g the global index
//   partials[b]  = sum over the block of 1/2 D_i |r_ci|^2
template <int CC>
__global__ void __launch_bounds__(128) k_interp_grad(InterpGradArgs a)
{
    __shared__ double s_red[4];
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double loss = 0.0;
    if (j < a.n) {
        const long long i = a.s0 + j;
        float w[15], dw[15];
        int nx, ny, nz, t0, t1, t2;
        load_record(a.rec, i, w, nx, ny, nz);
        load_record(a.drec, i, dw, t0, t1, t2);
        const float D = a.dcf ? a.dcf[i] : 1.f;
        const int Gy = a.G[1], Gz = a.G[2];
        float gk0 = 0.f, gk1 = 0.f, gk2 = 0.f;
        for (int c0 = 0; c0 < a.nch; c0 += CC) {
            const int ncc = min(CC, a.nch - c0);
            const float2* grid = a.grid + (long long)c0 * a.coil_stride;
            float2 y[CC], d0[CC], d1[CC], d2[CC];
#pragma unroll
            for (int c = 0; c < CC; ++c) y[c] = d0[c] = d1[c] = d2[c] = make_float2(0.f, 0.f);
#pragma unroll
            for (int jx = 0; jx < 5; ++jx) {
                const float wx = w[jx], dwx = dw[jx];
                if (wx == 0.f) continue;
                const int gx = nx - 2 + jx;
#pragma unroll
                for (int jy = 0; jy < 5; ++jy) {
                    const float wy = w[5 + jy], dwy = dw[5 + jy];
                    if (wy == 0.f) continue;
                    const long long row = ((long long)gx * Gy + (ny - 2 + jy)) * Gz + (nz - 2);
#pragma unroll
                    for (int jz = 0; jz < 5; ++jz) {
                        const float wz = w[10 + jz], dwz = dw[10 + jz];
                        const float wt = (wx * wy) * wz;
                        if (wz != 0.f && wt > a.thresh) {
                            const float ex = (dwx * wy) * wz, ey = (wx * dwy) * wz, ez = (wx * wy) * dwz;
#pragma unroll
                            for (int c = 0; c < CC; ++c)
                                if (c < ncc) {
                                    const float2 g = __ldg(grid + (long long)c * a.coil_stride + row + jz);
                                    y[c].x = fmaf(g.x, wt, y[c].x);
                                    y[c].y = fmaf(g.y, wt, y[c].y);
                                    d0[c].x = fmaf(g.x, ex, d0[c].x);
                                    d0[c].y = fmaf(g.y, ex, d0[c].y);
                                    d1[c].x = fmaf(g.x, ey, d1[c].x);
                                    d1[c].y = fmaf(g.y, ey, d1[c].y);
                                    d2[c].x = fmaf(g.x, ez, d2[c].x);
                                    d2[c].y = fmaf(g.y, ez, d2[c].y);
                                }
                        }
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < CC; ++c)
                if (c < ncc) {
                    const float2 m = a.ymeas[i * a.nch + c0 + c];
                    const float rx = y[c].x - m.x, ry = y[c].y - m.y;
                    loss += 0.5 * (double)D * ((double)rx * rx + (double)ry * ry);
                    gk0 += D * (rx * d0[c].x + ry * d0[c].y);
                    gk1 += D * (rx * d1[c].x + ry * d1[c].y);
                    gk2 += D * (rx * d2[c].x + ry * d2[c].y);
                    if (a.rv) a.rv[i * a.nch + c0 + c] = make_float2(D * rx, D * ry);
                }
        }
        if (a.grad_k) {
            const long long g = a.sorted[i];
            a.grad_k[3 * g + 0] = gk0;
            a.grad_k[3 * g + 1] = gk1;
            a.grad_k[3 * g + 2] = gk2;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = loss;
    __syncthreads();
    if (threadIdx.x == 0) a.partials[blockIdx.x] = s_red[0] + s_red[1] + s_red[2] + s_red[3];
}

// ---------------------------------------------------------------------------
// The same passes over the quad grid (fwd_x_quad.cuh): four lanes per sample,
// one coil of the quad each, so that a warp's load of one tap takes one
// 32-byte sector per sample.  A lane adds its coil's value and derivatives
// over the taps in the order of the kernels above with the same products and
// tests, and the coil sums run in coil order: the same bits.
//
// Bound by latency: registers decide how many warps hide it.  The 30 factors of
// a sample in every lane's registers, with the 125 taps unrolled, spilled 390
// bytes at seven blocks per SM; the x and y factors are now read from shared
// memory where they are used, eight taps' loads in flight at a time.  1 572 864
// samples, 12 coils: k_interp_grad 7.93 ms, this kernel with the factors in
// registers 2.36 ms, now 1.14 ms at eight blocks per SM.  Sixteen loads in flight
// at six blocks per SM cost 2 % of a loss evaluation more, four at eight 4 %,
// six or seven blocks with eight loads 5 and 1 %, the rows unrolled 13 %.
// ---------------------------------------------------------------------------
struct GradSums {
    float2 y, d0, d1, d2;
};

constexpr int QG_SAMPLES = 32;   // samples per block of 128 threads
// shared floats of a sample: (factor, derivative) pairs of x, then of y; eight
// samples this far apart fall in different banks
constexpr int QG_PITCH = 20;

// A sample's factors and their derivatives: along z in registers, along x and
// y in shared memory, which the sample's four lanes share.  Where all three
// supports of every sample of the warp hold exactly four candidates, these are
// moved to the positions 0 .. 3 of each axis (`four`), else candidates sit at
// 0 .. 4.
struct QuadTaps {
    float wz[5], dwz[5];
    const float* xy;
    long long base;   // grid point of candidate (0, 0, 0); may lie outside the grid unless four
    bool four;
};

// all 32 lanes of the warp; xy: the sample's shared floats
CGS_D void quad_taps(const TapRecord* rec, const TapRecord* drec, long long i, int Gy, int Gz, float* xy, QuadTaps& t)
{
    float w[15], dw[15];
    int nx, ny, nz, t0, t1, t2;
    load_record(rec, i, w, nx, ny, nz);
    load_record(drec, i, dw, t0, t1, t2);
    bool ok = true;
    int sh[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float* u = w + 5 * a;
        sh[a] = u[0] == 0.f;
        ok = ok && u[1] != 0.f && u[2] != 0.f && u[3] != 0.f && ((u[0] == 0.f) != (u[4] == 0.f));
    }
    t.four = __all_sync(0xffffffffu, ok);
    if (t.four) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                w[5 * a + q] = sh[a] ? w[5 * a + q + 1] : w[5 * a + q];
                dw[5 * a + q] = sh[a] ? dw[5 * a + q + 1] : dw[5 * a + q];
            }
        nx += sh[0];
        ny += sh[1];
        nz += sh[2];
    }
    t.base = ((long long)(nx - 2) * Gy + (ny - 2)) * Gz + (nz - 2);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        t.wz[q] = w[10 + q];
        t.dwz[q] = dw[10 + q];
    }
    if ((threadIdx.x & 3) == 0) {
#pragma unroll
        for (int q = 0; q < 10; ++q) *reinterpret_cast<float2*>(xy + 2 * q) = make_float2(w[q], dw[q]);
    }
    __syncwarp();
    t.xy = xy;
}

// (factor, derivative): read where it is used (volatile), so that the compiler
// does not keep the factors or the taps' weights across the coils; "memory", as
// the asm reads what quad_taps stored
CGS_D float2 xy_pair(const QuadTaps& t, int q)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(smem_addr(t.xy + 2 * q)) : "memory");
    return v;
}

// Value and coordinate derivatives of one coil at one sample; g: the coil's
// first point (points 4 apart)
template <int N>
CGS_D GradSums quad_grad_run(const float2* __restrict__ g, const QuadTaps& t, int Gy, int Gz, float thresh)
{
    GradSums r;
    r.y = r.d0 = r.d1 = r.d2 = make_float2(0.f, 0.f);
    const float2* b = g + t.base * 4;
#pragma unroll 1   // unrolled, the compiler keeps the planes' addresses across the coils and spills
    for (int jx = 0; jx < N; ++jx, b += (long long)Gy * Gz * 4) {
        const float2 fx = xy_pair(t, jx);
#pragma unroll 1
        for (int y0 = 0; y0 < N; y0 += N == 4 ? 2 : 1) {
            constexpr int NY = N == 4 ? 2 : 1;
            float2 v[NY][N];
#pragma unroll
            for (int q = 0; q < NY; ++q) {
                const float2* row = b + (long long)(y0 + q) * Gz * 4;
                const float wxy = N == 4 ? 0.f : fx.x * xy_pair(t, 5 + y0 + q).x;
#pragma unroll
                for (int jz = 0; jz < N; ++jz)   // with N = 4 every candidate lies in the grid
                    if (N == 4 || wxy * t.wz[jz] > thresh) v[q][jz] = __ldg(row + jz * 4);
            }
#pragma unroll
            for (int q = 0; q < NY; ++q) {
                const float2 fy = xy_pair(t, 5 + y0 + q);
                const float wxy = fx.x * fy.x, ax = fx.y * fy.x, ay = fx.x * fy.y;
#pragma unroll
                for (int jz = 0; jz < N; ++jz) {
                    const float wz = t.wz[jz], dwz = t.dwz[jz];
                    const float wt = wxy * wz;   // 0 outside the support or the grid
                    if (wt > thresh) {
                        const float ex = ax * wz, ey = ay * wz, ez = wxy * dwz;
                        r.y.x = fmaf(v[q][jz].x, wt, r.y.x);
                        r.y.y = fmaf(v[q][jz].y, wt, r.y.y);
                        r.d0.x = fmaf(v[q][jz].x, ex, r.d0.x);
                        r.d0.y = fmaf(v[q][jz].y, ex, r.d0.y);
                        r.d1.x = fmaf(v[q][jz].x, ey, r.d1.x);
                        r.d1.y = fmaf(v[q][jz].y, ey, r.d1.y);
                        r.d2.x = fmaf(v[q][jz].x, ez, r.d2.x);
                        r.d2.y = fmaf(v[q][jz].y, ez, r.d2.y);
                    }
                }
            }
        }
    }
    return r;
}
CGS_D GradSums quad_grad_sums(const float2* __restrict__ g, const QuadTaps& t, int Gy, int Gz, float thresh)
{
    return t.four ? quad_grad_run<4>(g, t, Gy, Gz, thresh) : quad_grad_run<5>(g, t, Gy, Gz, thresh);
}

__global__ void __launch_bounds__(4 * QG_SAMPLES, 8) k_interp_grad_quad(InterpGradArgs a)
{
    __shared__ double s_red[QG_SAMPLES / 8];
    __shared__ __align__(8) float s_xy[QG_SAMPLES * QG_PITCH];
    const int lane = threadIdx.x & 31, sub = threadIdx.x & 3, lead = lane & ~3;
    const long long j = (long long)blockIdx.x * QG_SAMPLES + threadIdx.x / 4;
    const bool on = j < a.n;
    double loss = 0.0;
    float gk0 = 0.f, gk1 = 0.f, gk2 = 0.f;
    const long long i = a.s0 + (on ? j : 0);
    if (a.n > 0) {
        QuadTaps t;
        quad_taps(a.rec, a.drec, i, a.G[1], a.G[2], s_xy + QG_PITCH * (threadIdx.x / 4), t);
        const float D = a.dcf ? a.dcf[i] : 1.f;
        for (int c0 = 0; c0 < a.nch; c0 += 4) {
            const int c = c0 + sub;
            const GradSums r = quad_grad_sums(a.grid + (long long)(c0 / 4) * a.coil_stride + sub, t, a.G[1], a.G[2],
                                              a.thresh);
            float p0 = 0.f, p1 = 0.f, p2 = 0.f;
            if (on && c < a.nch) {
                const float2 m = a.ymeas[i * a.nch + c];
                const float rx = r.y.x - m.x, ry = r.y.y - m.y;
                loss += 0.5 * (double)D * ((double)rx * rx + (double)ry * ry);
                p0 = rx * r.d0.x + ry * r.d0.y;
                p1 = rx * r.d1.x + ry * r.d1.y;
                p2 = rx * r.d2.x + ry * r.d2.y;
                if (a.rv) a.rv[i * a.nch + c] = make_float2(D * rx, D * ry);
            }
            // the quad's coils in order (every lane of the sample)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float b0 = __shfl_sync(0xffffffffu, p0, lead + q), b1 = __shfl_sync(0xffffffffu, p1, lead + q);
                const float b2 = __shfl_sync(0xffffffffu, p2, lead + q);
                if (c0 + q < a.nch) {
                    gk0 = fmaf(D, b0, gk0);
                    gk1 = fmaf(D, b1, gk1);
                    gk2 = fmaf(D, b2, gk2);
                }
            }
        }
        if (a.grad_k && on && sub < 3) a.grad_k[3 * (long long)a.sorted[i] + sub] = sub == 0 ? gk0 : sub == 1 ? gk1 : gk2;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) s_red[threadIdx.x >> 5] = loss;
    __syncthreads();
    if (threadIdx.x == 0) a.partials[blockIdx.x] = s_red[0] + s_red[1] + s_red[2] + s_red[3];
}

int interp_grad_blocks(long long n, bool quad)
{
    const int per = quad ? QG_SAMPLES : 128;
    return (int)std::max<long long>((n + per - 1) / per, 1);
}

cudaError_t launch_interp_grad(const InterpGradArgs& a, cudaStream_t s)
{
    if (a.quad) k_interp_grad_quad<<<(unsigned)interp_grad_blocks(a.n, true), 4 * QG_SAMPLES, 0, s>>>(a);
    else k_interp_grad<2><<<(unsigned)interp_grad_blocks(a.n, false), 128, 0, s>>>(a);
    return cudaGetLastError();
}

// Sum of the loss partials in one block, in a fixed order: one value to copy
// back instead of all of them.
__global__ void __launch_bounds__(1024) k_loss_sum(double* partials, int n)
{
    __shared__ double s[32];
    double v = 0.0;
    for (int i = threadIdx.x; i < n; i += 1024) v += partials[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = s[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) partials[0] = v;
    }
}

cudaError_t launch_loss_sum(double* partials, int n, cudaStream_t s)
{
    k_loss_sum<<<1, 1024, 0, s>>>(partials, n);
    return cudaGetLastError();
}

// Finiteness of device coordinates: *bad = 1 when any is NaN or Inf.
__global__ void k_check_finite(const double* __restrict__ v, long long n, int* bad)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && !isfinite(v[i])) atomicExch(bad, 1);
}

cudaError_t launch_check_finite(const double* v, long long n, int* bad, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_check_finite<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(v, n, bad);
    return cudaGetLastError();
}

// Values and coordinate derivatives of E S u at one bin's samples, then
// either stored (outA) or contracted with a stored pair (A, dA).  One thread
// per sample; coils in chunks of CC.
template <int CC>
__global__ void __launch_bounds__(128) k_pair_grad(PairGradArgs a)
{
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= a.n) return;
    const long long i = a.s0 + j;
    float w[15], dw[15];
    int nx, ny, nz, t0, t1, t2;
    load_record(a.rec, i, w, nx, ny, nz);
    load_record(a.drec, i, dw, t0, t1, t2);
    const float D = a.dcf ? a.dcf[i] : 1.f;
    const int Gy = a.G[1], Gz = a.G[2];
    float gk0 = 0.f, gk1 = 0.f, gk2 = 0.f;
    for (int c0 = 0; c0 < a.nch; c0 += CC) {
        const int ncc = min(CC, a.nch - c0);
        const float2* grid = a.grid + (long long)c0 * a.coil_stride;
        float2 y[CC], d0[CC], d1[CC], d2[CC];
#pragma unroll
        for (int c = 0; c < CC; ++c) y[c] = d0[c] = d1[c] = d2[c] = make_float2(0.f, 0.f);
#pragma unroll
        for (int jx = 0; jx < 5; ++jx) {
            const float wx = w[jx], dwx = dw[jx];
            if (wx == 0.f) continue;
            const int gx = nx - 2 + jx;
#pragma unroll
            for (int jy = 0; jy < 5; ++jy) {
                const float wy = w[5 + jy], dwy = dw[5 + jy];
                if (wy == 0.f) continue;
                const long long row = ((long long)gx * Gy + (ny - 2 + jy)) * Gz + (nz - 2);
#pragma unroll
                for (int jz = 0; jz < 5; ++jz) {
                    const float wz = w[10 + jz], dwz = dw[10 + jz];
                    const float wt = (wx * wy) * wz;
                    if (wz != 0.f && wt > a.thresh) {
                        const float ex = (dwx * wy) * wz, ey = (wx * dwy) * wz, ez = (wx * wy) * dwz;
#pragma unroll
                        for (int c = 0; c < CC; ++c)
                            if (c < ncc) {
                                const float2 g = __ldg(grid + (long long)c * a.coil_stride + row + jz);
                                y[c].x = fmaf(g.x, wt, y[c].x);
                                y[c].y = fmaf(g.y, wt, y[c].y);
                                d0[c].x = fmaf(g.x, ex, d0[c].x);
                                d0[c].y = fmaf(g.y, ex, d0[c].y);
                                d1[c].x = fmaf(g.x, ey, d1[c].x);
                                d1[c].y = fmaf(g.y, ey, d1[c].y);
                                d2[c].x = fmaf(g.x, ez, d2[c].x);
                                d2[c].y = fmaf(g.y, ez, d2[c].y);
                            }
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < CC; ++c)
            if (c < ncc) {
                const long long e = i * a.nch + c0 + c;
                if (a.outA) {
                    a.outA[e] = y[c];
                    a.outdA[3 * e + 0] = d0[c];
                    a.outdA[3 * e + 1] = d1[c];
                    a.outdA[3 * e + 2] = d2[c];
                } else {
                    // Re(conj(B) dA + conj(dB) A), B = y, dB = d*
                    const float2 A = a.A[e];
                    gk0 += A.x * d0[c].x + A.y * d0[c].y;
                    gk1 += A.x * d1[c].x + A.y * d1[c].y;
                    gk2 += A.x * d2[c].x + A.y * d2[c].y;
                    if (a.dA) {
                        const float2 e0 = a.dA[3 * e + 0], e1 = a.dA[3 * e + 1], e2 = a.dA[3 * e + 2];
                        gk0 += y[c].x * e0.x + y[c].y * e0.y;
                        gk1 += y[c].x * e1.x + y[c].y * e1.y;
                        gk2 += y[c].x * e2.x + y[c].y * e2.y;
                    }
                }
            }
    }
    if (!a.outA) {
        const long long g = a.sorted[i];
        const float f = a.scale * D;
        a.grad_k[3 * g + 0] += f * gk0;
        a.grad_k[3 * g + 1] += f * gk1;
        a.grad_k[3 * g + 2] += f * gk2;
    }
}

__global__ void __launch_bounds__(4 * QG_SAMPLES, 8) k_pair_grad_quad(PairGradArgs a)
{
    __shared__ __align__(8) float s_xy[QG_SAMPLES * QG_PITCH];
    const int lane = threadIdx.x & 31, sub = threadIdx.x & 3, lead = lane & ~3;
    const long long j = (long long)blockIdx.x * QG_SAMPLES + threadIdx.x / 4;
    const bool on = j < a.n;
    const long long i = a.s0 + (on ? j : 0);
    QuadTaps t;
    quad_taps(a.rec, a.drec, i, a.G[1], a.G[2], s_xy + QG_PITCH * (threadIdx.x / 4), t);
    const float D = a.dcf ? a.dcf[i] : 1.f;
    float gk[3] = {0.f, 0.f, 0.f};
    for (int c0 = 0; c0 < a.nch; c0 += 4) {
        const int c = c0 + sub;
        const GradSums r = quad_grad_sums(a.grid + (long long)(c0 / 4) * a.coil_stride + sub, t, a.G[1], a.G[2],
                                          a.thresh);
        const long long e = i * a.nch + c;
        const bool mine = on && c < a.nch;
        if (a.outA) {
            if (mine) {
                a.outA[e] = r.y;
                a.outdA[3 * e + 0] = r.d0;
                a.outdA[3 * e + 1] = r.d1;
                a.outdA[3 * e + 2] = r.d2;
            }
            continue;
        }
        // Re(conj(B) dA + conj(dB) A), B = y, dB = d*, each product pair rounded
        // as k_pair_grad rounds it
        float p[3] = {0.f, 0.f, 0.f}, q[3] = {0.f, 0.f, 0.f};
        if (mine) {
            const float2 A = a.A[e];
            p[0] = __fmaf_rn(A.x, r.d0.x, __fmul_rn(A.y, r.d0.y));
            p[1] = __fmaf_rn(A.x, r.d1.x, __fmul_rn(A.y, r.d1.y));
            p[2] = __fmaf_rn(A.x, r.d2.x, __fmul_rn(A.y, r.d2.y));
            if (a.dA) {
                const float2 e0 = a.dA[3 * e + 0], e1 = a.dA[3 * e + 1], e2 = a.dA[3 * e + 2];
                q[0] = __fmaf_rn(r.y.x, e0.x, __fmul_rn(r.y.y, e0.y));
                q[1] = __fmaf_rn(r.y.y, e1.y, __fmul_rn(r.y.x, e1.x));
                q[2] = __fmaf_rn(r.y.x, e2.x, __fmul_rn(r.y.y, e2.y));
            }
        }
        // the quad's coils in order (every lane of the sample)
#pragma unroll
        for (int l = 0; l < 4; ++l)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const float pl = __shfl_sync(0xffffffffu, p[d], lead + l), ql = __shfl_sync(0xffffffffu, q[d], lead + l);
                if (c0 + l < a.nch) {
                    gk[d] = __fadd_rn(gk[d], pl);
                    if (a.dA) gk[d] = __fadd_rn(gk[d], ql);
                }
            }
    }
    if (a.outA || !on || sub >= 3) return;
    const long long g = a.sorted[i];
    const float f = a.scale * D;
    const float sum = sub == 0 ? gk[0] : sub == 1 ? gk[1] : gk[2];
    a.grad_k[3 * g + sub] += f * sum;
}

cudaError_t launch_pair_grad(const PairGradArgs& a, cudaStream_t s)
{
    if (a.n == 0) return cudaSuccess;
    if (a.quad) {
        k_pair_grad_quad<<<(unsigned)((a.n + QG_SAMPLES - 1) / QG_SAMPLES), 4 * QG_SAMPLES, 0, s>>>(a);
        return cudaGetLastError();
    }
    k_pair_grad<2><<<(unsigned)((a.n + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

// Iterative density weights (Pipe and Menon, Magn. Reson. Med. 41:179-186,
// 1999): w <- w / (C * w) at the samples, C * w the interpolation of the
// spread weights.  v is the spread input (w, 0) and u the interpolated sum.
// A sample without any tap in the grid (C * w = 0) gets weight 0, as a hull
// sample's Voronoi cell does.
__global__ void k_pm_update(float* __restrict__ w, float2* __restrict__ v, const float2* __restrict__ u, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float c = u[i].x;
    const float nw = c > 0.f ? w[i] / c : 0.f;
    w[i] = nw;
    v[i] = make_float2(nw, 0.f);
}

cudaError_t launch_pm_update(float* w, float2* v, const float2* u, long long n, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_pm_update<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(w, v, u, n);
    return cudaGetLastError();
}

__global__ void k_pm_init(float* __restrict__ w, float2* __restrict__ v, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    w[i] = 1.f;
    if (v) v[i] = make_float2(1.f, 0.f);
}

cudaError_t launch_pm_init(float* w, float2* v, long long n, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_pm_init<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(w, v, n);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The same iteration over the transposed tap matrix.  The values are real, so
// the grid is one float a point; the spreading is a gather of each touched
// point's row (no other point is read), the interpolation ends with the
// update.  Sums run in the order of k_spread and k_interp with the same fused
// multiply-adds: the same weights bit for bit.  16 bins, 1 572 864 samples,
// grid 256 x 256 x 192, an iteration: k_spread 1.46 + k_interp 0.18 ms against
// 0.66 + 0.20 (the rows' scattered reads bound the gather); over slices, where
// the matrix is in that form (k_pm_slices), 0.31 + 0.20.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_pm_spread(PmArgs a)
{
    const int pts = a.G[0] * a.tb;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.nj * pts) return;
    const unsigned* p = a.ptr + a.j0 * pts + e;
    unsigned q = __ldg(p);
    const unsigned e1 = __ldg(p + 1);
    if (q == e1) return;
    float acc = 0.f;
    for (; q + 1 < e1; q += 2) {   // four or eight taps in flight: 0.83 ms
        const int2 u = __ldg(a.ent + q), v = __ldg(a.ent + q + 1);
        const float wu = __ldg(a.w + u.x), wv = __ldg(a.w + v.x);
        acc = fmaf(wu, __int_as_float(u.y), acc);
        acc = fmaf(wv, __int_as_float(v.y), acc);
    }
    if (q < e1) {
        const int2 u = __ldg(a.ent + q);
        acc = fmaf(__ldg(a.w + u.x), __int_as_float(u.y), acc);
    }
    const long long j = e / pts;
    const int i = (int)(e - j * pts), x = i / a.tb;
    const int2 t = a.tiles[a.j0 + j];
    a.grid[(long long)(t.x - a.bin0) * a.Ng + (long long)x * a.G[1] * a.G[2] + t.y + (i - x * a.tb)] = acc;
}

// One thread per sample; rows away from the ends of the grid are read as two
// aligned 16-byte loads (8 points from the multiple of 4 at or below the row).
__global__ void __launch_bounds__(128) k_pm_interp(PmArgs a)
{
    const int bin = a.bin0 + blockIdx.y;
    const long long s0 = a.bin_off[bin], s1 = a.bin_off[bin + 1];
    const long long i = s0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= s1) return;
    const float* grid = a.grid + (long long)blockIdx.y * a.Ng;   // Ng is a multiple of 4
    float w[15];
    int nx, ny, nz;
    load_record(a.rec, i, w, nx, ny, nz);
    const int Gy = a.G[1], Gz = a.G[2];
    float acc = 0.f;
#pragma unroll
    for (int jx = 0; jx < 5; ++jx) {
        const float wx = w[jx];
        if (wx == 0.f) continue;
#pragma unroll
        for (int jy = 0; jy < 5; ++jy) {
            const float wxy = wx * w[5 + jy];
            if (wxy == 0.f) continue;
            const long long row = ((long long)(nx - 2 + jx) * Gy + (ny - 2 + jy)) * Gz + (nz - 2);
            const long long r0 = row & ~3LL;
            float v[8];
            const bool vec = row >= 0 && r0 + 8 <= a.Ng;
            const int sh = vec ? (int)(row - r0) : 0;
            if (vec) {
                const float4 u0 = __ldg(reinterpret_cast<const float4*>(grid + r0));
                const float4 u1 = __ldg(reinterpret_cast<const float4*>(grid + r0) + 1);
                v[0] = u0.x; v[1] = u0.y; v[2] = u0.z; v[3] = u0.w;
                v[4] = u1.x; v[5] = u1.y; v[6] = u1.z; v[7] = u1.w;
            }
#pragma unroll
            for (int jz = 0; jz < 5; ++jz) {
                const float wz = w[10 + jz];
                const float wt = wxy * wz;
                if (wz != 0.f && wt > a.thresh) {
                    const float g = vec ? (sh == 0 ? v[jz] : sh == 1 ? v[jz + 1] : sh == 2 ? v[jz + 2] : v[jz + 3])
                                        : __ldg(grid + row + jz);
                    acc = fmaf(g, wt, acc);
                }
            }
        }
    }
    a.w[i] = acc > 0.f ? a.w[i] / acc : 0.f;
}

cudaError_t launch_pm_step(const PmArgs& a, long long max_bin, cudaStream_t s)
{
    const long long np = a.nj * a.G[0] * a.tb;
    if (np > 0) k_pm_spread<<<(unsigned)((np + 255) / 256), 256, 0, s>>>(a);
    return launch_pm_interp(a, max_bin, s);
}

cudaError_t launch_pm_interp(const PmArgs& a, long long max_bin, cudaStream_t s)
{
    if (max_bin > 0) k_pm_interp<<<dim3((unsigned)((max_bin + 127) / 128), (unsigned)a.nbins), 128, 0, s>>>(a);
    return cudaGetLastError();
}

// per bin the largest weight (weights are not negative: ordered as integers),
// and the last bin that holds each sample
__global__ void __launch_bounds__(256) k_pm_max(const float* __restrict__ w, const int* __restrict__ sorted,
                                                const long long* __restrict__ bin_off, unsigned* mx, int* owner)
{
    const int bin = blockIdx.y;
    unsigned m = 0;
    for (long long i = bin_off[bin] + (long long)blockIdx.x * blockDim.x + threadIdx.x; i < bin_off[bin + 1];
         i += (long long)gridDim.x * blockDim.x) {
        m = max(m, __float_as_uint(w[i]));
        atomicMax(owner + sorted[i], bin + 1);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(mx + bin, m);
}

__global__ void __launch_bounds__(256) k_pm_scatter(const float* __restrict__ w, const int* __restrict__ sorted,
                                                    const long long* __restrict__ bin_off, const unsigned* mx,
                                                    const int* owner, float* __restrict__ out)
{
    const int bin = blockIdx.y;
    const float m = __uint_as_float(mx[bin]);
    const float inv = m > 0.f ? 1.f / m : 0.f;
    for (long long i = bin_off[bin] + (long long)blockIdx.x * blockDim.x + threadIdx.x; i < bin_off[bin + 1];
         i += (long long)gridDim.x * blockDim.x)
        if (owner[sorted[i]] == bin + 1) out[sorted[i]] = w[i] * inv;
}

cudaError_t launch_pm_finish(const float* w, const int* sorted, const long long* bin_off, int nbins, long long max_bin,
                             long long ns, unsigned* mx, int* owner, float* out, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(mx, 0, (size_t)nbins * sizeof(unsigned), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(owner, 0, (size_t)ns * sizeof(int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(out, 0, (size_t)ns * sizeof(float), s);
    if (e != cudaSuccess || max_bin == 0) return e;
    const dim3 grid((unsigned)std::min<long long>((max_bin + 255) / 256, 1024), (unsigned)nbins);
    k_pm_max<<<grid, 256, 0, s>>>(w, sorted, bin_off, mx, owner);
    k_pm_scatter<<<grid, 256, 0, s>>>(w, sorted, bin_off, mx, owner, out);
    return cudaGetLastError();
}

}  // namespace cgs
