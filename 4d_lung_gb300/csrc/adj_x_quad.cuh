// adj_x_quad.cuh -- adjoint x pass of the centred FFT (Fourier.cpp:19-42,
// sign +1) from the quad grid (fwd_x_quad.cuh) that the sliced gather
// (k_spread_quad, spread_csr.cu) fills: of the listed tiles only the touched
// points hold values, and only those are read.
//
// A unit is TBQ columns x 4 coils.  Stage 1 loads its rows straight from the
// grid into registers, coil fastest (a point's four coils are one 32-byte
// sector), row by row where the line mask has a bit; all of a thread's loads
// are in flight together, so the pass needs no staging, and 73 % of the
// points of a wave-CAIPI bin's tiles are not read at all.  Stage 2 stores the
// kept rows per coil plane, column fastest.  The arithmetic is
// k_fft_strided_tma's, so every value keeps its bits.  The gather and this pass
// take 1.33 + 2.32 ms on 16 bins of 128 x 128 x 96, 12 coils, against 4.05 ms
// for the two fused in one block per SM (spread_adjx.cuh), whose gather and
// transform both waited on the same shared-memory pipe.
#pragma once
#include "fwd_x_quad.cuh"

namespace cgs {

template <int R1, int R2, int TBQ>
struct AdjQuadLayout {
    using Q = QuadLayout<R1, R2, TBQ>;
    static constexpr int NT = Q::NT;
    // blocks of 256 threads, four per SM (64 registers): their loads and
    // transforms overlap better than two blocks of 8 columns (16 bins of the
    // 256 x 256 x 192 grid, 12 coils: 2.43 -> 2.32 ms; three blocks 2.47).  Lines
    // of 352, 448 and 512 points: 8 columns (fft_adj_quad_tile_cols), 512 threads
    // of 128 registers, the stage of more than 16 rows in two turns.
    static constexpr int MINB = Q::RM <= 16 ? 4 : Q::NT > 384 ? 1 : Q::MINB;
    static constexpr size_t smem_bytes = ((size_t)Q::L * Q::W + Q::L + R2) * sizeof(float2);
};

template <int R1, int R2, int TBQ, int MODE>
__global__ void __launch_bounds__(AdjQuadLayout<R1, R2, TBQ>::NT, AdjQuadLayout<R1, R2, TBQ>::MINB)
k_adj_x_quad(AdjXQuadArgs a, int nunits, int per_quad, int nsub)
{
    using Q = QuadLayout<R1, R2, TBQ>;
    constexpr int L = Q::L, NT = Q::NT, W = Q::W, SIGN = +1;
    constexpr bool FOLD = SignFold<R1, R2>::value;
    static_assert(MODE != PRUNE_OUT || R2 % 4 == 0, "output pruning needs R2 % 4 == 0");
    extern __shared__ float4 s_adjq[];
    float2* s_y = reinterpret_cast<float2*>(s_adjq);   // [k1][n2][slot]
    float2* s_tw = s_y + L * W;
    const int tid = threadIdx.x;
    if (FOLD) {
        for (int m = tid; m < L; m += NT) {
            const int n2 = m / R1, k1 = m - n2 * R1;
            const float2 w = a.tw[n2 * k1];
            s_tw[n2 * (R1 + 1) + k1] = ((n2 + k1) & 1) ? cneg(w) : w;
        }
    } else {
        for (int m = tid; m < L; m += NT) s_tw[m] = a.tw[m];
    }
    __syncthreads();
    const int nq = (a.nch + 3) / 4;
    // stage 1: coil fastest, then column, then n2; stage 2: column fastest, then k1, then coil
    const int coil1 = tid & 3, col1 = (tid >> 2) % TBQ, n2 = tid / W;
    const int col2 = tid % TBQ, g2 = tid / TBQ;
    const int coil2a = g2 / R1, k1sa = g2 - coil2a * R1;   // of the first turn
    for (int u = blockIdx.x; u < nunits; u += gridDim.x) {
        const int q = u / per_quad, rem = u - q * per_quad;   // quads outer, as the forward pass
        const int t = rem / nsub, s = rem - t * nsub;
        const int2 e = a.tiles[t];
        const int nc = min(4, a.nch - 4 * q);
        const long long slot = e.x - a.bin0;
        const int b0 = e.y + s * TBQ;
        auto rows = [&](float2 (&v)[R1], int n2) {
#pragma unroll
            for (int n1 = 0; n1 < R1; ++n1) v[n1] = make_float2(0.f, 0.f);
            if (coil1 < nc) {
                const unsigned m = __ldg(a.lmask + ((a.j0 + t) * R2 + n2) * a.tb + s * TBQ + col1);
                const float2* src = a.in + ((slot * nq + q) * a.Ng + (long long)n2 * a.B + b0 + col1) * 4 + coil1;
                const long long step = (long long)R2 * a.B * 4;
#pragma unroll
                for (int n1 = 0; n1 < R1; ++n1)
                    if ((m >> n1) & 1u) v[n1] = __ldg(src + n1 * step);
            }
            if (!FOLD) {
#pragma unroll
                for (int n1 = 0; n1 < R1; ++n1) v[n1] = parity(v[n1], R2 * n1 + n2);
            }
            Dft<R1, SIGN>::run(v);
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) {
                float2 tv = v[k1];
                if (FOLD) tv = table_twiddle<SIGN>(tv, s_tw[n2 * (R1 + 1) + k1]);
                else if (k1 > 0) tv = table_twiddle<SIGN>(tv, s_tw[n2 * k1]);
                v[k1] = tv;
            }
        };
        auto put = [&](const float2 (&v)[R1], int n2) {
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) s_y[(k1 * R2 + n2) * W + Q::slot(coil1, col1, k1)] = v[k1];
        };
        float2 v[R1];
        if (n2 < R2) rows(v, n2);
        // the exchange is free once every thread has left stage 2 of the last unit
        __syncthreads();
        if (n2 < R2) put(v, n2);
#pragma unroll 1
        for (int turn = 1; turn < Q::T1; ++turn) {
            const int m2 = n2 + turn * Q::NG;
            if (m2 >= R2) break;
            rows(v, m2);
            put(v, m2);
        }
        __syncthreads();
#pragma unroll 1
        for (int turn = 0; turn < Q::T2; ++turn) {
            const int coil2 = turn == 0 ? coil2a : (g2 + turn * (NT / TBQ)) / R1;
            const int k1s = turn == 0 ? k1sa : g2 + turn * (NT / TBQ) - coil2 * R1;
            if (coil2 >= nc) break;
            float2 w[R2];
#pragma unroll
            for (int m = 0; m < R2; ++m) w[m] = s_y[(k1s * R2 + m) * W + Q::slot(coil2, col2, k1s)];
            Dft<R2, SIGN>::run(w);
            const int b = b0 + col2;
            if (b < a.B) {
                float2* out = a.out + (slot * a.nch + 4 * q + coil2) * a.out_bs + b;
                if constexpr (MODE == PRUNE_OUT) {
                    float2* o = out + (long long)k1s * a.B;
                    const long long step = (long long)R1 * a.B;
#pragma unroll
                    for (int k2 = R2 / 4; k2 < 3 * R2 / 4; ++k2)
                        o[(k2 - R2 / 4) * step] = FOLD ? w[k2] : parity(w[k2], k1s + R1 * k2);
                } else {
#pragma unroll
                    for (int k2 = 0; k2 < R2; ++k2) {
                        const int l = k1s + R1 * k2, lo = l - a.out_off;
                        if (lo >= 0 && lo < a.Lout) out[(long long)lo * a.B] = FOLD ? w[k2] : parity(w[k2], l);
                    }
                }
            }
        }
    }
}

}  // namespace cgs
