// fwd_x_quad.cuh -- forward x pass of the centred FFT (Fourier.cpp:19-42,
// sign -1) for four coils at a time, into a grid that holds the coils of a
// quad side by side.
//
// Layout of the forward grid: coils in quads, point p of quad q and coil
// 4 q + c at ((slot * nq + q) * Ng + p) * 4 + c (the last quad padded with
// zeros).  A point's four coils are one 32-byte sector, so
//   * the interpolation's lanes read whole sectors with nothing beside the
//     taps in them (a coil plane's 4-tap z run straddles two sectors);
//   * the pass can store exactly the points that some tap reads: of a listed
//     tile's points a wave-CAIPI bin touches about a quarter (a touch mask,
//     one bit per point, made from the transposed tap matrix).
//
// The arithmetic is k_fft_strided_tma's (the same codelets, twiddles and
// order on every line), so every stored value keeps its bits.
//
// A unit is TBQ columns x 4 coils; a block walks units round-robin.  The
// input rows of the four coils come by TMA into one stage, refilled for the
// next unit as soon as stage 1 has read it (two or more blocks per SM keep
// copies in flight meanwhile).  Stage 1 takes its threads column-fastest (as
// the input lies in shared memory), stage 2 coil-fastest (as the output lies
// in the grid); the exchange rows between them are XOR-swizzled so that both
// sides are free of bank conflicts.  Units of 8 columns (512 threads, two
// blocks per SM) where the input is half-pruned and the codelets have at most
// 16 points, else 4 (the longer codelets' registers, twice the input rows).
//
// Measured, 16 bins of 128 x 128 x 96, 12 coils (grid 256 x 256 x 192), against
// coil planes: this pass 2.83 -> 1.98 ms, the interpolation after it 3.19 ->
// 0.81 ms; one bin 245 -> 176 and 296 -> 72 us.  Bound by its exchange and
// codelets now: 7.4 GB in 1.98 ms is 3.7 TB/s.
#pragma once
#include "fft_passes.cuh"

namespace cgs {

template <int R1, int R2, int TBQ>
struct QuadLayout {
    static constexpr int L = R1 * R2;
    static constexpr int RM = R1 > R2 ? R1 : R2;
    static constexpr int W = 4 * TBQ;            // exchange row: coils x columns
    // thread groups of W: one per row group of the longer codelet's stage up to
    // 24, else 16, and a stage with more rows takes them in two turns.  A 28- or
    // 32-point codelet wants 128 registers: 16 W threads are two blocks per SM,
    // all busy in its stage, where RM W threads were one, half idle there.  20
    // coils of a 512 x 512 x 352 grid: 4.64 -> 3.33 ms (coil planes 3.98); 8
    // coils of 352, 448 and 512 x 192 x 192: 404, 355, 349 -> 232, 227, 229 us
    // (coil planes 301, 271, 286).  Images of more than 340 of 512 rows leave room
    // for one block (417 rows: 397 -> 438 us, coil planes 1006).
    static constexpr int NG = RM <= 24 ? RM : 16;
    static constexpr int NT = W * NG;
    static constexpr int T1 = (R2 + NG - 1) / NG, T2 = (R1 + NG - 1) / NG;   // turns of the two stages
    // resident blocks asked of the compiler: 64 to 102 registers a thread (two
    // of L = 320's blocks per SM instead of one: 1.31 -> 0.77 ms, 16 coils of
    // a 320 x 320 x 224 grid)
    static constexpr int MINB = RM <= 16 ? (NT <= 256 ? 3 : 2) : 2;
    static constexpr int R2W = (R2 + 3) / 4;     // mask words of a row group k1
    // the x rows of one coil, rounded up to 128 bytes
    __host__ __device__ static int coil_elems(int rows) { return (rows * TBQ + 15) & ~15; }
    static size_t smem_bytes(int rows)
    {
        return 128 + ((size_t)4 * coil_elems(rows) + (size_t)L * W + L + R2) * sizeof(float2) + sizeof(uint64_t);
    }
    // exchange slot of (coil, column) in a row n2: TBQ = 8 -> 32 slots, two
    // 128-byte halves; TBQ = 4 -> 16 slots
    CGS_D static int slot(int coil, int col, int n2)
    {
        if (TBQ == 8) return (coil * 8 + (col ^ ((coil & 2) << 1))) ^ ((n2 & 1) << 3);
        return (coil * 4 + col) ^ ((n2 & 3) << 2);
    }
};

template <int R1, int R2, int TBQ, int MODE>
__global__ void __launch_bounds__(QuadLayout<R1, R2, TBQ>::NT,
                                  QuadLayout<R1, R2, TBQ>::MINB)
k_fwd_x_quad(FwdXQuadArgs a, const __grid_constant__ CUtensorMap tmap, int nunits, int per_quad, int nsub,
             int box_rows, int nbox)
{
    using Q = QuadLayout<R1, R2, TBQ>;
    constexpr int L = Q::L, NT = Q::NT, W = Q::W, SIGN = -1;
    constexpr bool FOLD = SignFold<R1, R2>::value;
    static_assert(TBQ == 4 || TBQ == 8, "exchange swizzle");
    static_assert(MODE != PRUNE_IN || R1 % 4 == 0, "input pruning needs R1 % 4 == 0");
    extern __shared__ float4 s_pipe[];
    const uint32_t pad = (128u - (smem_addr(s_pipe) & 127u)) & 127u;
    const int ce = Q::coil_elems(box_rows * nbox);
    float2* s_in = reinterpret_cast<float2*>(reinterpret_cast<char*>(s_pipe) + pad);   // [coil][row][TBQ]
    float2* s_y = s_in + 4 * ce;                                                       // [k1][n2][slot]
    float2* s_tw = s_y + L * W;
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(s_tw + L + R2);
    __shared__ int4 s_unit[2];   // {first coil, workspace slot, first column, mask entry}
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
    if (tid == 0) {
        mbar_init(s_bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    const int my_n = nunits > (int)blockIdx.x ? (nunits - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const int nq = (a.nch + 3) / 4;

    auto issue = [&](int k) {   // thread 0 only
        const int u = (int)blockIdx.x + k * (int)gridDim.x;
        const int q = u / per_quad, rem = u - q * per_quad;   // quads outer: blocks in flight share coil planes
        const int t = rem / nsub, s = rem - t * nsub;
        int slot, b0;
        if (a.tiles) {
            const int2 e = a.tiles[t];
            slot = e.x - a.bin0;
            b0 = e.y + s * TBQ;
        } else {
            slot = t;
            b0 = s * TBQ;
        }
        s_unit[k & 1] = make_int4(4 * q, slot, b0, rem);
        const int nc = min(4, a.nch - 4 * q);
        mbar_arrive_expect_tx(s_bar, (uint32_t)(nc * nbox * box_rows * TBQ) * (uint32_t)sizeof(float2));
        for (int c = 0; c < nc; ++c)
            for (int r = 0; r < nbox; ++r)
                tma_load_4d(s_in + c * ce + r * box_rows * TBQ, &tmap, b0, r * box_rows, 0,
                            slot * a.nch + 4 * q + c, s_bar);
    };

    // stage 1: column fastest, then n2, then coil; stage 2: coil fastest, then column, then k1
    const int col1 = tid % TBQ, g1 = tid / TBQ;
    const int coil1a = g1 / R2, n2a = g1 - coil1a * R2;   // of the first turn
    const int slot1a = Q::slot(coil1a & 3, col1, n2a);
    const int coil2 = tid & 3, col2 = (tid >> 2) % TBQ, k1a = tid / W;
    auto load_mask = [&](uint32_t (&mw)[Q::R2W], int entry, int k1) {
        if (a.mask) {
            const uint32_t* m = a.mask + ((long long)entry * R1 + k1) * Q::R2W;
            if constexpr (Q::R2W % 4 == 0) {
#pragma unroll
                for (int w = 0; w < Q::R2W / 4; ++w) {
                    const uint4 v4 = __ldg(reinterpret_cast<const uint4*>(m) + w);
                    mw[4 * w] = v4.x;
                    mw[4 * w + 1] = v4.y;
                    mw[4 * w + 2] = v4.z;
                    mw[4 * w + 3] = v4.w;
                }
            } else {
#pragma unroll
                for (int w = 0; w < Q::R2W; ++w) mw[w] = __ldg(m + w);
            }
        } else {
#pragma unroll
            for (int w = 0; w < Q::R2W; ++w) mw[w] = 0xffffffffu;
        }
    };

    if (tid == 0 && my_n > 0) issue(0);
    for (int k = 0; k < my_n; ++k) {
        const bool ok = mbar_wait_bounded(s_bar, (uint32_t)(k & 1), PIPE_WAIT_NS);
        if (__syncthreads_or(!ok)) {
            // timeout: report, let the copies already issued land, leave
            if (tid == 0) {
                atomicExch(a.err, 1);
                mbar_wait_bounded(s_bar, (uint32_t)(k & 1), PIPE_WAIT_NS);
            }
            return;
        }
        const int4 un = s_unit[k & 1];
        // touch-mask bytes of a row group k1 (one per k2, a bit per column), of the first turn ahead
        uint32_t mw[Q::R2W];
        load_mask(mw, un.w, k1a < R1 ? k1a : 0);
#pragma unroll 1
        for (int turn = 0; turn < Q::T1; ++turn) {
            const int coil1 = turn == 0 ? coil1a : (g1 + turn * (NT / TBQ)) / R2;
            const int n2 = turn == 0 ? n2a : g1 + turn * (NT / TBQ) - coil1 * R2;
            if (coil1 >= 4) break;
            const int slot1 = turn == 0 ? slot1a : Q::slot(coil1, col1, n2);
            float2 v[R1];
            if (un.x + coil1 >= a.nch) {
                // a padding coil of the last quad: zeros
#pragma unroll
                for (int q = 0; q < R1; ++q) v[q] = make_float2(0.f, 0.f);
            } else {
                const float2* src = s_in + coil1 * ce + col1;
                if constexpr (MODE == PRUNE_IN) {
#pragma unroll
                    for (int n1 = 0; n1 < R1; ++n1) {
                        if (n1 >= R1 / 4 && n1 < 3 * R1 / 4) {
                            const float2 x = src[(n2 + R2 * (n1 - R1 / 4)) * TBQ];
                            v[n1] = FOLD ? x : parity(x, R2 * n1 + n2);
                        } else {
                            v[n1] = make_float2(0.f, 0.f);
                        }
                    }
                    DftMid<R1, SIGN>::run(v);
                } else {
#pragma unroll
                    for (int n1 = 0; n1 < R1; ++n1) {
                        const int l = R2 * n1 + n2;
                        const int li = l - a.in_off;
                        float2 x = make_float2(0.f, 0.f);
                        if (li >= 0 && li < a.Lin) x = src[li * TBQ];
                        v[n1] = FOLD ? x : parity(x, l);
                    }
                    Dft<R1, SIGN>::run(v);
                }
            }
#pragma unroll
            for (int q = 0; q < R1; ++q) {
                float2 tv = v[q];
                if (FOLD) tv = table_twiddle<SIGN>(tv, s_tw[n2 * (R1 + 1) + q]);
                else if (q > 0) tv = table_twiddle<SIGN>(tv, s_tw[n2 * q]);
                s_y[(q * R2 + n2) * W + slot1] = tv;
            }
        }
        __syncthreads();
        if (tid == 0 && k + 1 < my_n) {
            fence_proxy_async_smem();
            issue(k + 1);
        }
#pragma unroll 1
        for (int turn = 0; turn < Q::T2; ++turn) {
            const int k1 = k1a + turn * Q::NG;
            if (k1 >= R1) break;
            if (turn > 0) load_mask(mw, un.w, k1);
            float2 u[R2];
#pragma unroll
            for (int m = 0; m < R2; ++m) u[m] = s_y[(k1 * R2 + m) * W + Q::slot(coil2, col2, m)];
            Dft<R2, SIGN>::run(u);
            const int b = un.z + col2;
            if (b < a.B) {
                float2* o = a.out + (((long long)un.y * nq + (un.x >> 2)) * a.Ng + (long long)k1 * a.B + b) * 4 + coil2;
                const long long step = (long long)R1 * a.B * 4;
#pragma unroll
                for (int k2 = 0; k2 < R2; ++k2)
                    if ((mw[k2 / 4] >> ((k2 & 3) * 8 + col2)) & 1u)
                        o[k2 * step] = FOLD ? u[k2] : parity(u[k2], k1 + R1 * k2);
            }
        }
        // the next wait's barrier orders these reads of s_y before the next stage 1
    }
}

}  // namespace cgs
