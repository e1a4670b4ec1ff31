// Back-transformation of the sectors of order <= 128, for the one-block eigensolvers.
#pragma once
#include "cta_gemm.cuh"

namespace {

constexpr int kNB = 32;           // reflectors per panel
constexpr int kBtThreads = 512;

// Back-transformation V = Q Z with Q = H_0 ... H_{n-2}, 32 reflectors at a time (compact
// WY form), n <= 128.  Every warp keeps eight columns of Z in registers, transposed, as the
// accumulators of its MMA tiles; the three products of a panel, W^T = Z^T V, W2^T = W^T T^T
// and Z^T -= W2^T V^T, hand their accumulators on as A operands.  An accumulator's columns
// 2 q, 2 q + 1 of a lane are taken as the k index q of two MMAs (the order of a sum's terms
// is free), so no product's result moves between lanes: only V and T come from shared memory
// and the warps never wait for one another.  Bound by the FP64 MMA rate of one SM (2 n^3
// operations, 17 us at n = 128).
constexpr int kMaxN = 128;                       // order
constexpr int kLdV = kMaxN + 4;                  // Vs[k * kLdV + row]; = 4 mod 16
constexpr int kLdT = kNB + 4;                    // Ts[q][k * kLdT + n] = T_q(n, k); Gs alike
constexpr int kPanels = kMaxN / kNB;
constexpr size_t kBtSmem = sizeof(double) * (kMaxN * kLdV + 2 * kPanels * kNB * kLdT);

// row (or reflector) of position i of an 8-wide tile, so that a lane's accumulator columns
// 2 q, 2 q + 1 are rows q and q + 4
__device__ __forceinline__ int tile_pos(int i) { return (i >> 1) + 4 * (i & 1); }

__device__ void back_transform(double* A, int n, const double* TAU, const double* Z, double* sm) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q4 = lane & 3;
    double* Vs = sm;
    double* Ts = Vs + kMaxN * kLdV;
    double* Gs = Ts + kPanels * kNB * kLdT;
    const int nr = n - 1, np = (nr + kNB - 1) / kNB, nt = (n + 7) / 8;
    // the reflectors of every panel (zeros above, beyond n and beyond the last one)
    for (int k = warp; k < np * kNB; k += kBtThreads / 32)
        for (int row = lane; row < 8 * nt; row += 32)
            Vs[k * kLdV + row] = k >= nr || row >= n || row <= k ? 0.0 : (row == k + 1 ? 1.0 : A[(size_t)row + (size_t)k * n]);
    __syncthreads();
    // Gram matrices G_q = V_q^T V_q, four warps per panel, one row of 8 x 8 tiles each
    {
        const int q = warp >> 2, r = warp & 3;
        if (q < np) {
            double acc[4][2];
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[c][0] = acc[c][1] = 0.0;
            for (int i0 = kNB * q; i0 < 8 * nt; i0 += 4) {
                const double a = Vs[(kNB * q + 8 * r + g) * kLdV + i0 + q4];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (c >= r) nrg::cta_dmma(acc[c][0], acc[c][1], a, Vs[(kNB * q + 8 * c + g) * kLdV + i0 + q4]);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (c >= r)
#pragma unroll
                    for (int h = 0; h < 2; ++h) Gs[q * kNB * kLdT + (8 * r + g) * kLdT + 8 * c + 2 * q4 + h] = acc[c][h];
        }
    }
    __syncthreads();
    // T_q (dlarft, forward, columnwise): one warp per panel, row `lane` of T in registers
    if (warp < np) {
        const double* G = Gs + warp * kNB * kLdT;
        double* T = Ts + warp * kNB * kLdT;
        double row[kNB];
#pragma unroll
        for (int c = 0; c < kNB; ++c) {
            const int k = kNB * warp + c;
            const double tc = k < nr ? TAU[k] : 0.0;
            double s[2] = {0.0, 0.0};
#pragma unroll
            for (int q = 0; q < c; ++q) s[q & 1] = fma(row[q], G[q * kLdT + c], s[q & 1]);
            row[c] = lane == c ? tc : (lane < c ? -tc * (s[0] + s[1]) : 0.0);
            T[c * kLdT + lane] = row[c];
        }
    }
    __syncthreads();
    // this warp's columns
    const int col = 8 * warp + g;
    double z[kMaxN / 8][2];
#pragma unroll
    for (int t = 0; t < kMaxN / 8; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = 8 * t + q4 + 4 * h;
            z[t][h] = t < nt && row < n && col < n ? Z[(size_t)row + (size_t)col * n] : 0.0;
        }
    if (8 * warp < n) {
        for (int q = np - 1; q >= 0; --q) {
            const double* V = Vs + kNB * q * kLdV;
            const double* T = Ts + q * kNB * kLdT;
            double w[4][2], w2[4][2];
#pragma unroll
            for (int c = 0; c < 4; ++c) w[c][0] = w[c][1] = w2[c][0] = w2[c][1] = 0.0;
#pragma unroll
            for (int t = 0; t < kMaxN / 8; ++t)
                if (t >= 4 * q && t < nt) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            nrg::cta_dmma(w[c][0], w[c][1], z[t][h], V[(8 * c + tile_pos(g)) * kLdV + 8 * t + q4 + 4 * h]);
                }
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int d = 0; d < 4; ++d)
                        if (d <= c) nrg::cta_dmma(w2[d][0], w2[d][1], w[c][h], T[(8 * c + q4 + 4 * h) * kLdT + 8 * d + tile_pos(g)]);
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int h = 0; h < 2; ++h) w2[c][h] = -w2[c][h];
#pragma unroll
            for (int t = 0; t < kMaxN / 8; ++t)
                if (t >= 4 * q && t < nt) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            nrg::cta_dmma(z[t][0], z[t][1], w2[c][h], V[(8 * c + q4 + 4 * h) * kLdV + 8 * t + tile_pos(g)]);
                }
        }
#pragma unroll
        for (int t = 0; t < kMaxN / 8; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = 8 * t + q4 + 4 * h;
                if (t < nt && row < n && col < n) A[(size_t)row + (size_t)col * n] = z[t][h];
            }
    }
}

}  // namespace
