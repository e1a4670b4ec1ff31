// FP64 eigensolver for the large symmetry sectors of one iteration (order > 128), spread
// over the whole GPU instead of one block per sector.  All large sectors advance together:
//   1. Householder tridiagonalisation (eig_tri.cu): orders up to 512 with the matrix on
//      chip, larger ones streamed from L2 until the trailing block fits there.  Orders
//      beyond the streaming kernel's shared memory (about 3,600) take the kernels below,
//      blocked by panels of 32 columns (the dlatrd scheme): per column one block per sector
//      updates the column with the pending panel reflectors and forms the Householder
//      vector, then a many-block kernel computes the symmetric matrix-vector product with
//      the trailing matrix (column dot products, coalesced); after each panel the trailing
//      matrix takes the rank-64 update A -= [V W][W V]^T as one grouped GEMM;
//   2. divide and conquer: merges up to 128 rows inside one block per sector; larger
//      merges in phases (deflation, secular roots, Gu-Eisenstat z, rank-one eigenvectors,
//      final order) with the eigenvector update Z(:, kept) * U as a grouped GEMM;
//   3. back-transformation in panels of 64 reflectors: Gram matrix and V^T Z as grouped
//      GEMMs, the triangular factor T in one block, then Z -= (V T)(V^T Z).
#include "eig_dc.cuh"
#include "internal.hpp"


#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>


namespace {

constexpr int NB = 32;        // tridiagonalisation panel
constexpr int NBB = 64;       // back-transformation panel
constexpr int DC_LOW = kDcLeafRows;   // merges of up to this many rows run inside one block
constexpr int TPB = 256;
constexpr int CB = 32;        // columns per block in the symmetric matrix-vector product

struct LSec {
    long long a_off, e_off, w_off, i_off;
    int n, pad;
};

// workspace per sector: Z, U, Qt (n x n each), the panel V | W (n x 2 NB), y, the D&C
// vectors (16 n + 64), then the back-transformation's T factors and explicit reflector
// panels ((n + NBB)^2 bounds both)
long long lws_doubles(long long n) {
    return 3 * n * n + 2LL * NB * n + n + 16 * n + 64 + (n + NBB) * (n + NBB);
}
long long lws_ints(long long n) { return 12 * n + 64; }

struct LView {
    double *A, *Z, *U, *Qt, *VW, *y, *vec, *D, *E, *TAU, *R;
    int* I;
    Scratch S;
    int n;
};

__device__ LView lview(const LSec& s, double* eigbuf, double* wsd, int* wsi) {
    LView v;
    const long long n = s.n, sq = n * n;
    v.n = s.n;
    v.A = eigbuf + s.a_off;
    double* W = wsd + s.w_off;
    v.Z = W;
    v.U = W + sq;
    v.Qt = W + 2 * sq;
    v.VW = W + 3 * sq;
    v.y = v.VW + 2LL * NB * n;
    v.vec = v.y + n;
    v.D = v.vec;
    v.E = v.vec + n;
    v.TAU = v.vec + 2 * n;
    v.R = v.vec + 16 * n + 64;
    v.I = wsi + s.i_off;
    v.S = scratch_at(v.vec, v.I, s.n);
    return v;
}

// ---------------------------------------------------------------------------------
// tridiagonalisation
// ---------------------------------------------------------------------------------

// W(:, jj) for column c of the panel (rows c+1..n-1): dlatrd's w update
__device__ void finish_w(LView& L, int c, int jj, const double* t1s, double* t1, double* t2, double* red) {
    (void)t1s;
    const int n = L.n, tid = threadIdx.x, T = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nw = T >> 5;
    const double* V = L.VW;
    double* W = L.VW + (size_t)NB * n;
    const double* v = V + (size_t)jj * n;
    for (int q = warp; q < 2 * jj; q += nw) {
        const double* col = q < jj ? W + (size_t)q * n : V + (size_t)(q - jj) * n;
        double s = 0.0;
        for (int i = c + 1 + lane; i < n; i += 32) s = fma(col[i], v[i], s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) { if (q < jj) t1[q] = s; else t2[q - jj] = s; }
    }
    __syncthreads();
    const double tau = L.TAU[c];
    double* w = W + (size_t)jj * n;
    double part = 0.0;
    for (int i = c + 1 + tid; i < n; i += T) {
        double s = L.y[i];
        for (int q = 0; q < jj; ++q) s -= V[i + (size_t)q * n] * t1[q] + W[i + (size_t)q * n] * t2[q];
        s *= tau;
        w[i] = s;
        part += s * v[i];
    }
    const double wv = block_sum(part, red);
    const double al = -0.5 * tau * wv;
    for (int i = c + 1 + tid; i < n; i += T) w[i] += al * v[i];
    __syncthreads();
}

__global__ void __launch_bounds__(TPB) k_tri_col(const LSec* __restrict__ secs, int k, double* eigbuf,
                                                 double* wsd, int* wsi) {
    __shared__ double red[32];
    __shared__ double t1[NB], t2[NB];
    const LSec sec = secs[blockIdx.x];
    if (k > sec.n - 2) return;
    LView L = lview(sec, eigbuf, wsd, wsi);
    const int n = L.n, tid = threadIdx.x, T = blockDim.x;
    const int j = k % NB;
    if (j > 0) finish_w(L, k - 1, j - 1, nullptr, t1, t2, red);
    double* V = L.VW;
    double* W = L.VW + (size_t)NB * n;
    double* col = L.A + (size_t)k * n;
    // column k takes the pending updates of the panel's first j reflectors
    for (int i = k + tid; i < n; i += T) {
        double s = 0.0;
        for (int q = 0; q < j; ++q)
            s += V[i + (size_t)q * n] * W[k + (size_t)q * n] + W[i + (size_t)q * n] * V[k + (size_t)q * n];
        col[i] -= s;
    }
    __syncthreads();
    if (tid == 0) L.D[k] = col[k];
    const double alpha = col[k + 1];
    double part = 0.0;
    for (int i = k + 2 + tid; i < n; i += T) part += col[i] * col[i];
    const double xn2 = block_sum(part, red);
    double* v = V + (size_t)j * n;
    if (xn2 == 0.0) {
        for (int i = k + 1 + tid; i < n; i += T) v[i] = (i == k + 1) ? 1.0 : 0.0;
        if (tid == 0) { L.E[k] = alpha; L.TAU[k] = 0.0; }
        return;
    }
    const double beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
    const double tt = (beta - alpha) / beta;
    const double scal = 1.0 / (alpha - beta);
    for (int i = k + 1 + tid; i < n; i += T) {
        double vi = 1.0;
        if (i > k + 1) { vi = col[i] * scal; col[i] = vi; }
        v[i] = vi;
    }
    if (tid == 0) { L.E[k] = beta; L.TAU[k] = tt; }
}

// y(i) = sum_{l > k} A(l, i) v(l) for i > k: one warp per column, CB columns per block
__global__ void __launch_bounds__(TPB) k_tri_symv(const LSec* __restrict__ secs, int nsec, int k,
                                                  double* eigbuf, double* wsd, int* wsi) {
    extern __shared__ double vsm[];
    // find this block's sector among those still active at column k
    int s = 0, base = 0;
    for (; s < nsec; ++s) {
        const int n = secs[s].n;
        if (k > n - 2) continue;
        const int nb = (n - k - 1 + CB - 1) / CB;
        if ((int)blockIdx.x < base + nb) break;
        base += nb;
    }
    if (s >= nsec) return;
    LView L = lview(secs[s], eigbuf, wsd, wsi);
    const int n = L.n, m = n - k - 1;
    const int j = k % NB;
    const double* v = L.VW + (size_t)j * n + (k + 1);
    for (int i = threadIdx.x; i < m; i += blockDim.x) vsm[i] = v[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int c0 = ((int)blockIdx.x - base) * CB;
    for (int cc = warp; cc < CB; cc += nw) {
        const int ci = c0 + cc;
        if (ci >= m) break;
        const double* col = L.A + (size_t)(k + 1 + ci) * n + (k + 1);
        double s0 = 0.0, s1 = 0.0;
        int l = lane;
        for (; l + 32 < m; l += 64) {
            s0 = fma(col[l], vsm[l], s0);
            s1 = fma(col[l + 32], vsm[l + 32], s1);
        }
        if (l < m) s0 = fma(col[l], vsm[l], s0);
        double sum = s0 + s1;
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) L.y[k + 1 + ci] = sum;
    }
}

// W for the last column a sector processed in the panel starting at p
__global__ void __launch_bounds__(TPB) k_tri_finish(const LSec* __restrict__ secs, int p, double* eigbuf,
                                                    double* wsd, int* wsi) {
    __shared__ double red[32];
    __shared__ double t1[NB], t2[NB];
    const LSec sec = secs[blockIdx.x];
    const int c = min(p + NB - 1, sec.n - 2);
    if (c < p) return;
    LView L = lview(sec, eigbuf, wsd, wsi);
    finish_w(L, c, c - p, nullptr, t1, t2, red);
}

__global__ void k_tri_end(const LSec* __restrict__ secs, double* eigbuf, double* wsd, int* wsi) {
    const LSec sec = secs[blockIdx.x];
    if (threadIdx.x != 0) return;
    LView L = lview(sec, eigbuf, wsd, wsi);
    const int n = L.n;
    L.D[n - 1] = L.A[(size_t)(n - 1) + (size_t)(n - 1) * n];
    L.E[n - 1] = 0.0;
}

// ---------------------------------------------------------------------------------
// divide and conquer
// ---------------------------------------------------------------------------------
// leaves of the divide and conquer: one block per aligned range of DC_LOW rows of a
// sector runs every merge inside that range (all merges up to DC_LOW rows stay inside)
__global__ void __launch_bounds__(kLeafThreads) k_dc_low(const LSec* __restrict__ secs, int nsec, double* eigbuf,
                                                double* wsd, int* wsi, int* status) {
    extern __shared__ __align__(16) double sm[];
    int bid = blockIdx.x, sidx = 0;
    for (; sidx < nsec; ++sidx) {
        const int nc = (secs[sidx].n + DC_LOW - 1) / DC_LOW;
        if (bid < nc) break;
        bid -= nc;
    }
    if (sidx >= nsec) return;
    LView L = lview(secs[sidx], eigbuf, wsd, wsi);
    const int c0 = bid * DC_LOW;
    dc_leaf(c0, min(DC_LOW, L.n - c0), L.n, L.D, L.E, L.Z, sm, status);
}

struct Merge {
    int sec, a, mid, b;
    // block ranges of the parallel phases for the three thread mappings: one thread per
    // item (kMapItem), one warp per item (kMapWarp), one thread per few matrix entries
    // of the nn x nn merged block (kMapWide)
    int blk0[3], nblk[3];
};
constexpr int kMapItem = 0, kMapWarp = 1, kMapWide = 2;
constexpr int kWideItems = 8;   // matrix entries per thread in kMapWide

__device__ int find_merge(const Merge* ms, int nm, int map) {
    int lo = 0, hi = nm - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ms[mid].blk0[map] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(512) k_dc_prep(const LSec* __restrict__ secs, const Merge* __restrict__ ms,
                                                 double* eigbuf, double* wsd, int* wsi) {
    __shared__ double red[32];
    const Merge m = ms[blockIdx.x];
    LView L = lview(secs[m.sec], eigbuf, wsd, wsi);
    merge_prep(BlockG{}, m.a, m.mid, m.b, L.n, L.Z, L.D, L.E, L.S, red);
}

// phase 1 roots, 2 zhat, 3 rank-one vectors + values (one warp per root / entry / column),
// 4 final order + GEMM index lists (one thread per item), 5 deflated copies, 6 copy back
// (one thread per few entries)
__global__ void __launch_bounds__(TPB) k_dc_phase(const LSec* __restrict__ secs, const Merge* __restrict__ ms,
                                                  int nm, int phase, double* eigbuf, double* wsd, int* wsi,
                                                  int* status) {
    const int map = phase <= 3 ? kMapWarp : (phase == 4 ? kMapItem : kMapWide);
    const int mi = find_merge(ms, nm, map);
    const Merge m = ms[mi];
    LView L = lview(secs[m.sec], eigbuf, wsd, wsi);
    const int t = ((int)blockIdx.x - m.blk0[map]) * blockDim.x + threadIdx.x;
    const int T = m.nblk[map] * blockDim.x;
    const WarpLanes wl{(int)(threadIdx.x & 31)};
    switch (phase) {
        case 1: merge_roots(t >> 5, T >> 5, m.a, m.mid, L.E, L.S, status, wl); break;
        case 2: merge_zhat(t >> 5, T >> 5, m.a, m.mid, L.E, L.S, wl); break;
        case 3:
            merge_ucols(t >> 5, T >> 5, m.a, L.n, L.S, L.U, wl);
            merge_vals(t, T, m.a, m.b, L.S);
            break;
        case 4: {
            merge_rank(t, T, m.a, m.b, L.S);
            const int K = L.S.mk[m.a];
            // gathered columns of Z for the GEMM: a + perm[nd[q]] (ra reused after prep)
            for (int q = t; q < K; q += T) L.S.ra[m.a + q] = m.a + L.S.perm[m.a + L.S.nd[m.a + q]];
            break;
        }
        case 5: merge_deflated(t, T, m.a, m.b, L.n, L.Z, L.Qt, L.S); break;
        case 6: merge_copyback(t, T, m.a, m.b, L.n, L.Z, L.D, L.Qt, L.S); break;
        default: break;
    }
}

// scatter columns a + pos[j] of the nondeflated eigenvectors (rb reused)
__global__ void k_dc_poscols(const LSec* __restrict__ secs, const Merge* __restrict__ ms, int nm,
                             double* eigbuf, double* wsd, int* wsi) {
    const int mi = find_merge(ms, nm, kMapItem);
    const Merge m = ms[mi];
    LView L = lview(secs[m.sec], eigbuf, wsd, wsi);
    const int t = ((int)blockIdx.x - m.blk0[kMapItem]) * blockDim.x + threadIdx.x;
    const int T = m.nblk[kMapItem] * blockDim.x;
    const int K = L.S.mk[m.a];
    for (int j = t; j < K; j += T) L.S.rb[m.a + j] = m.a + L.S.pos[m.a + j];
}

// ---------------------------------------------------------------------------------
// back-transformation
// ---------------------------------------------------------------------------------
// explicit V panel (mr x b, ld mr) of reflectors jb .. jb+b-1 into U
__global__ void k_bt_vpanel(const LSec* __restrict__ secs, int q, double* eigbuf, double* wsd, int* wsi) {
    const LSec sec = secs[blockIdx.y];
    const int n = sec.n, nr = n - 1, jb = q * NBB;
    if (jb >= nr) return;
    LView L = lview(sec, eigbuf, wsd, wsi);
    const int b = min(NBB, nr - jb), r0 = jb + 1, mr = n - r0;
    const long long tot = (long long)mr * b;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot; e += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(e % mr), c = (int)(e / mr);
        const int k = jb + c, row = r0 + i;
        double v = 0.0;
        if (row == k + 1) v = 1.0;
        else if (row > k + 1) v = L.A[(size_t)row + (size_t)k * n];
        L.U[e] = v;
    }
}

// triangular factor T of the panel from the Gram matrix G (in Qt, b x b) and tau; T goes
// to Qt + NBB*NBB (b x b, ld NBB)
__global__ void k_bt_tfactor(const LSec* __restrict__ secs, int q, double* eigbuf, double* wsd, int* wsi) {
    extern __shared__ double tsm[];
    double* Ts = tsm;               // NBB x NBB
    double* G = tsm + NBB * NBB;    // the Gram matrix, staged
    const LSec sec = secs[blockIdx.x];
    const int n = sec.n, nr = n - 1, jb = q * NBB;
    if (jb >= nr) return;
    LView L = lview(sec, eigbuf, wsd, wsi);
    const int b = min(NBB, nr - jb);
    const int p = threadIdx.x;
    for (int e = threadIdx.x; e < NBB * NBB; e += blockDim.x) {
        Ts[e] = 0.0;
        G[e] = L.Qt[e];
    }
    __syncthreads();
    for (int c = 0; c < b; ++c) {
        const double tc = L.TAU[jb + c];
        double acc = 0.0;
        if (p < c)
            for (int qq = p; qq < c; ++qq) acc += Ts[p + qq * NBB] * (-tc * G[qq + c * NBB]);
        __syncthreads();
        if (p < c) Ts[p + c * NBB] = acc;
        if (p == 0) Ts[c + c * NBB] = tc;
        __syncthreads();
    }
    for (int e = threadIdx.x; e < NBB * NBB; e += blockDim.x) L.Qt[NBB * NBB + e] = Ts[e];
}

// ---- back-transformation in one pass per column block --------------------------------
// Panel q holds reflectors jb = 64 q .. jb + b - 1 (rows r0 = jb + 1 .. n - 1).  In R:
// the triangular factors T_q (NBB x NBB each) first, then the explicit panels
// V_q (mr x NBB, column-major, zero beyond b).
__device__ __forceinline__ long long bt_panel_off(int n, int q) {
    const long long npan = (n - 2) / NBB + 1;
    const long long before = (long long)q * (n - 1) - (long long)NBB * q * (q - 1) / 2;   // sum of mr
    return npan * NBB * NBB + (long long)NBB * before;
}

// explicit V_q, its Gram matrix and T_q (dlarft, forward, columnwise) for every panel of
// every sector at once: one block per (panel, sector)
__global__ void __launch_bounds__(256) k_bt_prep(const LSec* __restrict__ secs, double* eigbuf, double* wsd,
                                                 int* wsi) {
    extern __shared__ double bsm[];
    double* Vs = bsm;                  // chunk of the panel, Vs[c * 65 + r]
    double* G = Vs + NBB * 65;         // NBB x NBB, column-major
    double* Ts = G + NBB * NBB;        // NBB x NBB, column-major
    const LSec sec = secs[blockIdx.y];
    const int n = sec.n, nr = n - 1, q = blockIdx.x, jb = q * NBB;
    if (jb >= nr) return;
    LView L = lview(sec, eigbuf, wsd, wsi);
    const int b = min(NBB, nr - jb), r0 = jb + 1, mr = n - r0;
    double* Rp = L.R + bt_panel_off(n, q);
    double* Tq = L.R + (size_t)q * NBB * NBB;
    const int tid = threadIdx.x, ti = tid & 15, tj = tid >> 4;
    double g[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) g[a][c] = 0.0;
    for (int i0 = 0; i0 < mr; i0 += 64) {
        const int rows = min(64, mr - i0);
        for (int e = tid; e < 64 * NBB; e += 256) {
            const int r = e & 63, c = e >> 6;
            const int row = r0 + i0 + r, k = jb + c;
            double v = 0.0;
            if (r < rows && c < b) v = (row == k + 1) ? 1.0 : (row > k + 1 ? L.A[(size_t)row + (size_t)k * n] : 0.0);
            Vs[c * 65 + r] = v;
            if (r < rows) Rp[(size_t)(i0 + r) + (size_t)c * mr] = v;
        }
        __syncthreads();
        for (int r = 0; r < rows; ++r) {
            double x[4], y[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                x[a] = Vs[(ti * 4 + a) * 65 + r];
                y[a] = Vs[(tj * 4 + a) * 65 + r];
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int c = 0; c < 4; ++c) g[a][c] = fma(x[a], y[c], g[a][c]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) G[(ti * 4 + a) + (tj * 4 + c) * NBB] = g[a][c];
    for (int e = tid; e < NBB * NBB; e += 256) Ts[e] = 0.0;
    __syncthreads();
    for (int c = 0; c < b; ++c) {
        const double tc = L.TAU[jb + c];
        double acc = 0.0;
        if (tid < c)
            for (int qq = tid; qq < c; ++qq) acc += Ts[tid + qq * NBB] * (-tc * G[qq + c * NBB]);
        __syncthreads();
        if (tid < c) Ts[tid + c * NBB] = acc;
        if (tid == 0) Ts[c + c * NBB] = tc;
        __syncthreads();
    }
    for (int e = tid; e < NBB * NBB; e += 256) Tq[e] = Ts[e];
}

// 8-byte asynchronous global-to-shared copies (zero-filled when bytes is 0)
__device__ __forceinline__ void cp_async8(double* dst, const double* src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Z(:, c0 .. c0+CBK-1) <- H_0 ... H_{n-2} Z(:, ...) panel by panel (last panel first), the
// column block resident in shared memory; the result goes to the output
template <int CBK>
__global__ void __launch_bounds__(256, 1) k_bt_apply(const LSec* __restrict__ secs, int nsec, double* eigbuf,
                                                     double* wsd, int* wsi) {
    // The three small products of each panel, W = V^T Z, W2 = T W and Z -= V W2, on the
    // FP64 tensor pipe (mma.sync m8n8k4): the eight warps split the panel's 64 reflectors
    // (W, W2) or the chunk's 64 rows (the update) in slices of 8, and each warp covers the
    // CBK columns in tiles of 8.  What the products read streams through two shared
    // buffers of 64 x 65 doubles with asynchronous copies one step ahead: per panel the
    // chunks of 64 rows of V for W, then T, then the chunks again for the update, then the
    // next panel's first chunk.
    constexpr int NTJ = CBK / 8;
    // leading dimensions 4 mod 16 doubles (the Z block, the staged chunks and T): the
    // fragment loads and the row updates of a warp then fall on distinct bank pairs
    constexpr int VLD = NBB + 4;
    constexpr int BUF = NBB * VLD;
    extern __shared__ double asm_[];
    int bid = blockIdx.x, s = 0;
    for (; s < nsec; ++s) {
        const int nbk = (secs[s].n + CBK - 1) / CBK;
        if (bid < nbk) break;
        bid -= nbk;
    }
    if (s >= nsec) return;
    const LSec sec = secs[s];
    LView L = lview(sec, eigbuf, wsd, wsi);
    const int n = L.n, c0 = bid * CBK, nc = min(CBK, n - c0);
    const int ldz = n + ((4 - n) & 15);
    double* Zs = asm_;                      // Zs[j * ldz + row]
    double* Vb = Zs + (size_t)ldz * CBK;    // two buffers: Vs[c * VLD + r] (a chunk) or T (ld VLD)
    double* Ws = Vb + 2 * BUF;              // Ws[c * CBK + j]
    double* W2 = Ws + NBB * CBK;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, q4 = lane & 3;
    const int wr = 8 * warp;                // this warp's slice of reflectors / rows
    for (int j = 0; j < CBK; ++j)
        for (int row = tid; row < n; row += 256)
            Zs[(size_t)j * ldz + row] = j < nc ? L.Z[(size_t)row + (size_t)(c0 + j) * n] : 0.0;
    const int qmax = (n - 2) / NBB;
    // the load sequence: step t of panel q is a V chunk (t < C: for W; t > C: for the
    // update, chunk t - C - 1) or T (t == C), with C = ceil(mr / 64) chunks per pass
    auto chunks = [&](int q) { return (n - 1 - q * NBB + 63) / 64; };
    auto issue = [&](int q, int t, double* dst) {
        const int mr = n - 1 - q * NBB, C = chunks(q);
        if (t == C) {
            const double* Tq = L.R + (size_t)q * NBB * NBB;
            for (int e = tid; e < NBB * NBB; e += 256) cp_async8(dst + (e % NBB) + (e / NBB) * VLD, Tq + e, 8);
        } else {
            const int i0 = 64 * (t < C ? t : t - C - 1), rows = min(64, mr - i0);
            const double* Rp = L.R + bt_panel_off(n, q);
            for (int e = tid; e < 64 * NBB; e += 256) {
                const int r = e & 63, c = e >> 6;
                const int rr = r < rows ? r : rows - 1;   // in bounds; nothing is read when zero-filled
                cp_async8(dst + c * VLD + r, Rp + (size_t)(i0 + rr) + (size_t)c * mr, r < rows ? 8 : 0);
            }
        }
        cp_async_commit();
    };
    int buf = 0;
    issue(qmax, 0, Vb);
    for (int q = qmax; q >= 0; --q) {
        const int jb = q * NBB, r0 = jb + 1, mr = n - r0, C = chunks(q);
        double acc[NTJ][2];
#pragma unroll
        for (int t = 0; t < NTJ; ++t) acc[t][0] = acc[t][1] = 0.0;
        for (int t = 0; t <= 2 * C; ++t) {
            // the next step's load (the next panel's first chunk after the last step) into
            // the buffer the previous step has finished with
            double* nxt = Vb + (buf ^ 1) * BUF;
            if (t < 2 * C) issue(q, t + 1, nxt);
            else if (q > 0) issue(q - 1, 0, nxt);
            if (t < 2 * C || q > 0) cp_async_wait<1>();
            else cp_async_wait<0>();
            __syncthreads();
            const double* Vs = Vb + buf * BUF;
            if (t < C) {
                // W = V^T Z(r0:, :): W(i, j) for the warp's reflectors i
                const int i0 = 64 * t, rows = min(64, mr - i0);
                const double* zr = Zs + r0 + i0;
#pragma unroll 4
                for (int k0 = 0; k0 < 64; k0 += 4) {
                    const int kk = k0 + q4;
                    const double a = Vs[(wr + g) * VLD + kk];
#pragma unroll
                    for (int u = 0; u < NTJ; ++u) {
                        const double b = kk < rows ? zr[(size_t)(u * 8 + g) * ldz + kk] : 0.0;
                        nrg::cta_dmma(acc[u][0], acc[u][1], a, b);
                    }
                }
                if (t == C - 1) {
#pragma unroll
                    for (int u = 0; u < NTJ; ++u) {
                        Ws[(wr + g) * CBK + u * 8 + 2 * q4] = acc[u][0];
                        Ws[(wr + g) * CBK + u * 8 + 2 * q4 + 1] = acc[u][1];
                    }
                }
            } else if (t == C) {
                // W2 = T W (T upper triangular, zero below the diagonal)
#pragma unroll
                for (int u = 0; u < NTJ; ++u) acc[u][0] = acc[u][1] = 0.0;
#pragma unroll 4
                for (int k0 = 0; k0 < NBB; k0 += 4) {
                    const double a = Vs[(wr + g) + (k0 + q4) * VLD];
#pragma unroll
                    for (int u = 0; u < NTJ; ++u) nrg::cta_dmma(acc[u][0], acc[u][1], a, Ws[(k0 + q4) * CBK + u * 8 + g]);
                }
#pragma unroll
                for (int u = 0; u < NTJ; ++u) {
                    W2[(wr + g) * CBK + u * 8 + 2 * q4] = acc[u][0];
                    W2[(wr + g) * CBK + u * 8 + 2 * q4 + 1] = acc[u][1];
                }
            } else {
                // Z(r0:, :) -= V W2 on the chunk's 64 rows
                const int i0 = 64 * (t - C - 1), rows = min(64, mr - i0);
#pragma unroll
                for (int u = 0; u < NTJ; ++u) acc[u][0] = acc[u][1] = 0.0;
#pragma unroll 4
                for (int k0 = 0; k0 < NBB; k0 += 4) {
                    const double a = Vs[(k0 + q4) * VLD + wr + g];
#pragma unroll
                    for (int u = 0; u < NTJ; ++u) nrg::cta_dmma(acc[u][0], acc[u][1], a, W2[(k0 + q4) * CBK + u * 8 + g]);
                }
                const int row = wr + g;
                if (row < rows) {
                    double* zr = Zs + r0 + i0 + row;
#pragma unroll
                    for (int u = 0; u < NTJ; ++u) {
                        zr[(size_t)(u * 8 + 2 * q4) * ldz] -= acc[u][0];
                        zr[(size_t)(u * 8 + 2 * q4 + 1) * ldz] -= acc[u][1];
                    }
                }
            }
            __syncthreads();
            buf ^= 1;
        }
    }
    for (int j = 0; j < nc; ++j)
        for (int row = tid; row < n; row += 256)
            L.A[(size_t)row + (size_t)(c0 + j) * n] = Zs[(size_t)j * ldz + row];
}

__global__ void k_large_out(const LSec* __restrict__ secs, double* eigbuf, double* wsd, int* wsi) {
    const LSec sec = secs[blockIdx.y];
    LView L = lview(sec, eigbuf, wsd, wsi);
    const long long n = sec.n, sq = n * n;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < sq; e += (long long)gridDim.x * blockDim.x)
        L.A[e] = L.Z[e];
}

// the eigenvalues (ascending, the divide and conquer's order) to the output, one block
// per sector, as soon as the divide and conquer has finished
__global__ void k_large_evals(const LSec* __restrict__ secs, double* eigbuf, double* evals, double* wsd, int* wsi) {
    const LSec sec = secs[blockIdx.x];
    LView L = lview(sec, eigbuf, wsd, wsi);
    for (int i = threadIdx.x; i < sec.n; i += blockDim.x) evals[sec.e_off + i] = L.D[i];
}

}  // namespace

namespace nrg {

// ---------------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------------
// NRG_TRI_CLUSTER=0 takes the multi-kernel tridiagonalisation for every sector of order > 128
static bool tri_multi_kernel() {
    static const bool multi = [] {
        const char* e = getenv("NRG_TRI_CLUSTER");
        return e && e[0] == '0' && e[1] == 0;
    }();
    return multi;
}

int syev_large(nrg_context* ctx, const std::vector<SyevSector>& in, double* d_V, double* d_E, int slot_base,
               cudaEvent_t evals_ready) {
    const int ns = (int)in.size();
    if (ns == 0) return NRG_OK;
    cudaStream_t st = ctx->stream;
    std::vector<LSec> secs(ns);
    long long wd = 0, wi = 0;
    int maxn = 0;
    for (int s = 0; s < ns; ++s) {
        secs[s].a_off = in[s].a_off;
        secs[s].e_off = in[s].e_off;
        secs[s].n = in[s].n;
        secs[s].pad = 0;
        secs[s].w_off = wd;
        secs[s].i_off = wi;
        wd += lws_doubles(in[s].n);
        wi += lws_ints(in[s].n);
        maxn = std::max(maxn, in[s].n);
    }
    DevBuf& bsec = ctx->scratch.b[slot_base];
    DevBuf& bwd = ctx->scratch.b[slot_base + 1];
    DevBuf& bwi = ctx->scratch.b[slot_base + 2];
    DevBuf& bidx = ctx->scratch.b[slot_base + 3];
    DevBuf& bmrg = ctx->scratch.b[slot_base + 4];
    const int gslot = slot_base + 5;   // grouped GEMM problem lists (two slots)
    NRG_TRY(bsec.ensure(sizeof(LSec) * ns));
    NRG_TRY(bwd.ensure(sizeof(double) * (size_t)wd));
    NRG_TRY(bwi.ensure(sizeof(int) * (size_t)wi));
    // Sectors that fit on chip are reduced there (tri_resident).  Larger ones are streamed
    // from L2 until the trailing block fits (tri_stream); beyond its limit the multi-kernel
    // path is left: nbig sectors, the first ones (the list is sorted by decreasing order).
    const int res_max = tri_resident_max(), stream_max = tri_multi_kernel() ? 0 : tri_stream_max();
    int nbig = 0;
    while (nbig < ns && secs[nbig].n > stream_max) ++nbig;
    NRG_TRY(h2d_async(ctx, bsec.p, secs.data(), sizeof(LSec) * ns));
    const LSec* dsec = bsec.as<LSec>();
    double* wsd = bwd.as<double>();
    int* wsi = bwi.as<int>();
    // column index lists of the panel update [V W] and [W V] for every panel width jc
    {
        std::vector<int> idx(2 * NB * 2 * NB);
        for (int jc = 1; jc <= NB; ++jc)
            for (int q = 0; q < 2 * NB; ++q) {
                idx[(size_t)(jc - 1) * 4 * NB + q] = q < jc ? q : NB + (q - jc);            // [V W]
                idx[(size_t)(jc - 1) * 4 * NB + 2 * NB + q] = q < jc ? NB + q : q - jc;     // [W V]
            }
        NRG_TRY(bidx.ensure(sizeof(int) * idx.size()));
        NRG_TRY(h2d_async(ctx, bidx.p, idx.data(), sizeof(int) * idx.size()));
    }
    const int* didx = bidx.as<int>();
    const size_t symv_smem = sizeof(double) * (size_t)maxn;
    if (symv_smem > 48 * 1024)
        NRG_TRY(raise_smem_limit((const void*)k_tri_symv, symv_smem));

    // ---- 1. tridiagonalisation ----
    const bool clustered = nbig == 0;
    cudaEvent_t te[2] = {nullptr, nullptr};
    if (ctx->profiling) {
        NRG_CUDA_TRY(cudaEventCreate(&te[0]));
        NRG_CUDA_TRY(cudaEventCreate(&te[1]));
        NRG_CUDA_TRY(cudaEventRecord(te[0], st));
    }
    {
        std::vector<TriItem> items, streamed;
        for (int x = nbig; x < ns; ++x) {
            const int n = secs[x].n, c = std::max(0, n - res_max);   // columns before the trailing block
            double* vec = wsd + secs[x].w_off + 3LL * n * n + 2LL * NB * n + n;
            double* A = d_V + secs[x].a_off;
            if (c > 0) streamed.push_back(TriItem{A, vec, vec + n, vec + 2 * n, n, n, c});
            items.push_back(TriItem{A + c + (long long)c * n, vec + c, vec + n + c, vec + 2 * n + c, n - c, n, 0});
        }
        NRG_TRY(tri_stream(ctx, streamed, tri_wide_clusters() ? 16 : 8, ctx->scratch.b[slot_base == 24 ? 48 : 49]));
        NRG_TRY(tri_resident(ctx, items, ctx->scratch.b[slot_base == 24 ? 46 : 47]));
    }
    if (ctx->profiling) {
        NRG_CUDA_TRY(cudaEventRecord(te[1], st));
        if (clustered) {
            nrg_context::PendingTimer t{te[0], te[1], 0.0, 0.0};
            for (int x = 0; x < ns; ++x) {
                const double n = secs[x].n;
                t.flops += 4.0 / 3.0 * n * n * n;
                t.bytes += 8.0 * n * n * n / 3.0;
            }
            ctx->pending_tri.push_back(t);
        } else {
            cudaEventDestroy(te[0]);
            cudaEventDestroy(te[1]);
        }
    }
    for (int p = 0; !clustered && p < maxn - 1; p += NB) {
        for (int j = 0; j < NB; ++j) {
            const int k = p + j;
            if (k > maxn - 2) break;
            k_tri_col<<<nbig, TPB, 0, st>>>(dsec, k, d_V, wsd, wsi);
            int nblk = 0;
            for (int s = 0; s < nbig; ++s)
                if (k <= secs[s].n - 2) nblk += (secs[s].n - k - 1 + CB - 1) / CB;
            k_tri_symv<<<nblk, TPB, symv_smem, st>>>(dsec, nbig, k, d_V, wsd, wsi);
            ctx->launches += 2;
        }
        k_tri_finish<<<nbig, TPB, 0, st>>>(dsec, p, d_V, wsd, wsi);
        ctx->launches++;
        NRG_CUDA_TRY(cudaGetLastError());
        std::vector<GemmProblem> probs;
        for (int s = 0; s < nbig; ++s) {
            const int n = secs[s].n;
            const int c = std::min(p + NB - 1, n - 2);
            if (c < p) continue;
            const int jc = c - p + 1, r0 = p + jc;
            if (r0 >= n) continue;
            double* VW = wsd + secs[s].w_off + 3LL * n * n;
            GemmProblem P;
            std::memset(&P, 0, sizeof(P));
            P.M = n - r0; P.N = n - r0; P.K = 2 * jc;
            P.alpha = -1.0; P.beta = 1.0;
            P.A = VW + r0; P.a_si = 1; P.a_sk = n; P.a_ki = didx + (size_t)(jc - 1) * 4 * NB;
            P.B = VW + r0; P.b_sk = n; P.b_ki = didx + (size_t)(jc - 1) * 4 * NB + 2 * NB; P.b_sj = 1;
            P.C = d_V + secs[s].a_off + r0 + (long long)r0 * n; P.c_si = 1; P.c_sj = n;
            probs.push_back(P);
        }
        NRG_TRY(launch_ggemm(ctx, probs, gslot));
    }
    if (!clustered) {
        k_tri_end<<<nbig, 32, 0, st>>>(dsec, d_V, wsd, wsi);
        ctx->launches++;
    }

    // ---- 2. divide and conquer ----
    {
        NRG_TRY(raise_smem_limit((const void*)k_dc_low, kLeafSmem));
        int nchunk = 0;
        for (int x = 0; x < ns; ++x) nchunk += (secs[x].n + DC_LOW - 1) / DC_LOW;
        k_dc_low<<<nchunk, kLeafThreads, kLeafSmem, st>>>(dsec, ns, d_V, wsd, wsi, ctx->d_status.as<int>());
        ctx->launches++;
        NRG_CUDA_TRY(cudaGetLastError());
    }
    for (int s = DC_LOW; s < maxn; s *= 2) {
        std::vector<Merge> ms;
        int blk[3] = {0, 0, 0};
        for (int x = 0; x < ns; ++x) {
            const int n = secs[x].n;
            for (int a = 0; a + s < n; a += 2 * s) {
                Merge m;
                m.sec = x; m.a = a; m.mid = a + s; m.b = std::min(a + 2 * s, n);
                const long long nn = m.b - m.a;
                m.nblk[kMapItem] = (int)((nn + TPB - 1) / TPB);
                m.nblk[kMapWarp] = (int)((nn * 32 + TPB - 1) / TPB);
                m.nblk[kMapWide] = (int)((nn * nn + (long long)TPB * kWideItems - 1) / ((long long)TPB * kWideItems));
                for (int q = 0; q < 3; ++q) {
                    m.blk0[q] = blk[q];
                    blk[q] += m.nblk[q];
                }
                ms.push_back(m);
            }
        }
        if (ms.empty()) continue;
        const int nm = (int)ms.size();
        NRG_TRY(bmrg.ensure(sizeof(Merge) * nm));
        NRG_TRY(h2d_async(ctx, bmrg.p, ms.data(), sizeof(Merge) * nm));
        const Merge* dms = bmrg.as<Merge>();
        k_dc_prep<<<nm, 512, 0, st>>>(dsec, dms, d_V, wsd, wsi);
        for (int ph = 1; ph <= 4; ++ph)
            k_dc_phase<<<blk[ph <= 3 ? kMapWarp : kMapItem], TPB, 0, st>>>(dsec, dms, nm, ph, d_V, wsd, wsi,
                                                                           ctx->d_status.as<int>());
        k_dc_poscols<<<blk[kMapItem], TPB, 0, st>>>(dsec, dms, nm, d_V, wsd, wsi);
        ctx->launches += 6;
        NRG_CUDA_TRY(cudaGetLastError());
        // the number K of non-deflated roots of each merge stays on the device: the
        // GEMM is launched for K = nn and reads the true K (I[7n + a]) itself
        std::vector<GemmProblem> probs;
        for (int i = 0; i < nm; ++i) {
            const Merge& m = ms[i];
            const int n = secs[m.sec].n, nn = m.b - m.a;
            double* W = wsd + secs[m.sec].w_off;
            const long long sq = (long long)n * n;
            int* I = wsi + secs[m.sec].i_off;
            GemmProblem P;
            std::memset(&P, 0, sizeof(P));
            P.M = nn; P.N = nn; P.K = nn; P.alpha = 1.0; P.beta = 0.0;
            P.dyn_nk = I + 7LL * n + m.a;
            P.A = W + m.a; P.a_si = 1; P.a_sk = n; P.a_ki = I + 5LL * n + m.a;          // Z(:, a+perm[nd[q]])
            P.B = W + sq + m.a + (long long)m.a * n; P.b_sk = 1; P.b_sj = n;           // U block
            P.C = W + 2 * sq + m.a; P.c_si = 1; P.c_sj = n; P.c_ji = I + 6LL * n + m.a;  // Qt(:, a+pos[j])
            probs.push_back(P);
        }
        NRG_TRY(launch_ggemm(ctx, probs, gslot));
        k_dc_phase<<<blk[kMapWide], TPB, 0, st>>>(dsec, dms, nm, 5, d_V, wsd, wsi, ctx->d_status.as<int>());
        k_dc_phase<<<blk[kMapWide], TPB, 0, st>>>(dsec, dms, nm, 6, d_V, wsd, wsi, ctx->d_status.as<int>());
        ctx->launches += 2;
        NRG_CUDA_TRY(cudaGetLastError());
    }

    k_large_evals<<<ns, TPB, 0, st>>>(dsec, d_V, d_E, wsd, wsi);
    ctx->launches++;
    NRG_CUDA_TRY(cudaGetLastError());
    if (evals_ready) NRG_CUDA_TRY(cudaEventRecord(evals_ready, st));

    // ---- 3. back-transformation ----
    // one pass per column block with the block resident in shared memory, when it fits
    {
        int dev = 0, optin = 0;
        NRG_CUDA_TRY(cudaGetDevice(&dev));
        NRG_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        auto apply_smem = [&](int c) {   // Z block (ld up to maxn + 15), two staging buffers, W and W2
            return sizeof(double) * ((size_t)(maxn + 15) * c + 2 * NBB * (NBB + 4) + 2 * NBB * c);
        };
        const size_t prep_smem = sizeof(double) * (NBB * 65 + 2 * NBB * NBB);
        const int cbk = apply_smem(16) <= (size_t)optin ? 16 : (apply_smem(8) <= (size_t)optin ? 8 : 0);
        if (cbk > 0) {
            const int npan = (maxn - 2) / NBB + 1;
            NRG_TRY(raise_smem_limit((const void*)k_bt_prep, prep_smem));
            k_bt_prep<<<dim3(npan, ns), 256, prep_smem, st>>>(dsec, d_V, wsd, wsi);
            int nblk = 0;
            for (int x = 0; x < ns; ++x) nblk += (secs[x].n + cbk - 1) / cbk;
            const size_t sm = apply_smem(cbk);
            if (cbk == 16) {
                NRG_TRY(raise_smem_limit((const void*)k_bt_apply<16>, sm));
                k_bt_apply<16><<<nblk, 256, sm, st>>>(dsec, ns, d_V, wsd, wsi);
            } else {
                NRG_TRY(raise_smem_limit((const void*)k_bt_apply<8>, sm));
                k_bt_apply<8><<<nblk, 256, sm, st>>>(dsec, ns, d_V, wsd, wsi);
            }
            ctx->launches += 2;
            NRG_CUDA_TRY(cudaGetLastError());
            return NRG_OK;
        }
    }
    // otherwise panels of NBB reflectors on grouped GEMMs, last panel first
    const int qmax = (maxn - 2) / NBB;   // panels cover reflectors 0 .. n-2
    const size_t tf_smem = sizeof(double) * 2 * NBB * NBB;
    NRG_TRY(raise_smem_limit((const void*)k_bt_tfactor, tf_smem));
    for (int q = qmax; q >= 0; --q) {
        std::vector<int> act;
        for (int s = 0; s < ns; ++s)
            if (q * NBB < secs[s].n - 1) act.push_back(s);
        if (act.empty()) continue;
        k_bt_vpanel<<<dim3(16, ns), TPB, 0, st>>>(dsec, q, d_V, wsd, wsi);
        ctx->launches++;
        std::vector<GemmProblem> g1;
        for (int s : act) {
            const int n = secs[s].n, nr = n - 1, jb = q * NBB, b = std::min(NBB, nr - jb);
            const int r0 = jb + 1, mr = n - r0;
            double* W = wsd + secs[s].w_off;
            const long long sq = (long long)n * n;
            double* Vb = W + sq;            // U
            double* G = W + 2 * sq;         // Qt: G (NBB x NBB), T, then V^T Z
            GemmProblem P;
            std::memset(&P, 0, sizeof(P));
            P.M = b; P.N = b; P.K = mr; P.alpha = 1.0; P.beta = 0.0;
            P.A = Vb; P.a_si = mr; P.a_sk = 1;
            P.B = Vb; P.b_sk = 1; P.b_sj = mr;
            P.C = G; P.c_si = 1; P.c_sj = NBB;
            g1.push_back(P);
            GemmProblem Q;
            std::memset(&Q, 0, sizeof(Q));
            Q.M = b; Q.N = n; Q.K = mr; Q.alpha = 1.0; Q.beta = 0.0;
            Q.A = Vb; Q.a_si = mr; Q.a_sk = 1;
            Q.B = W + r0; Q.b_sk = 1; Q.b_sj = n;                       // Z(r0:, :)
            Q.C = G + 2 * NBB * NBB; Q.c_si = 1; Q.c_sj = b;            // Wt (b x n)
            g1.push_back(Q);
        }
        NRG_TRY(launch_ggemm(ctx, g1, gslot));
        k_bt_tfactor<<<ns, NBB, tf_smem, st>>>(dsec, q, d_V, wsd, wsi);
        ctx->launches++;
        std::vector<GemmProblem> g2, g3;
        for (int s : act) {
            const int n = secs[s].n, nr = n - 1, jb = q * NBB, b = std::min(NBB, nr - jb);
            const int r0 = jb + 1, mr = n - r0;
            double* W = wsd + secs[s].w_off;
            const long long sq = (long long)n * n;
            double* Vb = W + sq;
            double* Tm = W + 2 * sq + NBB * NBB;
            double* Wt = W + 2 * sq + 2 * NBB * NBB;
            double* VT = Vb + (long long)mr * NBB;     // (mr x b) after Vb in U
            GemmProblem P;
            std::memset(&P, 0, sizeof(P));
            P.M = mr; P.N = b; P.K = b; P.alpha = 1.0; P.beta = 0.0;
            P.A = Vb; P.a_si = 1; P.a_sk = mr;
            P.B = Tm; P.b_sk = 1; P.b_sj = NBB;
            P.C = VT; P.c_si = 1; P.c_sj = mr;
            g2.push_back(P);
            GemmProblem Q;
            std::memset(&Q, 0, sizeof(Q));
            Q.M = mr; Q.N = n; Q.K = b; Q.alpha = -1.0; Q.beta = 1.0;
            Q.A = VT; Q.a_si = 1; Q.a_sk = mr;
            Q.B = Wt; Q.b_sk = 1; Q.b_sj = b;
            Q.C = W + r0; Q.c_si = 1; Q.c_sj = n;
            g3.push_back(Q);
        }
        NRG_TRY(launch_ggemm(ctx, g2, gslot));
        NRG_TRY(launch_ggemm(ctx, g3, gslot));
    }
    k_large_out<<<dim3(32, ns), TPB, 0, st>>>(dsec, d_V, wsd, wsi);
    ctx->launches++;
    NRG_CUDA_TRY(cudaGetLastError());
    return NRG_OK;
}

}  // namespace nrg
