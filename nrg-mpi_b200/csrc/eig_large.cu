// FP64 eigensolver for the large symmetry sectors of one iteration (order > 128), spread
// over the whole GPU instead of one block per sector.  All large sectors advance together:
//   1. Householder tridiagonalisation (eig_tri.cu): orders up to 512 with the matrix on
//      chip, larger ones streamed from L2 until the trailing block fits there.  Orders
//      beyond the streaming kernel's shared memory (3,536) take the kernels below,
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
//
// That is the solver of the runs that keep their eigenvectors on the device.  For eigenvectors
// that go to a caller (EigSolver::Panel) steps 1 and 2 are those of eig_panel.cu.
#include "eig_dc.cuh"
#include "eig_sector.cuh"
#include "internal.hpp"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

namespace {

static_assert(DC_LOW == kDcLeafRows, "the leaves of the divide and conquer");

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
    dc_leaf<false>(c0, min(DC_LOW, L.n - c0), L.n, L.D, L.E, L.Z, sm, status);
}

// Merges beyond DC_LOW rows, all merges of one level at once, in five launches: poles and
// deflation (a block per merge), secular roots, Gu-Eisenstat z with the order of the results,
// rank-one eigenvectors with the deflated columns (a warp per item), and the eigenvector
// update as one grouped GEMM.  The children's blocks are read from one of two buffers and
// the merged block is written to the other, so nothing is copied back; the rows of the
// rank-one eigenvectors are the children's columns, so that the update is two products of
// half the inner length per merge and no operand is gathered.  Before: ten launches per
// level, the deflation scan on one thread (230..315 us at 1225 rows) and the update over
// the children's zero blocks.
struct Merge {
    int sec, a, mid, b;   // mid == b: a block without a partner at this level
    int blk0, nblk;       // blocks of the warp-per-item launches
};

__device__ int find_merge(const Merge* ms, int nm) {
    int lo = 0, hi = nm - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ms[mid].blk0 <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    return lo;
}

constexpr int kPrepThreads = 512;
constexpr size_t kPrepSmem = 200 * 1024;   // four doubles per row in shared memory up to 6,400 rows

// exclusive scans over the block of an int per thread: the sum, or the maximum with -1 first
__device__ int block_scan(int v, bool maximum, int* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = maximum ? max(x, y) : x + y;
    }
    __syncthreads();
    if (lane == 31) red[warp] = x;
    __syncthreads();
    int base = maximum ? -1 : 0;
    for (int w = 0; w < warp; ++w) base = maximum ? max(base, red[w]) : base + red[w];
    const int y = __shfl_up_sync(0xffffffffu, x, 1);
    const int before = lane == 0 ? (maximum ? -1 : 0) : y;
    return maximum ? max(base, before) : base + before;
}

// z, merge order, poles and deflation of one merge.  Deflated entries: negligible z, found in
// parallel, and the first of a pair of close poles, rotated into the second.  Whether a pair
// is close depends on its predecessor only through a rotation, so one thread visits just
// the entries that are close to the unrotated one before them, and what follows each as
// long as rotations go on.  df: the rotated entries in the order of the rotations, then the
// negligible ones; chain starts in `nd`'s tail are not needed: rotation r continues the
// one before when it shares its entry.
__global__ void __launch_bounds__(kPrepThreads) k_dc_prep(const LSec* __restrict__ secs, const Merge* __restrict__ ms,
                                                          long long z_off, double* eigbuf, double* wsd, int* wsi,
                                                          int* status) {
    extern __shared__ __align__(16) double psm[];
    __shared__ double red[32];
    __shared__ int ired[32];
    __shared__ int nflag, nrots;
    const Merge m = ms[blockIdx.x];
    if (m.mid == m.b) return;
    LView L = lview(secs[m.sec], eigbuf, wsd, wsi);
    const int n = L.n, a = m.a, nn = m.b - m.a, n1 = m.mid - m.a, t = threadIdx.x;
    const double* Z = L.Z + z_off * n * n;
    const bool in_smem = 4 * sizeof(double) * (size_t)nn <= kPrepSmem;
    double* Dm = in_smem ? psm : L.D + a;
    double* z = in_smem ? psm + nn : L.S.z + a;
    double* ds = in_smem ? psm + 2 * nn : L.S.ds + a;
    double* zs = in_smem ? psm + 3 * nn : L.S.zs + a;
    int *perm = L.S.perm + a, *nd = L.S.nd + a, *df = L.S.df + a, *flag = L.S.org + a, *kind = L.S.pos + a;
    const double beta = L.E[m.mid - 1], rho = 2.0 * fabs(beta), sg = beta >= 0.0 ? 1.0 : -1.0;
    for (int i = t; i < nn; i += kPrepThreads) {
        if (in_smem) Dm[i] = L.D[a + i];
        z[i] = (i < n1 ? Z[(size_t)(m.mid - 1) + (size_t)(a + i) * n] : sg * Z[(size_t)m.mid + (size_t)(a + i) * n]) *
               0.70710678118654752440;
    }
    if (t == 0) nflag = nrots = 0;
    __syncthreads();
    // stable merge order of the two ascending halves (first half wins ties)
    double dm = 0.0, zm = 0.0;
    for (int i = t; i < nn; i += kPrepThreads) {
        const bool one = i < n1;
        const double v = Dm[i];
        int lo = 0, hi = one ? nn - n1 : n1;
        const double* o = one ? Dm + n1 : Dm;
        while (lo < hi) {
            const int x = (lo + hi) >> 1;
            if (one ? o[x] < v : o[x] <= v) lo = x + 1; else hi = x;
        }
        const int r = (one ? i : i - n1) + lo;
        perm[r] = i;
        ds[r] = v;
        zs[r] = z[i];
        dm = fmax(dm, fabs(v));
        zm = fmax(zm, fabs(z[i]));
    }
    const double tol = 8.0 * kEps * block_max(fmax(dm, rho * zm), red);
    __syncthreads();
    // a run of entries per thread: kind 0 kept, 1 negligible, 2 rotated out
    const int run = (nn + kPrepThreads - 1) / kPrepThreads, r0 = min(t * run, nn), r1 = min(r0 + run, nn);
    int last = -1;
    for (int r = r0; r < r1; ++r) {
        const bool live = rho * fabs(zs[r]) > tol;
        kind[r] = live ? 0 : 1;
        if (live) last = r;
    }
    int prev = block_scan(last, true, ired);
    auto close_to = [&](double zj, double dj, double zl, double dl) {
        // |(d_j - d_l) c s| <= tol with c = z_j / r, s = -z_l / r, r^2 = z_j^2 + z_l^2
        return fabs(dj - dl) * fabs(zj * zl) <= tol * fma(zj, zj, zl * zl);
    };
    int mine = 0;
    {
        int l = prev;
        for (int r = r0; r < r1; ++r)
            if (kind[r] == 0) {
                if (l >= 0 && close_to(zs[r], ds[r], zs[l], ds[l])) ++mine;
                l = r;
            }
    }
    int at = block_scan(mine, false, ired);
    {
        int l = prev;
        for (int r = r0; r < r1; ++r)
            if (kind[r] == 0) {
                if (l >= 0 && close_to(zs[r], ds[r], zs[l], ds[l])) flag[at++] = r;
                l = r;
            }
    }
    if (t == kPrepThreads - 1) nflag = at;
    __syncthreads();
    if (t == 0 && nflag > 0) {
        int nrot = 0, done = -1;
        for (int f = 0; f < nflag; ++f) {
            int j = flag[f];
            if (j <= done) continue;
            int l = j - 1;
            while (kind[l] != 0) --l;           // the entry it is close to is still there: it was not visited
            double zl = zs[l], dl = ds[l];
            for (;;) {
                const double zj = zs[j], dj = ds[j];
                done = j;
                if (!close_to(zj, dj, zl, dl)) break;
                const double r = hypot(zj, zl), c_ = zj / r, s_ = -zl / r;
                L.S.ra[a + nrot] = perm[l];
                L.S.rb[a + nrot] = perm[j];
                L.S.rc[a + nrot] = c_;
                L.S.rs[a + nrot] = s_;
                df[nrot++] = l;
                const double tn = dl * c_ * c_ + dj * s_ * s_, dn = dl * s_ * s_ + dj * c_ * c_;
                zs[j] = zl = r;
                zs[l] = 0.0;
                ds[j] = dl = dn;
                ds[l] = tn;
                kind[l] = 2;
                l = j;
                do ++j; while (j < nn && kind[j] != 0);
                if (j >= nn) break;
            }
        }
        nrots = nrot;
    }
    __syncthreads();
    int nk = 0, nz = 0;
    for (int r = r0; r < r1; ++r) {
        nk += kind[r] == 0;
        nz += kind[r] == 1;
    }
    int qk = block_scan(nk, false, ired), qz = block_scan(nz, false, ired) + nrots;
    for (int r = r0; r < r1; ++r) {
        if (kind[r] == 0) {
            nd[qk] = perm[r];
            L.S.dd[a + qk] = ds[r];
            L.S.zz[a + qk] = zs[r];
            ++qk;
        } else if (kind[r] == 1) {
            df[qz++] = r;
        }
    }
    if (t == kPrepThreads - 1) {
        L.S.mk[a] = qk;             // roots
        L.S.mr[a] = nrots;
        L.S.mf[a] = qk + nrots;     // columns of the eigenvector update
    }
    __syncthreads();
    // deflated values follow the roots; df becomes the child column of the entry
    const int K = L.S.mk[a];
    for (int q = t; q < nn - K; q += kPrepThreads) {
        const int r = df[q];
        L.S.vals[a + K + q] = finite_value(ds[r], status);
        df[q] = perm[r];
    }
}

// the 32 lanes of a warp on one item
struct WarpItem {
    static constexpr int kPer = 32;
    __device__ double sum(double v) const {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
    __device__ double prod(double v) const {
        for (int o = 16; o > 0; o >>= 1) v *= __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
};

// phase 1 secular roots, 2 z and places of the results, 3 rank-one eigenvectors and deflated
// columns: one warp per item
template <int PHASE>
__global__ void __launch_bounds__(TPB) k_dc_items(const LSec* __restrict__ secs, const Merge* __restrict__ ms, int nm,
                                                  long long z_in, long long z_out, double* eigbuf, double* wsd, int* wsi,
                                                  int* status) {
    const Merge m = ms[find_merge(ms, nm)];
    LView L = lview(secs[m.sec], eigbuf, wsd, wsi);
    const int n = L.n, a = m.a, nn = m.b - m.a, lane = threadIdx.x & 31;
    const int e = ((int)blockIdx.x - m.blk0) * (TPB / 32) + (threadIdx.x >> 5);
    if (e >= nn) return;
    const WarpItem g;
    const bool alone = m.mid == m.b;
    const int K = alone ? 0 : L.S.mk[a];
    const double rho = 2.0 * fabs(L.E[m.mid - 1]);
    const double *dd = L.S.dd + a, *zz = L.S.zz + a, *tau = L.S.tau + a;
    const int* org = L.S.org + a;
    if constexpr (PHASE == 1) {
        if (e < K) {
            leaf_root(g, lane, K, dd, zz, rho, e, L.S.org + a + e, L.S.tau + a + e, status);
            __syncwarp();
            if (lane == 0) L.S.vals[a + e] = finite_value(dd[org[e]] + tau[e], status);
        }
    } else if constexpr (PHASE == 2) {
        if (alone) return;
        if (e < K) {
            const double di = dd[e];
            double p = 1.0;
            for (int j = lane; j < K - 1; j += 32) p *= quotient((di - dd[org[j]]) - tau[j], di - dd[j < e ? j : j + 1]);
            p = g.prod(p) * quotient(-((di - dd[org[K - 1]]) - tau[K - 1]), rho);
            if (lane == 0) L.S.zh[a + e] = copysign(root_of(fmax(p, 0.0)), zz[e]);
        }
        // place in ascending order, ties in list order (roots, then deflated values)
        const double* vals = L.S.vals + a;
        const double v = vals[e];
        int r = 0;
        for (int f = lane; f < nn; f += 32) {
            const double w = vals[f];
            r += (w < v) || (w == v && f < e);
        }
        r = __reduce_add_sync(0xffffffffu, r);
        if (lane == 0) {
            L.S.pos[a + e] = r;
            L.D[a + r] = v;
        }
    } else {
        const double* Z = L.Z + z_in * n * n;
        double* Q = L.Z + z_out * n * n;
        const int N = alone ? 0 : L.S.mf[a];
        const int *nd = L.S.nd + a, *df = L.S.df + a;
        if (e >= N) {
            // a column that only moves: a deflated one, or any of a block without a partner
            const int src = alone ? e : df[e - K], dst = alone ? e : L.S.pos[a + e];
            const bool one = a + src < m.mid;
            for (int i = a + lane; i < m.b; i += 32)
                Q[(size_t)i + (size_t)(a + dst) * n] = (i < m.mid) == one ? Z[(size_t)i + (size_t)(a + src) * n] : 0.0;
            return;
        }
        double* uc = L.U + (size_t)a + (size_t)(a + e) * n;
        for (int q = lane; q < nn - K; q += 32) uc[df[q]] = 0.0;
        if (e < K) {
            double q = 0.0;
            const double dj = dd[org[e]], tj = tau[e];
            for (int i = lane; i < K; i += 32) {
                const double u = quotient(L.S.zh[a + i], (dd[i] - dj) - tj);
                uc[nd[i]] = u;
                q = fma(u, u, q);
            }
            q = rsqrt(g.sum(q));
            for (int i = lane; i < K; i += 32) uc[nd[i]] *= q;
        } else {
            for (int i = lane; i < K; i += 32) uc[nd[i]] = 0.0;
            __syncwarp();
            if (lane == 0) uc[df[e - K]] = 1.0;
        }
        const int nrot = L.S.mr[a];
        if (nrot == 0) return;
        __syncwarp();
        // rotated columns: the rows take the rotations, last one first; rotations that share
        // no entry run side by side (a chain shares each entry with the next rotation)
        const int *ra = L.S.ra + a, *rb = L.S.rb + a;
        for (int r0 = lane; r0 < nrot; r0 += 32) {
            if (r0 + 1 < nrot && ra[r0 + 1] == rb[r0]) continue;   // not the last of its chain
            for (int r = r0; r >= 0; --r) {
                const double c_ = L.S.rc[a + r], s_ = L.S.rs[a + r], x = uc[ra[r]], y = uc[rb[r]];
                uc[ra[r]] = fma(c_, x, -s_ * y);
                uc[rb[r]] = fma(s_, x, c_ * y);
                if (r == 0 || ra[r] != rb[r - 1]) break;
            }
        }
    }
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
// every sector at once: one block per (panel, sector).  The Gram matrix is on the FP64 MMA, each
// warp five 8 x 8 tiles of a row (tiles row + 0 .. 4 modulo 8 hold every pair of columns), the
// next 64 rows loaded meanwhile.  T is put together from two halves, whose recursions run in
// one warp each with a row of T per lane, T12 = -T1 G12 T2: the recursion over all 64 columns in
// shared memory, two barriers a column, was most of the kernel's 0.34 ms for 4 sectors of order
// 1150 (0.06 ms now).
constexpr int kPrepLd = NBB + 4;   // 4 mod 16 doubles: conflict-free MMA operands
constexpr size_t kBtPrepSmem = sizeof(double) * 3 * NBB * kPrepLd;
__global__ void __launch_bounds__(256) k_bt_prep(const LSec* __restrict__ secs, double* eigbuf, double* wsd,
                                                 int* wsi) {
    constexpr int LD = kPrepLd, H = NBB / 2, LDX = H + 4;
    extern __shared__ double bsm[];
    double* Vs = bsm;                  // 64 rows of the panel, Vs[c * LD + r]
    double* G = Vs + NBB * LD;         // G[i * LD + j], tiles of the upper triangle
    double* Ts = G + NBB * LD;         // T(p, c) at Ts[c * LD + p]
    const LSec sec = secs[blockIdx.y];
    const int n = sec.n, nr = n - 1, q = blockIdx.x, jb = q * NBB;
    if (jb >= nr) return;
    LView L = lview(sec, eigbuf, wsd, wsi);
    const int b = min(NBB, nr - jb), r0 = jb + 1, mr = n - r0;
    double* Rp = L.R + bt_panel_off(n, q);
    double* Tq = L.R + (size_t)q * NBB * NBB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q4 = lane & 3;
    const int r = tid & 63, cb = tid >> 6;   // the thread's row and columns cb + 4 u of a chunk
    double v[NBB / 4];
    auto load = [&](int i0) {
        const int row = r0 + i0 + r;
#pragma unroll
        for (int u = 0; u < NBB / 4; ++u) {
            const int c = cb + 4 * u, k = jb + c;
            v[u] = 0.0;
            if (i0 + r < mr && c < b) v[u] = row == k + 1 ? 1.0 : (row > k + 1 ? L.A[(size_t)row + (size_t)k * n] : 0.0);
        }
    };
    double acc[5][2];
#pragma unroll
    for (int d = 0; d < 5; ++d) acc[d][0] = acc[d][1] = 0.0;
    load(0);
    for (int i0 = 0; i0 < mr; i0 += 64) {
#pragma unroll
        for (int u = 0; u < NBB / 4; ++u) {
            const int c = cb + 4 * u;
            Vs[c * LD + r] = v[u];
            if (i0 + r < mr) Rp[(size_t)(i0 + r) + (size_t)c * mr] = v[u];
        }
        __syncthreads();
        if (i0 + 64 < mr) load(i0 + 64);
#pragma unroll 4
        for (int k0 = 0; k0 < 64; k0 += 4) {
            const double a = Vs[(8 * warp + g) * LD + k0 + q4];
#pragma unroll
            for (int d = 0; d < 5; ++d)
                nrg::cta_dmma(acc[d][0], acc[d][1], a, Vs[(8 * ((warp + d) & 7) + g) * LD + k0 + q4]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int d = 0; d < 5; ++d)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = 8 * warp + g, j = 8 * ((warp + d) & 7) + 2 * q4 + h;
            if (i <= j) G[i * LD + j] = acc[d][h];
            if (i > j && d < 4) G[j * LD + i] = acc[d][h];   // d = 4 has its mirror in another warp
        }
    for (int e = tid; e < H * H; e += 256) Ts[(e / H) * LD + H + e % H] = 0.0;   // below the diagonal blocks
    __syncthreads();
    if (warp < 2) {
        const double* Gd = G + warp * (H * LD + H);
        double* Td = Ts + warp * (H * LD + H);
        double row[H];
#pragma unroll
        for (int c = 0; c < H; ++c) {
            const int k = H * warp + c;
            const double tc = k < b ? L.TAU[jb + k] : 0.0;
            double s[2] = {0.0, 0.0};
#pragma unroll
            for (int p = 0; p < c; ++p) s[p & 1] = fma(row[p], Gd[p * LD + c], s[p & 1]);
            row[c] = lane == c ? tc : (lane < c ? -tc * (s[0] + s[1]) : 0.0);
            Td[c * LD + lane] = row[c];
        }
    }
    __syncthreads();
    // X = G12 T2, T12 = -T1 X: each warp two of the 4 x 4 tiles
    double* X = Vs;                    // X(p, c) at X[c * LDX + p]
    const int ti = warp >> 1;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int tj = 2 * (warp & 1) + u;
        double d0 = 0.0, d1 = 0.0;
#pragma unroll
        for (int k0 = 0; k0 < H; k0 += 4)
            nrg::cta_dmma(d0, d1, G[(8 * ti + g) * LD + H + k0 + q4], Ts[(H + 8 * tj + g) * LD + H + k0 + q4]);
        X[(8 * tj + 2 * q4) * LDX + 8 * ti + g] = d0;
        X[(8 * tj + 2 * q4 + 1) * LDX + 8 * ti + g] = d1;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int tj = 2 * (warp & 1) + u;
        double d0 = 0.0, d1 = 0.0;
#pragma unroll
        for (int k0 = 0; k0 < H; k0 += 4)
            nrg::cta_dmma(d0, d1, Ts[(k0 + q4) * LD + 8 * ti + g], X[(8 * tj + g) * LDX + k0 + q4]);
        Ts[(H + 8 * tj + 2 * q4) * LD + 8 * ti + g] = -d0;
        Ts[(H + 8 * tj + 2 * q4 + 1) * LD + 8 * ti + g] = -d1;
    }
    __syncthreads();
    for (int e = tid; e < NBB * NBB; e += 256) Tq[e] = Ts[(e / NBB) * LD + e % NBB];
}

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
            Zs[(size_t)j * ldz + row] = j < nc ? L.ZV[(size_t)row + (size_t)(c0 + j) * n] : 0.0;
    const int qmax = (n - 2) / NBB;
    // the load sequence: step t of panel q is a V chunk (t < C: for W; t > C: for the
    // update, chunk t - C - 1) or T (t == C), with C = ceil(mr / 64) chunks per pass
    auto chunks = [&](int q) { return (n - 1 - q * NBB + 63) / 64; };
    auto issue = [&](int q, int t, double* dst) {
        const int mr = n - 1 - q * NBB, C = chunks(q);
        if (t == C) {
            const double* Tq = L.R + (size_t)q * NBB * NBB;
            for (int e = tid; e < NBB * NBB; e += 256) nrg::cp_async8(dst + (e % NBB) + (e / NBB) * VLD, Tq + e, 8);
        } else {
            const int i0 = 64 * (t < C ? t : t - C - 1), rows = min(64, mr - i0);
            const double* Rp = L.R + bt_panel_off(n, q);
            for (int e = tid; e < 64 * NBB; e += 256) {
                const int r = e & 63, c = e >> 6;
                const int rr = r < rows ? r : rows - 1;   // in bounds; nothing is read when zero-filled
                nrg::cp_async8(dst + c * VLD + r, Rp + (size_t)(i0 + rr) + (size_t)c * mr, r < rows ? 8 : 0);
            }
        }
        nrg::cp_async_commit();
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
            if (t < 2 * C || q > 0) nrg::cp_async_wait<1>();
            else nrg::cp_async_wait<0>();
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
// NRG_TRI_CLUSTER=0 (a test aid) takes the multi-kernel tridiagonalisation for every sector of order > 128
static bool tri_multi_kernel() {
    static const bool multi = [] {
        const char* e = getenv("NRG_TRI_CLUSTER");
        return e && e[0] == '0' && e[1] == 0;
    }();
    return multi;
}

int syev_large(nrg_context* ctx, const std::vector<SyevSector>& in, double* d_V, double* d_E, EigSolver solver,
               const EigSlots& slots, cudaEvent_t evals_ready) {
    const bool panel = solver == EigSolver::Panel;
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
        int levels = 0;
        for (int w = DC_LOW; w < in[s].n; w *= 2) ++levels;
        secs[s].z_sel = !panel && levels % 2 ? 2 : 0;
        secs[s].w_off = wd;
        secs[s].i_off = wi;
        wd += lws_doubles(in[s].n);
        wi += lws_ints(in[s].n);
        maxn = std::max(maxn, in[s].n);
    }
    DevBuf& bsec = ctx->scratch.b[slots.sectors];
    DevBuf& bwd = ctx->scratch.b[slots.doubles];
    DevBuf& bwi = ctx->scratch.b[slots.ints];
    DevBuf& bidx = ctx->scratch.b[slots.columns];
    DevBuf& bmrg = ctx->scratch.b[slots.merges];
    const int gslot = slots.products;   // grouped GEMM problem lists
    NRG_TRY(bsec.ensure(sizeof(LSec) * ns));
    NRG_TRY(bwd.ensure(sizeof(double) * (size_t)wd));
    NRG_TRY(bwi.ensure(sizeof(int) * (size_t)wi));
    // Sectors that fit on chip are reduced there (tri_resident).  Larger ones are streamed
    // from L2 until the trailing block fits (tri_stream); beyond its limit the multi-kernel
    // path is left: nbig sectors, the first ones (the list is sorted by decreasing order).
    const int res_max = tri_resident_max(), stream_max = tri_multi_kernel() ? 0 : tri_stream_max();
    int nbig = 0;
    while (!panel && nbig < ns && secs[nbig].n > stream_max) ++nbig;
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
    cudaEvent_t te[2] = {nullptr, nullptr};
    if (ctx->profiling) {
        NRG_CUDA_TRY(cudaEventCreate(&te[0]));
        NRG_CUDA_TRY(cudaEventCreate(&te[1]));
        NRG_CUDA_TRY(cudaEventRecord(te[0], st));
    }
    if (panel) {
        bool done = false;   // otherwise every sector takes the multi-kernel path
        NRG_TRY(panel_tridiagonal(ctx, dsec, ns, maxn, d_V, wsd, wsi, &done));
        nbig = done ? 0 : ns;
    } else {
        std::vector<TriItem> items, streamed;
        for (int x = nbig; x < ns; ++x) {
            const int n = secs[x].n, c = std::max(0, n - res_max);   // columns before the trailing block
            double* vec = wsd + secs[x].w_off + 3LL * n * n + 2LL * NB * n + n;
            double* A = d_V + secs[x].a_off;
            // the streamed matrix moves to the space of Z and U, which the divide and conquer fills later
            double* P = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(wsd + secs[x].w_off) + 127) & ~uintptr_t(127));
            if (c > 0) streamed.push_back(TriItem{A, vec, vec + n, vec + 2 * n, n, n, c, P});
            items.push_back(TriItem{A + c + (long long)c * n, vec + c, vec + n + c, vec + 2 * n + c, n - c, n, 0});
        }
        NRG_TRY(tri_stream(ctx, streamed, ctx->scratch.b[slots.streamed]));
        NRG_TRY(tri_resident(ctx, items, ctx->scratch.b[slots.on_chip]));
    }
    const bool clustered = nbig == 0;
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
    if (panel) {
        NRG_TRY(panel_merges(ctx, secs, dsec, maxn, d_V, wsd, wsi, bmrg, gslot));
    } else {
        NRG_TRY(raise_smem_limit((const void*)k_dc_low, kLeafSmem));
        int nchunk = 0;
        for (int x = 0; x < ns; ++x) nchunk += (secs[x].n + DC_LOW - 1) / DC_LOW;
        k_dc_low<<<nchunk, kLeafThreads, kLeafSmem, st>>>(dsec, ns, d_V, wsd, wsi, ctx->d_status.as<int>());
        ctx->launches++;
        NRG_CUDA_TRY(cudaGetLastError());
    }
    // the eigenvectors alternate between Z and Qt from level to level (in units of n x n)
    long long z_in = 0, z_out = 2;
    NRG_TRY(raise_smem_limit((const void*)k_dc_prep, kPrepSmem));
    for (int s = DC_LOW; !panel && s < maxn; s *= 2) {
        std::vector<Merge> ms;
        std::vector<GemmProblem> probs;
        int blk = 0, widest = 0;
        for (int x = 0; x < ns; ++x) {
            const int n = secs[x].n;
            for (int a = 0; a < n && s < n; a += 2 * s) {
                Merge m;
                m.sec = x; m.a = a; m.b = std::min(a + 2 * s, n); m.mid = std::min(a + s, m.b);
                const int nn = m.b - m.a;
                m.blk0 = blk;
                m.nblk = (nn + TPB / 32 - 1) / (TPB / 32);
                blk += m.nblk;
                ms.push_back(m);
                if (m.mid == m.b) continue;
                widest = std::max(widest, nn);
                // rows of each child: its block times its rows of the rank-one eigenvectors; the
                // number of columns stays on the device (I[9n + a], k_dc_prep)
                double* W = wsd + secs[x].w_off;
                const long long sq = (long long)n * n;
                int* I = wsi + secs[x].i_off;
                for (int c = 0; c < 2; ++c) {
                    const int r0 = c == 0 ? m.a : m.mid, r1 = c == 0 ? m.mid : m.b;
                    GemmProblem P;
                    std::memset(&P, 0, sizeof(P));
                    P.M = r1 - r0; P.N = nn; P.K = r1 - r0; P.alpha = 1.0; P.beta = 0.0;
                    P.dyn_n = I + 9LL * n + m.a;
                    P.A = W + z_in * sq + r0 + (long long)r0 * n; P.a_si = 1; P.a_sk = n;
                    P.B = W + sq + r0 + (long long)m.a * n; P.b_sk = 1; P.b_sj = n;
                    P.C = W + z_out * sq + r0 + (long long)m.a * n; P.c_si = 1; P.c_sj = n; P.c_ji = I + 4LL * n + m.a;
                    probs.push_back(P);
                }
            }
        }
        const int nm = (int)ms.size();
        NRG_TRY(bmrg.ensure(sizeof(Merge) * nm));
        NRG_TRY(h2d_async(ctx, bmrg.p, ms.data(), sizeof(Merge) * nm));
        const Merge* dms = bmrg.as<Merge>();
        int* d_status = ctx->d_status.as<int>();
        const size_t psm = std::min(kPrepSmem, 4 * sizeof(double) * (size_t)widest);
        k_dc_prep<<<nm, kPrepThreads, psm, st>>>(dsec, dms, z_in, d_V, wsd, wsi, d_status);
        k_dc_items<1><<<blk, TPB, 0, st>>>(dsec, dms, nm, z_in, z_out, d_V, wsd, wsi, d_status);
        k_dc_items<2><<<blk, TPB, 0, st>>>(dsec, dms, nm, z_in, z_out, d_V, wsd, wsi, d_status);
        k_dc_items<3><<<blk, TPB, 0, st>>>(dsec, dms, nm, z_in, z_out, d_V, wsd, wsi, d_status);
        ctx->launches += 4;
        NRG_CUDA_TRY(cudaGetLastError());
        NRG_TRY(launch_ggemm(ctx, probs, gslot));
        std::swap(z_in, z_out);
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
        const int cbk = apply_smem(16) <= (size_t)optin ? 16 : (apply_smem(8) <= (size_t)optin ? 8 : 0);
        if (cbk > 0) {
            const int npan = (maxn - 2) / NBB + 1;
            NRG_TRY(raise_smem_limit((const void*)k_bt_prep, kBtPrepSmem));
            k_bt_prep<<<dim3(npan, ns), 256, kBtPrepSmem, st>>>(dsec, d_V, wsd, wsi);
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
    // otherwise panels of NBB reflectors on grouped GEMMs, last panel first, on Z (Qt is their
    // workspace)
    for (int x = 0; x < ns; ++x)
        if (secs[x].z_sel != 0) {
            double* W = wsd + secs[x].w_off;
            const size_t sq = (size_t)secs[x].n * secs[x].n;
            NRG_CUDA_TRY(cudaMemcpyAsync(W, W + 2 * sq, sizeof(double) * sq, cudaMemcpyDeviceToDevice, st));
        }
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
