// Divide and conquer on tridiagonal blocks of up to 128 rows, one thread block each: the
// whole of a sector of order <= 128, or one aligned range of 128 rows of a larger one
// (whose merges beyond 128 rows follow in eig_large.cu).
//
// Cuppen tearing down to 1 x 1, then merges of 2, 4, ... 128 rows.  What bounds the leaves
// is latency (a few thousand dependent FP64 operations), so everything a merge touches is
// in shared memory and no thread waits for work that another could do:
//   * merges of up to 32 rows run one lane per row, 32 / (rows) of them side by side in a
//     warp; a warp carries its 32 rows through the first five levels without a block
//     barrier.  The merges of 64 and 128 rows take 256 and 512 threads, four lanes per
//     item.
//   * the eigenvector blocks are kept packed (the blocks of one level side by side, n x s),
//     which leaves room for the rank-one eigenvectors of the last merge beside them:
//     68 KB + 135 KB; only the result of the last merge goes to global memory;
//   * deflation by ballots: the serial scan of close poles runs only where a pair of
//     neighbouring poles is close;
//   * the rank-one eigenvectors are stored with their rows ordered by child, so that the
//     update Z U is two products of half the inner length (FP64 MMA), scaled to unit
//     norm as it is stored;
//   * the secular iteration starts from the evaluation that decides the nearer pole.
// Order 128: the leaves of a range take 0.19 ms for 0.49 (nine block or warp merges through
// global memory, one lane in four or a single thread at work), a whole block of order 128
// with its tridiagonalisation and back-transformation 0.45 ms for 0.97.
#pragma once
#include "eig_common.cuh"

namespace {

constexpr int kLeafThreads = 512, kDcLeafRows = 128;
constexpr int kLd = kDcLeafRows + 4;   // = 4 mod 16: conflict-free MMA fragments

// offsets of the level's blocks in the packed region: children (n x s), rank-one
// eigenvectors (rows x 2s) and the merged blocks, which are the next level's children.
// Two areas: A holds 64 columns, B 128.  Every offset is a multiple of the leading dimension,
// so the warps of the small levels stay in their own 32 rows (columns, for the rank-one
// eigenvectors) whatever level each has reached.
constexpr int kAreaA = 0, kAreaB = kLd * 64, kAreaEnd = kAreaB + kLd * 128;
__device__ __forceinline__ int child_off(int s) {
    return s == 64 || s == 16 || s == 4 ? kAreaA : (s == 32 ? kAreaB + kLd * 64 : kAreaB);
}
__device__ __forceinline__ int rank1_off(int s) {
    return s == 64 || s == 32 ? kAreaB : (s == 1 ? kAreaA : child_off(s) + kLd * s);
}

struct Leaf {
    double *D, *E, *z, *ds, *zs, *dd, *zz, *tau, *zh, *vals, *rc, *rs, *rn;
    int *perm, *nd, *df, *org, *pos, *ra, *rb, *row, *col, *cnt;   // cnt: K, K1, rotations, deflated per merge
};
constexpr int kLeafDoubles = 13 * kDcLeafRows + 10 * kDcLeafRows / 2;
__device__ __forceinline__ Leaf leaf_at(double* p) {
    Leaf L;
    double** d[] = {&L.D, &L.E, &L.z, &L.ds, &L.zs, &L.dd, &L.zz, &L.tau, &L.zh, &L.vals, &L.rc, &L.rs, &L.rn};
#pragma unroll
    for (int i = 0; i < 13; ++i) *d[i] = p + i * kDcLeafRows;
    int* q = reinterpret_cast<int*>(p + 13 * kDcLeafRows);
    int** e[] = {&L.perm, &L.nd, &L.df, &L.org, &L.pos, &L.ra, &L.rb, &L.row, &L.col, &L.cnt};
#pragma unroll
    for (int i = 0; i < 10; ++i) *e[i] = q + i * kDcLeafRows;
    return L;
}

// a / b with one correction of the reciprocal's quotient (Markstein): the accuracy of a
// division at a quarter of its latency, for operands away from the ends of the range
__device__ __forceinline__ double quotient(double a, double b) {
    const double r = 1.0 / b, q = a * r;
    return fma(fma(-q, b, a), r, q);
}

// The threads of one merge.  Lanes: W lanes of a warp (one merge of up to W rows, one lane
// per item); Threads: T threads of the block, four lanes per item.
template <int W>
struct Lanes {
    static constexpr int kPer = 1;
    int t;
    __device__ int rank() const { return t; }
    __device__ int size() const { return W; }
    __device__ void sync() const { __syncwarp(); }
    __device__ unsigned mask() const { return W == 32 ? 0xffffffffu : ((1u << W) - 1u) << ((threadIdx.x & 31) & ~(W - 1)); }
    __device__ double max(double v, double*) const {
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
    __device__ double sum(double v) const { return v; }
    __device__ double prod(double v) const { return v; }
    // bit i of word i / 32: the flag of item i
    __device__ void flags(bool f, unsigned (&w)[4], unsigned*) const {
        w[0] = (__ballot_sync(0xffffffffu, f) & mask()) >> ((threadIdx.x & 31) & ~(W - 1));
        w[1] = w[2] = w[3] = 0u;
    }
};
template <int T>
struct Threads {
    static constexpr int kPer = 4;
    int t;
    __device__ int rank() const { return t; }
    __device__ int size() const { return T; }
    __device__ void sync() const { __syncthreads(); }
    __device__ double max(double v, double* red) const {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if ((t & 31) == 0) red[t >> 5] = v;
        __syncthreads();
        double m = red[0];
        for (int i = 1; i < T / 32; ++i) m = fmax(m, red[i]);
        __syncthreads();
        return m;
    }
    // over the four lanes of an item; the shuffles name only those lanes, so the items of one
    // warp may leave their loops at different times
    __device__ unsigned four() const { return 0xfu << (t & 28); }
    __device__ double sum(double v) const {
        v += __shfl_xor_sync(four(), v, 1);
        return v + __shfl_xor_sync(four(), v, 2);
    }
    __device__ double prod(double v) const {
        v *= __shfl_xor_sync(four(), v, 1);
        return v * __shfl_xor_sync(four(), v, 2);
    }
    __device__ void flags(bool f, unsigned (&w)[4], unsigned* words) const {
        const unsigned m = __ballot_sync(0xffffffffu, f);
        if ((t & 31) == 0 && t < 128) words[t >> 5] = m;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = words[i];
        __syncthreads();
    }
};

__device__ __forceinline__ int below(const unsigned (&w)[4], int i) {   // flags set before item i
    int c = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (32 * q + 32 <= i) c += __popc(w[q]);
        else if (32 * q < i) c += __popc(w[q] & ((1u << (i - 32 * q)) - 1u));
    }
    return c;
}
__device__ __forceinline__ int last_below(const unsigned (&w)[4], int i) {   // the last of them, or -1
#pragma unroll
    for (int q = 3; q >= 0; --q) {
        const int n = i - 32 * q;
        if (n <= 0) continue;
        const unsigned m = n >= 32 ? w[q] : (w[q] & ((1u << n) - 1u));
        if (m) return 32 * q + 31 - __clz(m);
    }
    return -1;
}

// Root j of 1 + rho sum_i zz_i^2 / (dd_i - lambda) = 0 (rho > 0, dd ascending, zz != 0),
// returned as lambda = dd[org] + tau with org the pole nearer to the root, so that every
// difference dd_i - lambda = (dd_i - dd[org]) - tau keeps full relative accuracy.
// Iteration: the two-pole rational model of the secular function (the poles bounding the
// root carry the near terms, Bunch-Nielsen-Sorensen), solved as a quadratic, kept inside a
// bisection bracket; at most 100 steps.  The evaluation at the middle of the interval
// serves the choice of the origin and the first step.
template <class G>
__device__ void leaf_root(const G& g, int first, int K, const double* dd, const double* zz, double rho, int j, int* org,
                          double* tau, int* status) {
    const bool last = j == K - 1;
    int o = j;
    double t, lo = 0.0, hi, base = dd[j], gap = 0.0;
    if (last) {
        double zsq = 0.0;
        for (int i = first; i < K; i += G::kPer) zsq = fma(zz[i], zz[i], zsq);
        hi = rho * g.sum(zsq);
    } else {
        gap = dd[j + 1] - dd[j];
        hi = gap;
    }
    t = 0.5 * hi;
    for (int it = 0; it < 100; ++it) {
        double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;
        for (int i = first; i < K; i += G::kPer) {
            const double r = 1.0 / ((dd[i] - base) - t);
            const double q = zz[i] * zz[i] * r, dq = q * r;
            if (i <= j) { psi += q; dpsi += dq; } else { phi += q; dphi += dq; }
        }
        psi = rho * g.sum(psi); dpsi = rho * g.sum(dpsi); phi = rho * g.sum(phi); dphi = rho * g.sum(dphi);
        const double f = 1.0 + psi + phi;
        if (it == 0) {
            // the half of the interval that holds the root; its pole is the origin
            if (last) {
                if (f >= 0.0) hi = t; else lo = t;
            } else if (f >= 0.0) {
                hi = t;
            } else {
                o = j + 1;
                base = dd[o];
                t = lo = -0.5 * gap;
                hi = 0.0;
            }
        } else if (f > 0.0) hi = t;
        else if (f < 0.0) lo = t;
        if (f == 0.0 || fabs(f) <= 8.0 * K * kEps * (1.0 + fabs(psi) + fabs(phi))) break;
        const double D1 = (dd[j] - base) - t;
        bool ok = false;
        double eta = 0.0;
        if (!last) {
            // psi ~ a + b / (dd_j - x), phi ~ c + e2 / (dd_{j+1} - x), matched at t
            const double D2 = (dd[j + 1] - base) - t;
            const double b = dpsi * D1 * D1, a = psi - dpsi * D1;
            const double e2 = dphi * D2 * D2, c = phi - dphi * D2;
            const double C = 1.0 + a + c;
            const double B2 = -(C * (D1 + D2) + b + e2), C2 = D1 * D2 * f;
            const double disc = B2 * B2 - 4.0 * C * C2;
            if (disc >= 0.0 && C != 0.0) {
                const double sq = disc > 0.0 ? disc * rsqrt(disc) : 0.0;
                const double qq = -0.5 * (B2 + (B2 >= 0.0 ? sq : -sq));
                const double r1 = qq * (1.0 / C), r2 = (qq != 0.0) ? C2 * (1.0 / qq) : r1;
                double best = 1e300;
                if (t + r1 > lo && t + r1 < hi) { best = r1; ok = true; }
                if (t + r2 > lo && t + r2 < hi && fabs(r2) < fabs(best)) { best = r2; ok = true; }
                eta = best;
            }
        } else {
            const double b = dpsi * D1 * D1, C = 1.0 + psi - dpsi * D1;
            if (C > 0.0) {
                eta = ((dd[j] - base) + b * (1.0 / C)) - t;
                ok = (t + eta > lo && t + eta < hi);
            }
        }
        const double tn = ok ? t + eta : 0.5 * (lo + hi);
        if (tn == t) break;
        t = tn;
        if (hi - lo <= 2.0 * kEps * fmax(fabs(lo), fabs(hi))) break;
    }
    if (first == 0) {
        if (!(t == t)) atomicOr(status, NRG_DEV_SECULAR);
        *org = o;
        *tau = t;
    }
}

// C (rows x N, column pos[j] of dst, row offset in dst already applied) = Zc(:, col[k])
// U(k, j) rn[j], one warp per column tile of 8; dst element (i, j) at dst[i + j * ldd]
__device__ __forceinline__ void child_product(int warp, int nwarps, int M, int N, int Kc, const double* Zc, const int* col,
                                              const double* U, const double* rn, const int* pos, double* dst, long long ldd) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q4 = lane & 3;
    for (int j0 = 8 * warp; j0 < N; j0 += 8 * nwarps) {
        double acc[8][2];
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = 0.0;
        for (int k0 = 0; k0 < Kc; k0 += 4) {
            const int k = k0 + q4;
            const bool kin = k < Kc;
            const double b = kin && j0 + g < N ? U[k * kLd + j0 + g] : 0.0;
            const double* zc = Zc + (kin ? col[k] : 0) * kLd + g;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                if (8 * r >= M) break;
                const double x = kin && 8 * r + g < M ? zc[8 * r] : 0.0;
                nrg::cta_dmma(acc[r][0], acc[r][1], x, b);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = j0 + 2 * q4 + h;
            if (j >= N) continue;
            const double sc = rn[j];
            double* out = dst + (long long)pos[j] * ldd;
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (8 * r + g < M) out[8 * r + g] = acc[r][h] * sc;
        }
    }
}

// sqrt from rsqrt with one correction; p >= 0
__device__ __forceinline__ double root_of(double p) {
    if (p < 1e-280) return sqrt(p);
    const double r = rsqrt(p), q = p * r;
    return fma(0.5 * r, fma(-q, q, p), q);
}

// what the product of a merge needs: rows of the rank-one eigenvectors (child 1's first),
// columns of the result
struct MergeSize {
    int K, K1, rows, cols, ndf;
    bool dense;
};
__device__ __forceinline__ MergeSize merge_size(const int* cnt, int nn, int n1) {
    MergeSize m;
    m.K = cnt[0];
    const int c = cnt[1];
    m.dense = (c & 0xffff) != 0;            // rotations: every child column takes part
    m.K1 = m.dense ? n1 : c >> 16;
    m.rows = m.dense ? nn : m.K;
    m.cols = m.dense ? nn : m.K;
    m.ndf = nn - m.K;
    return m;
}

// One merge of the children [a, a + s) and [a + s, b) up to the rank-one eigenvectors U (row
// k, column a + j; rows ordered by child, not normalised: 1 / norm in rn) and the places of
// the results.  b == a: no merge, but the barriers are taken.
//
// MARK: *unsure is set when the merge decides close to its tolerance, or between values so
// close (relative to the largest) that their eigenvectors hang on the last bits.  Over 3.1
// million columns of random blocks (orders 64, 100 and 128) this solver and the panel solver
// decided otherwise on 10; a margin of 2% missed 2 of them, 6% one, a quarter none.  It marks
// 10% of the blocks of order 128, 16% of 100 and 2% of 64.
constexpr double kUnsure = 1.25, kUnsureGap = 1e-6;
template <bool MARK, class G>
__device__ void leaf_merge(const G& g, int a, int s, int b, const Leaf& L, const double* Zc, double* U, double* red,
                           unsigned* words, int* status, int* unsure) {
    const int t = g.rank(), T = g.size();
    const int nn = b - a, n1 = s;                       // nn > s, or 0
    const double beta = L.E[a + s - 1];
    const double rho = 2.0 * fabs(beta), sg = beta >= 0.0 ? 1.0 : -1.0;
    const double r2 = 0.70710678118654752440;
    double* Da = L.D + a;
    double *z = L.z + a, *ds = L.ds + a, *zs = L.zs + a;
    int *perm = L.perm + a, *nd = L.nd + a, *df = L.df + a, *cnt = L.cnt + a;
    // z = [last row of Z1, sign(beta) * first row of Z2] / sqrt(2); stable merge order of the
    // two ascending halves (first half wins ties)
    for (int i = t; i < nn; i += T) {
        const bool one = i < n1;
        const double zi = s == 1 ? 1.0 : (one ? Zc[(a + s - 1) + kLd * i] : Zc[(a + s) + kLd * (i - n1)]);
        z[i] = (one ? zi : sg * zi) * r2;
        const double v = Da[i];
        int lo = 0, hi = one ? nn - n1 : n1;
        const double* o = one ? Da + n1 : Da;
        while (lo < hi) {
            const int m = (lo + hi) >> 1;
            if (one ? o[m] < v : o[m] <= v) lo = m + 1; else hi = m;
        }
        perm[(one ? i : i - n1) + lo] = i;
    }
    g.sync();
    double dm = 0.0, zm = 0.0;
    for (int r = t; r < nn; r += T) {
        const int p = perm[r];
        const double dv = Da[p], zv = z[p];
        ds[r] = dv;
        zs[r] = zv;
        dm = fmax(dm, fabs(dv));
        zm = fmax(zm, fabs(zv));
    }
    const double tol = 8.0 * kEps * g.max(fmax(dm, rho * zm), red);
    g.sync();
    // ---- deflation: negligible z, then close neighbours among the others ----
    const bool in = t < nn;
    if (MARK && in) {
        const double zr = rho * fabs(zs[t]);
        if ((zr > tol / kUnsure && zr < tol * kUnsure) ||
            (t > 0 && ds[t] - ds[t - 1] <= kUnsureGap / (8.0 * kEps) * tol))
            *unsure = 1;
    }
    unsigned live[4], close[4];
    g.flags(in && rho * fabs(zs[in ? t : 0]) > tol, live, words);
    const bool kept = in && ((live[(t >> 5) & 3] >> (t & 31)) & 1u);
    bool near = false;
    if (kept) {
        const int l = last_below(live, t);
        if (l >= 0) {
            // |(d_j - d_l) c s| <= tol with c = z_j / r, s = -z_l / r, r^2 = z_j^2 + z_l^2
            const double zj = zs[t], zl = zs[l];
            near = fabs(ds[t] - ds[l]) * fabs(zj * zl) <= tol * fma(zj, zj, zl * zl);
        }
    }
    g.flags(near, close, words);
    if ((close[0] | close[1] | close[2] | close[3]) == 0u) {
        if (in) {
            const int q = below(live, t);
            if (kept) nd[q] = t; else df[t - q] = t;
        }
        if (t == 0 && nn > 0) {
            cnt[0] = below(live, nn);
            cnt[1] = 0;
        }
    } else if (t == 0) {
        int K = 0, ndf = 0, nrot = 0, jlam = -1;
        double zl = 0.0, dl = 0.0;   // z and d of the pending entry jlam
        for (int j = 0; j < nn; ++j) {
            const double zj = zs[j], dj = ds[j];
            if (rho * fabs(zj) <= tol) { df[ndf++] = j; continue; }
            if (jlam < 0) { jlam = j; zl = zj; dl = dj; continue; }
            if (fabs(dj - dl) * fabs(zj * zl) <= tol * fma(zj, zj, zl * zl)) {
                const double r = hypot(zj, zl);
                const double c_ = zj / r, s_ = -zl / r;
                zs[j] = r;
                zs[jlam] = 0.0;
                L.ra[a + nrot] = perm[jlam];
                L.rb[a + nrot] = perm[j];
                L.rc[a + nrot] = c_;
                L.rs[a + nrot] = s_;
                ++nrot;
                const double tn = dl * c_ * c_ + dj * s_ * s_;
                const double dn = dl * s_ * s_ + dj * c_ * c_;
                ds[j] = dn;
                ds[jlam] = tn;
                df[ndf++] = jlam;
                zl = r;
                dl = dn;
            } else {
                nd[K++] = jlam;
                zl = zj;
                dl = dj;
            }
            jlam = j;
        }
        if (jlam >= 0) nd[K++] = jlam;
        cnt[0] = K;
        cnt[1] = nrot;
    }
    g.sync();
    const int K = nn > 0 ? cnt[0] : 0, nrot = nn > 0 ? cnt[1] : 0;
    // poles, and the row of the rank-one eigenvectors that each takes: child by child
    const int src = t < K ? perm[nd[t]] : 0;
    unsigned c1[4];
    g.flags(t < K && src < n1, c1, words);
    const int K1 = __popc(c1[0]) + __popc(c1[1]) + __popc(c1[2]) + __popc(c1[3]);
    double *dd = L.dd + a, *zz = L.zz + a, *rn = L.rn + a;
    int *row = L.row + a, *col = L.col + a;
    if (t < K) {
        dd[t] = ds[nd[t]];
        zz[t] = zs[nd[t]];
        const int q = below(c1, t), k = nrot ? src : (src < n1 ? q : K1 + (t - q));
        row[t] = k;
        if (!nrot) col[k] = src < n1 ? src : src - n1;
    }
    if (nrot)
        for (int k = t; k < nn; k += T) col[k] = k < n1 ? k : k - n1;
    g.sync();
    if (t == 0 && nn > 0 && !nrot) cnt[1] = K1 << 16;
    // ---- secular roots, Gu-Eisenstat z, rank-one eigenvectors ----
    constexpr int P = G::kPer;
    const int item = t / P, first = t % P, step = T / P;
    int* org = L.org + a;
    double *tau = L.tau + a, *zh = L.zh + a;
    for (int j = item; j < K; j += step) leaf_root(g, first, K, dd, zz, rho, j, org + j, tau + j, status);
    if (nrot)
        for (int e = t; e < nn * nn; e += T) U[(e / nn) * kLd + a + e % nn] = 0.0;
    g.sync();
    for (int i = item; i < K; i += step) {
        double p = 1.0;
        const double di = dd[i];
        for (int j = first; j < K - 1; j += P)
            p *= quotient((di - dd[org[j]]) - tau[j], di - dd[j < i ? j : j + 1]);
        p = g.prod(p) * quotient(-((di - dd[org[K - 1]]) - tau[K - 1]), rho);
        if (first == 0) zh[i] = copysign(root_of(fmax(p, 0.0)), zz[i]);
    }
    g.sync();
    for (int j = item; j < K; j += step) {
        double q = 0.0;
        const double dj = dd[org[j]], tj = tau[j];
        for (int i = first; i < K; i += P) {
            const double u = quotient(zh[i], (dd[i] - dj) - tj);
            U[row[i] * kLd + a + j] = u;
            q = fma(u, u, q);
        }
        q = g.sum(q);
        if (first == 0) rn[j] = rsqrt(q);
    }
    // the merged values, nondeflated roots first, and their places in ascending order (ties
    // keep list order)
    double* vals = L.vals + a;
    for (int e = t; e < nn; e += T) vals[e] = finite_value(e < K ? dd[org[e]] + tau[e] : ds[df[e - K]], status);
    if (nrot)
        for (int q = t; q < nn - K; q += T) {
            U[perm[df[q]] * kLd + a + K + q] = 1.0;
            rn[K + q] = 1.0;
        }
    g.sync();
    // rotated columns: the rows of U take the rotations instead, last one first
    for (int j = t; nrot && j < nn; j += T)
        for (int r = nrot - 1; r >= 0; --r) {
            double *ux = U + L.ra[a + r] * kLd + a + j, *uy = U + L.rb[a + r] * kLd + a + j;
            const double c_ = L.rc[a + r], s_ = L.rs[a + r], x = *ux, y = *uy;
            *ux = fma(c_, x, -s_ * y);
            *uy = fma(s_, x, c_ * y);
        }
    int* pos = L.pos + a;
    for (int e = t; e < nn; e += T) {
        int r = e;
        if (K < nn) {
            const double v = vals[e];
            r = 0;
            for (int f = 0; f < nn; ++f) r += (vals[f] < v) || (vals[f] == v && f < e);
        }
        pos[e] = r;
        Da[r] = vals[e];
    }
    g.sync();
}

// deflated columns (no rotations) to their places, rows of the other child zero; and the
// whole block where there was nothing to merge.  dst: row i, column j at dst[i + j * ldd]
__device__ __forceinline__ void leaf_deflated(int t, int T, int a, int s, int nn, const MergeSize& m, const Leaf& L,
                                              const double* Zc, double* dst, long long ldd) {
    if (m.dense) return;
    for (int e = t; e < nn * m.ndf; e += T) {
        const int i = e % nn, q = e / nn, src = L.perm[a + L.df[a + q]];
        const bool mine = (i < s) == (src < s);
        const double v = !mine ? 0.0 : (s == 1 ? 1.0 : Zc[a + i + kLd * (src < s ? src : src - s)]);
        dst[i + (long long)L.pos[a + m.K + q] * ldd] = v;
    }
}

// the levels of one warp's 32 rows: merges of W = 2 s rows, 32 / W at a time
template <int W, bool MARK>
__device__ void warp_level(int r0, int nl, const Leaf& L, double* area, double* Zg, long long ldz, int* status, int* unsure) {
    constexpr int s = W / 2;
    const int lane = threadIdx.x & 31;
    const Lanes<W> g{lane & (W - 1)};
    const double* Zc = area + child_off(s);
    double* U = area + rank1_off(s);
    const bool last = W >= nl;                          // the range's last merge: to global memory
    double* out = last ? Zg : area + child_off(2 * s);
    const long long ldd = last ? ldz : kLd;
    const int a = r0 + (lane & ~(W - 1));
    const int b = a + s < nl ? min(a + W, nl) : a;      // b == a: no second child
    leaf_merge<MARK>(g, a, s, b, L, Zc, U, nullptr, nullptr, status, unsure);
    if constexpr (W <= 8) {
        // one lane per column of the result
        const int nn = b - a, j = g.t;
        if (nn > 0) {
            const MergeSize m = merge_size(L.cnt + a, nn, s);
            if (j < m.cols) {
                const double sc = L.rn[a + j];
                double* o = out + a + (last ? (long long)(L.pos[a + j]) * ldd : (long long)L.pos[a + j] * ldd);
                for (int i = 0; i < nn; ++i) {
                    const int k0 = i < s ? 0 : m.K1, k1 = i < s ? m.K1 : m.rows;
                    double q = 0.0;
                    for (int k = k0; k < k1; ++k)
                        q = fma(s == 1 ? 1.0 : Zc[a + i + kLd * L.col[a + k]], U[k * kLd + a + j], q);
                    o[i] = q * sc;
                }
            }
            leaf_deflated(g.t, W, a, s, nn, m, L, Zc, out + a, ldd);
        }
    } else {
#pragma unroll 1
        for (int q = 0; q < 32 / W; ++q) {
            const int aq = r0 + q * W, nn = aq + s < nl ? min(W, nl - aq) : 0;
            if (nn == 0) continue;
            const MergeSize m = merge_size(L.cnt + aq, nn, s);
            child_product(0, 1, s, m.cols, m.K1, Zc + aq, L.col + aq, U + aq, L.rn + aq, L.pos + aq, out + aq, ldd);
            child_product(0, 1, nn - s, m.cols, m.rows - m.K1, Zc + aq + s, L.col + aq + m.K1, U + aq + m.K1 * kLd,
                          L.rn + aq, L.pos + aq, out + aq + s, ldd);
            leaf_deflated(lane, 32, aq, s, nn, m, L, Zc, out + aq, ldd);
        }
    }
    if (b == a && a < nl) {
        // nothing to merge: the block as it is
        const int nn = min(s, nl - a);
        for (int j = 0; j < nn; ++j)
            for (int i = g.t; i < nn; i += W) out[a + i + (long long)j * ldd] = s == 1 ? 1.0 : Zc[a + i + kLd * j];
    }
    __syncwarp();
}

// the merges of 2 s = 512 / (512 / T) rows: T threads each
template <int T, bool MARK>
__device__ void block_level(int s, int nl, const Leaf& L, double* area, double* Zg, long long ldz, double* red,
                            unsigned* words, int* status, int* unsure) {
    const int tid = threadIdx.x, mi = tid / T, a = 2 * s * mi;
    const Threads<T> g{tid % T};
    const double* Zc = area + child_off(s);
    double* U = area + rank1_off(s);
    const bool last = 2 * s >= nl;
    double* out = last ? Zg : area + child_off(2 * s);
    const long long ldd = last ? ldz : kLd;
    const int b = a + s < nl ? min(a + 2 * s, nl) : a;
    leaf_merge<MARK>(g, a, s, b, L, Zc, U, red + 16 * mi, words + 4 * mi, status, unsure);
    const int nn = b - a;
    if (nn > 0) {
        const MergeSize m = merge_size(L.cnt + a, nn, s);
        const int w = g.t >> 5;
        if (w & 1)
            child_product(w >> 1, T / 64, nn - s, m.cols, m.rows - m.K1, Zc + a + s, L.col + a + m.K1, U + a + m.K1 * kLd,
                          L.rn + a, L.pos + a, out + a + s, ldd);
        else
            child_product(w >> 1, T / 64, s, m.cols, m.K1, Zc + a, L.col + a, U + a, L.rn + a, L.pos + a, out + a, ldd);
        leaf_deflated(g.t, T, a, s, nn, m, L, Zc, out + a, ldd);
    } else if (a < nl) {
        const int w = nl - a;
        for (int e = g.t; e < w * w; e += T) out[a + e % w + (long long)(e / w) * ldd] = Zc[a + e % w + kLd * (e / w)];
    }
    __syncthreads();
}

constexpr size_t kLeafSmem = sizeof(double) * (kAreaEnd + kLeafDoubles + 32 + 4);

// Rows c0 .. c0 + nl - 1 (nl <= 128) of a tridiagonal matrix of order n: eigenvalues
// (ascending) to D, eigenvectors to the diagonal block of Z (leading dimension n); the rest
// of those columns of Z is set to zero.  512 threads; sm: kLeafSmem bytes.
template <bool MARK>
__device__ void dc_leaf(int c0, int nl, int n, double* D, const double* E, double* Z, double* sm, int* status,
                        int* unsure = nullptr) {
    const int tid = threadIdx.x, warp = tid >> 5;
    double* area = sm;
    const Leaf L = leaf_at(sm + kAreaEnd);
    double* red = sm + kAreaEnd + kLeafDoubles;
    unsigned* words = reinterpret_cast<unsigned*>(red + 32);
    double* Zg = Z + c0 + (long long)c0 * n;
    // rank-one tearing at every boundary: each leaf is 1 x 1
    if (tid < kDcLeafRows) {
        double dv = 0.0, ev = 0.0;
        if (tid < nl) {
            const int i = c0 + tid;
            dv = D[i];
            ev = finite_value(E[i], status);
            if (i > 0) dv -= fabs(E[i - 1]);
            if (i < n - 1) dv -= fabs(ev);
            dv = finite_value(dv, status);
        }
        L.D[tid] = dv;
        L.E[tid] = ev;
    }
    // the rows outside the range
    for (int c = warp; nl < n && c < nl; c += kLeafThreads / 32) {
        double* zc = Z + (long long)(c0 + c) * n;
        for (int i = tid & 31; i < n; i += 32)
            if (i < c0 || i >= c0 + nl) zc[i] = 0.0;
    }
    __syncthreads();
    if (32 * warp < nl && warp < 4) {
        const int r0 = 32 * warp;
        if (nl == 1) {
            if (tid == 0) Zg[0] = 1.0;
        } else {
            warp_level<2, MARK>(r0, nl, L, area, Zg, n, status, unsure);
            if (nl > 2) warp_level<4, MARK>(r0, nl, L, area, Zg, n, status, unsure);
            if (nl > 4) warp_level<8, MARK>(r0, nl, L, area, Zg, n, status, unsure);
            if (nl > 8) warp_level<16, MARK>(r0, nl, L, area, Zg, n, status, unsure);
            if (nl > 16) warp_level<32, MARK>(r0, nl, L, area, Zg, n, status, unsure);
        }
    }
    __syncthreads();
    if (nl > 32) block_level<256, MARK>(32, nl, L, area, Zg, n, red, words, status, unsure);
    if (nl > 64) block_level<512, MARK>(64, nl, L, area, Zg, n, red, words, status, unsure);
    if (tid < nl) D[c0 + tid] = L.D[tid];
}

}  // namespace
