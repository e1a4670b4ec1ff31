// Householder tridiagonalisation with the matrix resident on chip.
//
// A group of CL blocks (one block for small orders, 2..16 blocks of a cluster for larger
// ones) holds the whole symmetric block: column j belongs to block j % CL, inside the
// block to one warp (or to G warps that split the rows), rows lie across the lanes, the
// entries in registers: a column step reads no global or L2 memory.  What bounds a step is
// its dependent chain (a warp-wide FP64 sum takes 176 cycles, a square root 286, a general
// division 430, rsqrt or a reciprocal 80, a message between blocks 320..390, measured), so
// the chain is kept short:
//
// Step k uses the rank-2 form of the reduction (A <- A - v w^T - w v^T, no panel), with the
// reflector's vector not normalised: u = x - beta e, tau = 1 / (beta (beta - alpha)).
//   1. one thread per row, in every block of the group: y = A u of the previous reflector
//      and row k of A are there, the sum u.y too; w = tau y - (tau^2/2)(y.u) u and the
//      updated column x = a - u w_k - w u_k.  No reduction is needed here.
//   2. one pass over the live tile applies the pending rank-2 update and accumulates the
//      products with x (3 FMAs per element), with x(k+1) left out: the norm of x is not
//      known yet.  A ninth warp forms it meanwhile, with beta, u(k+1) = alpha - beta and
//      tau, and stores the normalised reflector.
//   3. column sums by halving exchanges; y(j) = sum + u(k+1) A(k+1, j), since row k + 1 of A
//      is sent along anyway; u.y from sums over the tile taken beside the column sums,
//      completed by the receiver with the same row.
// Two block barriers per step; between blocks one one-way message (st.async, which signals
// the receiver's mbarrier by byte count; no fence that would wait for the reflectors'
// global stores).  Two exchange buffers suffice: a block sends step k + 2 only after it
// has received all of step k + 1, which every block sends after its last read of step k's
// buffer; a block whose columns are done leaves the loop.  Nothing is sent to a block that
// will not wait for it: st.async may still be in flight when its sender has passed a cluster
// barrier, so only a receiver's wait shows that it is done and the receiver may leave.
//
// Against the panel kernels (eig_panel.cu), which stream the trailing matrix from L2 and
// cross two cluster barriers and about eight block barriers per column: 1.5..2.4 us per
// column for 6.5..7; order 128 0.20 ms for 0.9 (one block there), 512 1.2 ms for 3.3.  With this
// reduction alone whole runs went to 37.5 ms from 53 (N_keep = 250), 453 from 567 (N_keep =
// 2048 with the FDM spectrum) and 146 from 218 (eight models side by side); with the divide and
// conquer of eig_dc.cuh as well they take 21.4, 283 and 102.
#include "cta_gemm.cuh"
#include "internal.hpp"

#include <algorithm>
#include <array>
#include <atomic>
#include <cstdlib>

namespace {

constexpr int kTriWarps = 8;                        // that hold the matrix
constexpr int kTriRows = 32 * kTriWarps;            // threads with a row of the vectors
constexpr int kTriActive = kTriRows + 32;           // and the warp of the norms
// whole warpgroups are launched, so that the matrix's warps can take the registers that
// the norm's does not need: 256 x 224 + 128 x 56 = 384 x 168, what the launch allots
constexpr int kTriThreads = kTriRows + 128, kMatrixRegs = 224, kNormRegs = 56;
constexpr unsigned kAll = 0xffffffffu;

// the work of one block: its part of one matrix
struct TriTask {
    double *A, *D, *E, *TAU;   // n x n, leading dimension lda; n values each
    int n, lda;
    int variant;               // index of the plan below, -1: an idle block of the cluster
    int rank;                  // of the block in its group
};

// Plans: CL blocks, G row groups of warps, R rows per lane, C1 columns per warp.  The tile
// is 64 entries per thread where it can be (72 spill a little and still beat keeping the
// rest in shared memory: 0.92 against 0.99 ms at order 384).  An order takes the first plan
// that holds it; a plan with more blocks than needed is no faster per step (measured, one
// matrix at a time: 0.20 ms at order 128, 0.26 at 160, 0.47 at 256, 0.63 at 320, 0.92 at
// 384, 1.21 at 512).
template <int CL_, int G_, int R_, int C1_>
struct Plan {
    static constexpr int CL = CL_, G = G_, R = R_, C1 = C1_;
    static constexpr int NC = kTriWarps / G;                 // column warps
    static constexpr int NR = 32 * G * R;                    // padded rows
    static constexpr int kCols = NC * C1;                    // own columns at most
    static constexpr int kMax = NR < CL * kCols ? NR : CL * kCols;   // largest order
    // shared memory, in doubles: the exchange buffers (two of y | a per row and of the
    // blocks' parts of u.y), two barriers, v | w and x by row, the column sums by row
    // group, row k + 1 of the own columns, the warps' parts of u.y, scalars.  Row i of an
    // exchange buffer is at (i % CL) kSrc + i / CL: what one block sends is contiguous, and
    // with kSrc odd consecutive rows still lie on different banks.
    static constexpr int kSrc = kCols | 1, kEx = CL * kSrc;
    static constexpr int kBuf = 0, kUY = kBuf + (CL > 1 ? 4 * kEx : 0), kBar = kUY + 2 * CL;
    __host__ __device__ static constexpr int at(int i) { return (i % CL) * kSrc + i / CL; }
    static constexpr int kVW = kBar + 2, kX = kVW + 2 * NR, kPart = kX + NR, kRow = kPart + G * kCols;
    static constexpr int kP = kRow + kCols, kScal = kP + kTriWarps, kDoubles = kScal + 8;
    static constexpr size_t kBytes = sizeof(double) * kDoubles;
};
using PlanS = Plan<1, 1, 2, 8>;      // orders up to 64
using Plan0 = Plan<1, 1, 4, 16>;     // 128
using Plan1 = Plan<2, 1, 5, 10>;     // 160
using Plan2 = Plan<4, 2, 4, 16>;     // 256
using Plan3 = Plan<8, 2, 5, 10>;     // 320
using Plan4 = Plan<8, 2, 6, 12>;     // 384
using Plan5 = Plan<16, 4, 4, 16>;    // 512

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void send16(unsigned dst, double a, double b, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bar_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// waits for the phase of the given parity, for at most about a second
__device__ bool bar_wait(unsigned bar, unsigned parity) {
    unsigned long long t0 = 0;
    for (int it = 0; it < (1 << 24); ++it) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n"
            " mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((it & 255) == 255) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            else if (t - t0 > 1000000000ull) return false;
        }
    }
    return false;
}
__device__ __forceinline__ double bfly(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
    return v;
}
// Column sums over the 32 lanes by halving exchanges, one column per lane in the end: a
// group of four columns takes two levels (quad), up to eight groups the other three, so
// the chain is five exchanges long for any number of columns.  Lane l ends with the sum of
// column (l >> 3) of group l & 7.
__device__ __forceinline__ double quad(const double (&a)[4], int lane) {
    const bool h16 = lane & 16, h8 = lane & 8;
    double k0 = h16 ? a[2] : a[0], k1 = h16 ? a[3] : a[1];
    k0 += __shfl_xor_sync(kAll, h16 ? a[0] : a[2], 16);
    k1 += __shfl_xor_sync(kAll, h16 ? a[1] : a[3], 16);
    const double k = h8 ? k1 : k0;
    return k + __shfl_xor_sync(kAll, h8 ? k0 : k1, 8);
}
template <int N>   // groups
__device__ __forceinline__ double octet(double (&k)[8], int lane) {
#pragma unroll
    for (int h = 4; h >= 1; h >>= 1) {
        const bool up = lane & h;
#pragma unroll
        for (int g = 0; g < h; ++g) {
            if (g >= N) continue;
            const double other = g + h < N ? k[g + h] : 0.0;
            const double keep = up ? other : k[g];
            k[g] = keep + __shfl_xor_sync(kAll, up ? k[g] : other, h);
        }
    }
    return k[0];
}
__device__ __forceinline__ void send8(unsigned dst, double a, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
                 "l"(__double_as_longlong(a)), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void step_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kTriActive) : "memory"); }

template <class P>
__device__ __forceinline__ void tri_init(const TriTask& t, double* sm) {
    const int tid = threadIdx.x, n = t.n;
    // step 0 reads y = 0 and column 0, and the scalars of no reflector
    if constexpr (P::CL > 1)
        for (int i = tid; i < n; i += kTriThreads)
            reinterpret_cast<double2*>(sm + P::kBuf)[P::at(i)] = make_double2(0.0, t.A[i]);
    for (int i = tid; i < P::NR; i += kTriThreads) {
        if constexpr (P::CL == 1) if (i < P::kCols) {
            sm[P::kPart + i] = 0.0;
            sm[P::kRow + i] = i < n ? t.A[i] : 0.0;
        }
        sm[P::kVW + 2 * i] = sm[P::kVW + 2 * i + 1] = sm[P::kX + i] = 0.0;
    }
    if (tid < 2 * P::CL) sm[P::kUY + tid] = 0.0;
    if (tid < kTriWarps + 8) sm[P::kP + tid] = 0.0;
}

template <class P>
__device__ __forceinline__ void tri_load(const TriTask& t, double* sm, double (&a)[P::C1][P::R]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wc = warp / P::G, rg = warp % P::G;
    const int n = t.n;
#pragma unroll
    for (int c = 0; c < P::C1; ++c) {
        const int j = t.rank + P::CL * (wc + P::NC * c);
#pragma unroll
        for (int u = 0; u < P::R; ++u) {
            const int i = 32 * (u * P::G + rg) + lane;
            a[c][u] = (i < n && j < n) ? t.A[(size_t)i + (size_t)j * t.lda] : 0.0;
        }
    }
}

// scalars of the current reflector, from the ninth warp (after kScal)
enum { kTau = 0, kH = 1, kAlpha = 2, kDiag = 3, kScale = 4 };

// beta, tau, u(k+1) and the factor of the normalised reflector, from the sum of squares
// below alpha; un: the factor that u takes itself
struct Reflector {
    double beta, h, tau, scal, un;
};
__device__ __forceinline__ Reflector reflector(double ss, double al) {
    Reflector r{al, 0.0, 0.0, 0.0, 1.0};
    if (ss == 0.0) return r;
    const double q = fma(al, al, ss);
    // the root and the quotients from rsqrt and reciprocals: sqrt and a general division
    // take four to six times as long
    if (q > 1e-150 && q < 1e150) {
        const double s = rsqrt(q), b = q * s;
        r.beta = -copysign(fma(0.5 * s, fma(-b, b, q), b), al);
        r.h = al - r.beta;
        r.tau = 1.0 / (-r.beta * r.h);
        r.scal = 1.0 / r.h;
    } else {
        // far from one the squares and cubes of u would leave the range: normalise
        r.beta = -copysign(sqrt(q), al);
        r.un = 1.0 / (al - r.beta);
        r.tau = (r.beta - al) / r.beta;
        r.h = 1.0;
        r.scal = r.un;
    }
    return r;
}

// the norm of x, beta, tau and u(k+1) of column k, and the stores of the reflector
template <class P>
__device__ __forceinline__ void tri_norm(const TriTask& t, double* sm, int k) {
    const int lane = threadIdx.x & 31, n = t.n;
    const double* xs = sm + P::kX;
    double* sc = sm + P::kScal;
    double s0 = 0.0, s1 = 0.0;
    int i = (k & ~31) + lane;
    for (; i + 32 < n; i += 64) {
        const double x0 = xs[i], x1 = xs[i + 32];
        s0 = fma(x0, x0, s0);
        s1 = fma(x1, x1, s1);
    }
    if (i < n) s0 = fma(xs[i], xs[i], s0);
    const Reflector f = reflector(bfly(s0 + s1), sc[kAlpha]);
    if (lane == 0) {
        sc[kTau] = f.tau;
        sc[kH] = f.h;
        sc[kScale] = f.un;
    }
    if ((k + 1) % P::CL == t.rank) {   // a block that is in the loop as long as this column
        double* ref = t.A + (size_t)k * t.lda;
        for (int r = ((k + 2) & ~31) + lane; r < n; r += 32)
            if (r >= k + 2) ref[r] = xs[r] * f.scal;
        if (lane == 0) {
            t.D[k] = sc[kDiag];
            t.E[k] = f.beta;
            t.TAU[k] = f.h * f.h * f.tau;   // (beta - alpha) / beta
        }
    }
}

// whether block r of the group is in the loop at step k + 1, and so waits for what step k sends
template <class P>
__device__ __forceinline__ bool awaits(int r, int k, int n) {
    return ((r - (k + 2)) & (P::CL - 1)) <= n - 1 - (k + 2);   // it has a column from k + 2 on
}

// the steps of the ninth warp
template <class P>
__device__ __forceinline__ void tri_norm_steps(const TriTask& t, double* sm, unsigned base) {
    const int lane = threadIdx.x & 31, n = t.n;
    const int jblock = t.rank + P::CL * ((n - t.rank + P::CL - 1) / P::CL - 1);
    const unsigned bar0 = smem_addr(sm + P::kBar), uy0 = smem_addr(sm + P::kUY);
    const double *pw = sm + P::kP, *sc = sm + P::kScal;
    for (int k = 0; k < n - 1 && jblock > k; ++k) {
        step_sync();
        tri_norm<P>(t, sm, k);
        step_sync();
        if (sc[kScale] != 1.0) step_sync();
        if (P::CL > 1 && k < n - 2 && lane < P::CL && awaits<P>(lane, k, n)) {
            // the block's part of u.y
            const int nb = (k + 1) & 1;
            double s = 0.0;
#pragma unroll
            for (int r = 0; r < kTriWarps; r += 2) s += pw[r] + pw[r + 1];
            send8(map_rank(uy0 + 8 * (nb * P::CL + t.rank), base + lane), s, map_rank(bar0 + 8 * nb, base + lane));
        }
    }
}

// rank-2 update and products of the columns in registers, rows from U0 and groups of four
// columns from G0 on
template <class P, int U0, int G0, class J>
__device__ __forceinline__ void tri_pass(double (&a)[P::C1][P::R], const double (&vr)[P::R], const double (&wr)[P::R],
                                         const double (&xr)[P::R], const double2* vw, const double* xs, J jcol,
                                         double (&kk)[8], double& p, int lane) {
#pragma unroll
    for (int g = G0; g < (P::C1 + 3) / 4; ++g) {
        double acc[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            acc[c] = 0.0;
            if (4 * g + c >= P::C1) continue;
            const int j = jcol(4 * g + c);
            const double2 e = vw[j];
#pragma unroll
            for (int u = U0; u < P::R; ++u) {
                double x = a[4 * g + c][u];
                x = fma(-vr[u], e.y, x);
                x = fma(-wr[u], e.x, x);
                a[4 * g + c][u] = x;
                acc[c] = fma(x, xr[u], acc[c]);
            }
            p = fma(acc[c], xs[j], p);
        }
        kk[g] = quad(acc, lane);
    }
}

// the column steps; base: cluster rank of the group's first block
template <class P>
__device__ __forceinline__ void tri_steps(const TriTask& t, double* sm, double (&a)[P::C1][P::R], unsigned base,
                                          int* status) {
    constexpr int CL = P::CL, G = P::G, R = P::R, C1 = P::C1, NC = P::NC, NR = P::NR;
    constexpr int NG = (C1 + 3) / 4;                               // groups of four columns
    static_assert(NG <= 8, "a lane per column");
    constexpr int RT = (NR + kTriRows - 1) / kTriRows;             // rows per thread of the vectors
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wc = warp / G, rg = warp % G;
    const int n = t.n, rank = t.rank;
    const int cnt = (n - rank + CL - 1) / CL;                      // own columns of the block
    const int jblock = rank + CL * (cnt - 1);                      // the last one
    const unsigned bar0 = smem_addr(sm + P::kBar), buf0 = smem_addr(sm + P::kBuf);
    double2* vw = reinterpret_cast<double2*>(sm + P::kVW);
    double *xs = sm + P::kX, *part = sm + P::kPart, *rowv = sm + P::kRow, *pw = sm + P::kP, *sc = sm + P::kScal;
    // the last own column of this warp
    const int mlast = cnt - 1 - ((cnt - 1 - wc) % NC + NC) % NC;   // largest m <= cnt-1 with m % NC == wc
    const int jlast = mlast >= 0 ? rank + CL * mlast : -1;
    // the column of this lane after the column sums: number lane >> 3 of group lane & 7
    const int lg = lane & 7, lc = lane >> 3;
    const int ml = wc + NC * (4 * lg + lc);
    const bool has = lg < NG && 4 * lg + lc < C1 && ml < cnt;
    double v[RT];                                                  // of this thread's rows
#pragma unroll
    for (int e = 0; e < RT; ++e) v[e] = 0.0;
    bool late = false;

    for (int k = 0; k < n - 1 && jblock > k; ++k) {
        const int b = k & 1;
        if constexpr (CL > 1) {
            // after a wait that ran out the steps go on without waiting: the result is
            // flagged, and no block is left waiting for another
            if (k > 0 && !late) {
                late = !__all_sync(kAll, bar_wait(bar0 + 8 * b, ((k - 1) >> 1) & 1));
                if (late && lane == 0) atomicOr(status, NRG_DEV_TIMEOUT);
            }
            // step k + 1 brings 16 bytes per column from k + 1 on and 8 per block that has one
            if (tid == 0 && k < n - 2)
                bar_expect(bar0 + 8 * (b ^ 1), 16u * (unsigned)(n - 1 - k) + 8u * (unsigned)min(CL, n - 1 - k));
        }
        // ---- 1. w of the previous reflector and column k, one thread per row ----
        {
            const double tau = sc[kTau], h = sc[kH];
            auto ya_of = [&](int i) {
                if constexpr (CL > 1) {
                    return reinterpret_cast<const double2*>(sm + P::kBuf)[b * P::kEx + P::at(i)];
                } else {
                    double y = part[i];
#pragma unroll
                    for (int g = 1; g < G; ++g) y += part[g * P::kCols + i];
                    const double av = rowv[i];
                    return make_double2(fma(h, av, y), av);
                }
            };
            const double2 yk = ya_of(k);
            double s = 0.0;
            if constexpr (CL > 1) {
                const double* uy = sm + P::kUY + b * CL;
                if (n - 1 - k >= CL - 1 || k == 0) {
#pragma unroll
                    for (int r = 0; r < CL; r += 2) {
                        const double2 e = *reinterpret_cast<const double2*>(uy + r);
                        s += e.x + e.y;
                    }
                } else {
                    for (int r = 0; r < CL; ++r)   // the blocks that still have a column
                        if (((r - k) & (CL - 1)) <= n - 1 - k) s += uy[r];
                }
            } else {
#pragma unroll
                for (int r = 0; r < kTriWarps; r += 2) s += pw[r] + pw[r + 1];
            }
            s = fma(h, fma(-h, yk.y, 2.0 * yk.x), s);
            const double cf = -0.5 * tau * (tau * s);
            const double wk = fma(cf, h, tau * yk.x);
            if (tid == 0) sc[kDiag] = fma(-2.0 * wk, h, yk.y);
#pragma unroll
            for (int e = 0; e < RT; ++e) {
                const int i = tid + e * kTriRows;
                if (i > k && i < n) {
                    const double2 ya = ya_of(i);
                    const double w = fma(cf, v[e], tau * ya.x);
                    const double x = fma(-w, h, fma(-v[e], wk, ya.y));
                    vw[i] = make_double2(v[e], w);
                    if (i == k + 1) sc[kAlpha] = x;
                    v[e] = i == k + 1 ? 0.0 : x;
                    xs[i] = v[e];
                }
            }
        }
        step_sync();
        // ---- 2. rank-2 update and the products with x; the norm beside them ----
        const int rk = k + 1;                       // the row that goes out with the sums
        if (jlast >= rk) {
            double vr[R], wr[R], xr[R];
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int i = 32 * (u * G + rg) + lane;
                const double2 e = vw[i];
                vr[u] = e.x;
                wr[u] = e.y;
                xr[u] = xs[i];
            }
            double kk[8], p = 0.0;
#pragma unroll
            for (int g = 0; g < NG; ++g) kk[g] = 0.0;
            // straight-line code, so that the groups' chains overlap;
            // the first halves of the rows and of the groups are left out once they are done
            {
                const bool late_rows = 32 * ((R / 2 - 1) * G + rg) + 31 < rk;
                const bool late_cols = rank + CL * (wc + NC * (4 * (NG / 2) - 1)) < rk;
                auto jcol = [&](int c) { return min(rank + CL * (wc + NC * c), NR - 1); };
                if (late_rows) {
                    if (late_cols) tri_pass<P, R / 2, NG / 2>(a, vr, wr, xr, vw, xs, jcol, kk, p, lane);
                    else tri_pass<P, R / 2, 0>(a, vr, wr, xr, vw, xs, jcol, kk, p, lane);
                } else {
                    tri_pass<P, 0, 0>(a, vr, wr, xr, vw, xs, jcol, kk, p, lane);
                }
            }
            // row k + 1 of the own columns
            if ((rk >> 5) % G == rg) {
                const int uk = (rk >> 5) / G;
                if (lane == (rk & 31)) {
#pragma unroll
                    for (int u = 0; u < R; ++u)
                        if (u == uk) {
#pragma unroll
                            for (int c = 0; c < C1; ++c) rowv[wc + NC * c] = a[c][u];
                        }
                }
            }
            p = bfly(p);
            const double tot = octet<NG>(kk, lane);
            if (has) part[rg * P::kCols + ml] = tot;
            if (lane == 0) pw[warp] = p;
        } else if (lane == 0) {
            pw[warp] = 0.0;
        }
        step_sync();
        {
            const double un = sc[kScale];
            if (un != 1.0) {
                // the rare normalised reflector: what was formed with x takes the factor
#pragma unroll
                for (int e = 0; e < RT; ++e) v[e] *= un;
                if (has && jlast >= rk) part[rg * P::kCols + ml] *= un;
                if (tid < kTriWarps) pw[tid] *= un * un;
                step_sync();
            }
        }
        if constexpr (CL > 1) {
            // ---- 3. the sums and row k + 1 of the own columns to every block ----
            if (k < n - 2) {
                const double h = sc[kH];
                const unsigned bar = bar0 + 8 * (b ^ 1);
                // a warp sends 32 columns to one block at a time
                constexpr int kParts = (P::kCols + 31) / 32;
                for (int e = warp; e < CL * kParts; e += kTriWarps) {
                    const int r = e % CL, m = 32 * (e / CL) + lane;
                    if (m < cnt && rank + CL * m >= rk && awaits<P>(r, k, n)) {
                        double y = part[m];
#pragma unroll
                        for (int g = 1; g < G; ++g) y += part[g * P::kCols + m];
                        const double av = rowv[m];
                        send16(map_rank(buf0 + 16 * ((b ^ 1) * P::kEx + rank * P::kSrc + m), base + r), fma(h, av, y), av,
                               map_rank(bar, base + r));
                    }
                }
            }
        }
        // the last diagonal entry: row n - 1 of column n - 1, updated in this pass
        if (k == n - 2 && jblock == n - 1 && tid == 0) {
            t.D[n - 1] = rowv[cnt - 1];
            t.E[n - 1] = 0.0;
        }
    }
}

// IN_CLUSTER: the launch has clusters, whose blocks meet once before the steps
template <class P, bool IN_CLUSTER>
__device__ __forceinline__ void tri_run(const TriTask& t, double* sm, unsigned cta, int* status) {
    const int warp = threadIdx.x >> 5;
    tri_init<P>(t, sm);
    if (P::CL > 1 && threadIdx.x == 0) {
        const unsigned bar = smem_addr(sm + P::kBar);
        bar_init(bar);
        bar_init(bar + 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // every block of the group has loaded its columns and set up its barriers before the
    // first of them sends, or stores a reflector
    auto meet = [&]() {
        __syncthreads();
        if constexpr (IN_CLUSTER) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        if constexpr (P::CL > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    };
    const unsigned base = cta - (unsigned)t.rank;
    if (warp < kTriWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kMatrixRegs));
        double a[P::C1][P::R];
        tri_load<P>(t, sm, a);
        meet();
        tri_steps<P>(t, sm, a, base, status);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kNormRegs));
        meet();
        if (warp == kTriWarps) tri_norm_steps<P>(t, sm, base);
    }
    if constexpr (IN_CLUSTER && P::CL == 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// MAXCL: cluster size of the launch
template <int MAXCL>
__global__ void __launch_bounds__(kTriThreads, 1) k_tri_res(const TriTask* __restrict__ tasks, int* status) {
    extern __shared__ __align__(16) double tri_sm[];
    const TriTask t = tasks[blockIdx.x];
    unsigned cta = 0;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(cta));
    bool ran = true;
    if (MAXCL == 8 && t.variant == 0) tri_run<Plan0, true>(t, tri_sm, cta, status);
    else if (MAXCL == 8 && t.variant == 1) tri_run<Plan1, true>(t, tri_sm, cta, status);
    else if (MAXCL == 8 && t.variant == 2) tri_run<Plan2, true>(t, tri_sm, cta, status);
    else if (MAXCL == 8 && t.variant == 3) tri_run<Plan3, true>(t, tri_sm, cta, status);
    else if (MAXCL == 8 && t.variant == 4) tri_run<Plan4, true>(t, tri_sm, cta, status);
    else if (MAXCL == 16 && t.variant == 5) tri_run<Plan5, true>(t, tri_sm, cta, status);
    else ran = false;
    __syncwarp();
    if (!ran) asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
    // the blocks leave together (every message to one of them has been waited for)
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// ---------------------------------------------------------------------------------
// larger orders: the matrix streamed from L2 until the trailing block fits on chip
// ---------------------------------------------------------------------------------
// The same step with the tile in global memory (L2): column j in block j % CL, columns
// full.  Up to NBS rank-2 updates are kept back as vectors u_q, w_q, replicated in every
// block's shared memory, so that a step only reads the matrix; then one pass applies them
// (FP64 MMA, inner length 2 NBS).  The sums that arrive are those of the matrix as stored:
//   a = A(k, :) - sum_q (u_q(k) w_q + w_q(k) u_q),   y = A x - sum_q (u_q (w_q.x) + w_q (u_q.x)),
// with w_q.x and u_q.x from a run of rows per block, sent beside the column sums: still one
// message per step.  The first such pass moves the matrix to columns that start on 128 bytes
// (odd orders put every other column off by 8, and a load of a warp then touches a line more:
// 10.0 against 9.3 thousand cycles for a product of order 870 on average); the last one brings
// the trailing block back.  Bound by the L2 stream of a block (8 m^2 / CL bytes per step, m the
// trailing order, at 40 of the 44..48 bytes per cycle that eight warps reach) and, below m
// of about 600, by the chain of the step.  Order 1225: 9.1 ms to order 512 (9.8 before the
// aligned columns and the 16 x 8 x 8 MMA on row pairs) and 1.1 ms on chip, against 17.2 ms of
// eig_panel.cu's cluster kernel (panels of 32 columns, two cluster barriers per column, 8 blocks;
// with 16 that one is no faster).
constexpr int kStreamSlots = 7;   // kept updates at most (NBS), fewer where they do not fit

struct StreamTask {
    double *A, *D, *E, *TAU, *P;   // P: n columns of stream_ld(n), 128-byte aligned
    int n, stop, rank, keep;       // stop: columns to reduce; keep: updates kept back
};

__host__ __device__ inline int stream_ld(int n) { return (n + 1 + 15) & ~15; }

struct StreamLayout {
    int ld, nr, cols, keep;
    __host__ __device__ StreamLayout(int n, int CL, int keep_) {
        ld = ((n + 1 + 15) & ~15) + 4;            // = 4 mod 16: conflict-free MMA operands
        cols = ((n + CL - 1) / CL) | 1;           // row i of an exchange buffer: (i % CL) cols + i / CL
        nr = CL * cols;
        keep = keep_;
    }
    __host__ __device__ int u() const { return 0; }
    __host__ __device__ int w() const { return (keep + 1) * ld; }
    __host__ __device__ int buf() const { return 2 * (keep + 1) * ld; }
    __host__ __device__ int dots(int) const { return buf() + 4 * nr; }
    __host__ __device__ int uy(int CL) const { return dots(CL) + 4 * keep * CL; }
    __host__ __device__ int bar(int CL) const { return uy(CL) + 2 * CL; }
    __host__ __device__ int tsum(int CL) const { return bar(CL) + 2; }
    __host__ __device__ int part(int CL) const { return tsum(CL) + 8 * kStreamSlots; }
    __host__ __device__ int row(int CL) const { return part(CL) + cols; }
    __host__ __device__ int p(int CL) const { return (row(CL) + cols + 1) & ~1; }
    __host__ __device__ int scal(int CL) const { return p(CL) + kTriWarps; }
    __host__ __device__ int doubles(int CL) const { return scal(CL) + 8; }
};

// the sums over the warp of four values: lane l ends with the total of value (l >> 3) & 3
__device__ __forceinline__ double sum4(const double (&a)[4], int lane) {
    double k = quad(a, lane);
    k += __shfl_xor_sync(kAll, k, 4);
    k += __shfl_xor_sync(kAll, k, 2);
    return k + __shfl_xor_sync(kAll, k, 1);
}

// the ninth warp: norm of the new column, reflector, the block's sums of u.y and of the kept
// updates' products
template <int CL>
__device__ __forceinline__ void stream_norm_steps(const StreamTask& t, double* sm, unsigned to0) {
    const int n = t.n, rank = t.rank, keep = t.keep;
    const StreamLayout lay(n, CL, keep);
    const int lane = threadIdx.x & 31;
    double* U = sm + lay.u();
    double *tsum = sm + lay.tsum(CL), *pw = sm + lay.p(CL), *sc = sm + lay.scal(CL);
    const unsigned bar0 = smem_addr(sm + lay.bar(CL)), uy0 = smem_addr(sm + lay.uy(CL)), dots0 = smem_addr(sm + lay.dots(CL));
    const int ld = lay.ld;
    const int par = (int)(((reinterpret_cast<uintptr_t>(t.A) >> 3) + (uintptr_t)rank * n) & 1);
    int np = 0;                            // kept updates (complete pairs)
    for (int k = 0; k <= t.stop; ++k) {
        const int b = k & 1;
        const bool fin = k == t.stop;      // only completes the last update and applies what is kept
        const int full = np + (k > 0);     // pairs once this step has formed w
        const bool apply = fin || full == keep;
        const int next = apply ? 0 : full;
        const int nw = full * ld + par;    // the new column
        step_sync();
        if (fin) break;
        // the norm of the new column, beta, u(k+1) and tau; the reflector's stores
        const double* xs = U + nw;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int i = k + 2 + lane;
        for (; i + 96 < n; i += 128) {
            s0 = fma(xs[i], xs[i], s0);
            s1 = fma(xs[i + 32], xs[i + 32], s1);
            s2 = fma(xs[i + 64], xs[i + 64], s2);
            s3 = fma(xs[i + 96], xs[i + 96], s3);
        }
        for (; i < n; i += 32) s0 = fma(xs[i], xs[i], s0);
        const Reflector r = reflector(bfly((s0 + s1) + (s2 + s3)), sc[kAlpha]);
        if (lane == 0) {
            sc[kTau] = r.tau;
            sc[kH] = r.h;
            sc[kScale] = r.un;
        }
        if ((k + 1) % CL == rank) {
            double* ref = t.A + (size_t)k * n;
            for (int e = k + 2 + lane; e < n; e += 32) ref[e] = xs[e] * r.scal;
            if (lane == 0) {
                t.D[k] = sc[kDiag];
                t.E[k] = r.beta;
                t.TAU[k] = r.h * r.h * r.tau;   // (beta - alpha) / beta
            }
        }
        step_sync();
        if (sc[kScale] != 1.0) step_sync();
        const unsigned bar = bar0 + 8 * (b ^ 1);
        if (lane < CL) {
            double s = 0.0;
#pragma unroll
            for (int r = 0; r < kTriWarps; r += 2) s += pw[r] + pw[r + 1];
            send8(map_rank(uy0 + 8 * ((b ^ 1) * CL + rank), to0 + lane), s, map_rank(bar, to0 + lane));
        }
        for (int e = lane; e < next * CL; e += 32) {
            const int q = e / CL, r = e % CL;
            send16(map_rank(dots0 + 16 * (((b ^ 1) * keep + q) * CL + rank), to0 + r), tsum[8 * q], tsum[8 * q + 1],
                   map_rank(bar, to0 + r));
        }
        np = next;
    }
}

template <int CL>
__device__ __forceinline__ void stream_steps(const StreamTask& t, double* sm, unsigned to0, int* status) {
    constexpr int NBS = kStreamSlots;
    const int n = t.n, rank = t.rank, keep = t.keep;
    const StreamLayout lay(n, CL, keep);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *U = sm + lay.u(), *W = sm + lay.w();
    double* tsum = sm + lay.tsum(CL);      // (w_q.x, u_q.x) of the kept updates
    double* part = sm + lay.part(CL);
    double* rowv = sm + lay.row(CL);
    double* pw = sm + lay.p(CL);
    double* sc = sm + lay.scal(CL);
    const unsigned bar0 = smem_addr(sm + lay.bar(CL)), buf0 = smem_addr(sm + lay.buf());
    const int cnt = (n - rank + CL - 1) / CL, ld = lay.ld;
    // CL is even, so every own column's offset (rank + CL m) n has the parity of rank n; with
    // vectors stored from index par on, rows pair up on 16-byte boundaries in A and in them
    const int par = (int)(((reinterpret_cast<uintptr_t>(t.A) >> 3) + (uintptr_t)rank * n) & 1);
    auto first_own = [&](int i0) { return (i0 - rank + CL - 1) / CL; };
    auto ex = [&](int i) { return (int)((unsigned)i % CL) * lay.cols + (int)((unsigned)i / CL); };
    int np = 0;                            // kept updates (complete pairs), u_q and w_q in slot q
    const int ldp = stream_ld(n);
    bool packed = true;                    // the matrix is still in A
    bool late = false;
    for (int k = 0; k <= t.stop; ++k) {
        const int b = k & 1;
        const bool fin = k == t.stop;      // only completes the last update and applies what is kept
        const int full = np + (k > 0);     // pairs once this step has formed w
        const bool apply = fin || full == keep;
        const int next = apply ? 0 : full;
        const int cur = np * ld + par, nw = full * ld + par;   // u of the last reflector, the new column
        if (k > 0 && !late) {
            late = !__all_sync(kAll, bar_wait(bar0 + 8 * b, ((k - 1) >> 1) & 1));
            if (late && lane == 0) atomicOr(status, NRG_DEV_TIMEOUT);
        }
        // step k + 1 brings the columns from k + 1 on, and from every block its parts of
        // u.y and of the kept updates' products
        if (tid == 0 && !fin && k < t.stop)
            bar_expect(bar0 + 8 * (b ^ 1), 16u * (unsigned)(n - 1 - k) + (8u + 16u * (unsigned)next) * CL);
        if (np > 0) {
            // totals over the blocks and what a kept update adds at row k: one warp each
            if (warp < np) {
                const double2* in = reinterpret_cast<const double2*>(sm + lay.dots(CL)) + (b * keep + warp) * CL;
                double2 e = lane < CL ? in[lane] : make_double2(0.0, 0.0);
                const double u = U[warp * ld + par + k], w = W[warp * ld + par + k];
                e.x = bfly(e.x);
                e.y = bfly(e.y);
                if (lane == 0) {
                    double2* o = reinterpret_cast<double2*>(tsum + 8 * warp);
                    o[0] = e;
                    o[1] = make_double2(u, w);
                    o[2] = make_double2(fma(u, e.x, w * e.y), 2.0 * u * w);
                    o[3].x = 2.0 * e.x * e.y;
                }
            }
            asm volatile("bar.sync 2, %0;" ::"n"(kTriRows) : "memory");
        }
        // ---- 1. w of the last reflector and column k ----
        const double tau = sc[kTau], h = sc[kH];
        const double2* in = reinterpret_cast<const double2*>(sm + lay.buf()) + b * lay.nr;
        double uk[NBS], wk[NBS], t1[NBS], t2[NBS];
        double2 yk = in[ex(k)];
        double s = 0.0;
        {
            const double2* uy = reinterpret_cast<const double2*>(sm + lay.uy(CL) + b * CL);
#pragma unroll
            for (int r = 0; r < CL / 2; ++r) s += uy[r].x + uy[r].y;
        }
#pragma unroll
        for (int q = 0; q < NBS; ++q) {
            uk[q] = wk[q] = t1[q] = t2[q] = 0.0;
            if (q < np) {
                const double2* o = reinterpret_cast<const double2*>(tsum + 8 * q);
                const double2 e0 = o[0], e1 = o[1], e2 = o[2];
                t1[q] = e0.x;
                t2[q] = e0.y;
                uk[q] = e1.x;
                wk[q] = e1.y;
                yk.x -= e2.x;
                yk.y -= e2.y;
                s -= o[3].x;
            }
        }
        yk.x = fma(h, yk.y, yk.x);
        s = fma(h, fma(-h, yk.y, 2.0 * yk.x), s);
        const double cf = -0.5 * tau * (tau * s);
        const double wpiv = fma(cf, h, tau * yk.x);
        if (tid == 0) sc[kDiag] = fma(-2.0 * wpiv, h, yk.y);
        for (int i = k + 1 + tid; i < n; i += kTriRows) {
            double2 ya = in[ex(i)];
#pragma unroll
            for (int q = 0; q < NBS; ++q)
                if (q < np) {
                    const double uq = U[q * ld + par + i], wq = W[q * ld + par + i];
                    ya.y = fma(-uk[q], wq, fma(-wk[q], uq, ya.y));
                    ya.x = fma(-uq, t1[q], fma(-wq, t2[q], ya.x));
                }
            ya.x = fma(h, ya.y, ya.x);
            const double u = k > 0 ? U[cur + i] : 0.0;
            const double w = fma(cf, u, tau * ya.x);
            if (k > 0) W[cur + i] = w;
            if (!fin) {
                const double x = fma(-w, h, fma(-u, wpiv, ya.y));
                if (i == k + 1) sc[kAlpha] = x;
                U[nw + i] = i == k + 1 ? 0.0 : x;
            }
        }
        if (fin) {
            // the last reflector's entries at row k, which stays in the trailing block
            if (tid == 0) {
                U[cur + k] = h;
                W[cur + k] = wpiv;
            }
        } else if (tid < 16 && tid <= k) {
            U[nw + k - tid] = 0.0;     // a product that starts up to 15 rows early
        }
        step_sync();
        // ---- 2. products with the new column; every warp keeps its own columns, warp + 8 i of
        // the block's ----
        const double* xs = U + nw;
        const int r0 = fin ? k : k + 1, mR = first_own(r0);
        const int lds = packed ? n : ldp, rs = r0 - ((r0 + par) & (packed && !(apply && full > 0) ? 1 : 15));
        const double* src = packed ? t.A : t.P + par;
        const int mw = mR + ((warp - mR) & (kTriWarps - 1));           // the warp's first live column
        if (apply && full > 0) {
            // the kept updates go into the matrix on the way: 8 columns x RU rows at a time as MMA
            // accumulators, the next rows' entries loaded meanwhile.  Row 2 g + h of 16 rows is
            // row g of tile h, so that a lane loads and stores row pairs.  Rows before the trailing
            // block's are dead storage, rows and columns beyond the end are not stored.
            constexpr int TU = 4, RU = 16 * TU;
            const int g = lane >> 2, q4 = lane & 3;
            double* dst = fin ? t.A : t.P + par;
            const int ldd = fin ? n : ldp;
            int pa[4], pb[4];              // offsets in shared memory
            bool have[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int q = 4 * e + q4, at = (q < full ? q : q - full) * ld + par;
                have[e] = q < 2 * full;
                pa[e] = (have[e] ? (q < full ? lay.u() : lay.w()) + at : par) + 2 * g;
                pb[e] = have[e] ? (q < full ? lay.w() : lay.u()) + at : par;
            }
            for (int m0 = mw; m0 < cnt; m0 += 8 * kTriWarps) {
                const int lb = rank + CL * min(m0 + kTriWarps * g, cnt - 1);
                double bf[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) bf[e] = have[e] ? -sm[pb[e] + lb] : 0.0;
                const int mc0 = m0 + 2 * kTriWarps * q4, mc1 = mc0 + kTriWarps;
                const size_t j0 = rank + CL * min(mc0, cnt - 1), j1 = rank + CL * min(mc1, cnt - 1);
                const double *c0 = src + j0 * lds + 2 * g, *c1 = src + j1 * lds + 2 * g;
                double *d0 = dst + j0 * ldd + 2 * g, *d1 = dst + j1 * ldd + 2 * g;
                double s0 = 0.0, s1 = 0.0;
                auto fetch = [&](int R, double2 (&x)[TU][2]) {
                    const double *p0 = c0 + R, *p1 = c1 + R;
                    if (R + RU <= n) {
#pragma unroll
                        for (int u = 0; u < TU; ++u) {
                            x[u][0] = *reinterpret_cast<const double2*>(p0 + 16 * u);
                            x[u][1] = *reinterpret_cast<const double2*>(p1 + 16 * u);
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < TU; ++u) {
                            const int i = R + 2 * g + 16 * u;
                            x[u][0] = x[u][1] = make_double2(0.0, 0.0);
                            if (i + 1 < n) {
                                x[u][0] = *reinterpret_cast<const double2*>(p0 + 16 * u);
                                x[u][1] = *reinterpret_cast<const double2*>(p1 + 16 * u);
                            } else if (i < n) {
                                x[u][0].x = p0[16 * u];
                                x[u][1].x = p1[16 * u];
                            }
                        }
                    }
                };
                const bool in0 = mc0 < cnt, in1 = mc1 < cnt;
                auto apply_at = [&](int R, double2 (&x)[TU][2]) {
#pragma unroll
                    for (int e = 0; e < 4; e += 2)
                        if (4 * e < 2 * full) {
                            // beyond n it reads on into what follows the vector: rows that are not kept
                            const double *lo = sm + pa[e] + R, *hi = sm + pa[e + 1] + R;
#pragma unroll
                            for (int u = 0; u < TU; ++u)
                                nrg::cta_dmma16(x[u][0].x, x[u][1].x, x[u][0].y, x[u][1].y,
                                                *reinterpret_cast<const double2*>(lo + 16 * u),
                                                *reinterpret_cast<const double2*>(hi + 16 * u), bf[e], bf[e + 1]);
                        }
                    double *o0 = d0 + R, *o1 = d1 + R;
                    const double* xr = xs + R + 2 * g;
                    if (R + RU <= n && !(fin && R == rs)) {
#pragma unroll
                        for (int u = 0; u < TU; ++u) {
                            if (in0) *reinterpret_cast<double2*>(o0 + 16 * u) = x[u][0];
                            if (in1) *reinterpret_cast<double2*>(o1 + 16 * u) = x[u][1];
                            const double2 xv = *reinterpret_cast<const double2*>(xr + 16 * u);
                            s0 = fma(x[u][0].y, xv.y, fma(x[u][0].x, xv.x, s0));
                            s1 = fma(x[u][1].y, xv.y, fma(x[u][1].x, xv.x, s1));
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < TU; ++u) {
                            const int i = R + 2 * g + 16 * u;
                            if (i + 1 < n) {
                                const bool kept = !fin || i + 1 >= r0;
                                if (kept && in0) *reinterpret_cast<double2*>(o0 + 16 * u) = x[u][0];
                                if (kept && in1) *reinterpret_cast<double2*>(o1 + 16 * u) = x[u][1];
                                const double2 xv = *reinterpret_cast<const double2*>(xr + 16 * u);
                                s0 = fma(x[u][0].y, xv.y, fma(x[u][0].x, xv.x, s0));
                                s1 = fma(x[u][1].y, xv.y, fma(x[u][1].x, xv.x, s1));
                            } else if (i < n) {
                                if (in0) o0[16 * u] = x[u][0].x;
                                if (in1) o1[16 * u] = x[u][1].x;
                                s0 = fma(x[u][0].x, xr[16 * u], s0);
                                s1 = fma(x[u][1].x, xr[16 * u], s1);
                            }
                        }
                    }
                    if (R == rs && g == (r0 - rs) >> 1 && !fin) {   // row k + 1
                        const bool odd = (r0 - rs) & 1;
                        if (in0) rowv[mc0] = odd ? x[0][0].y : x[0][0].x;
                        if (in1) rowv[mc1] = odd ? x[0][1].y : x[0][1].x;
                    }
                };
                double2 x[TU][2], y[TU][2];
                fetch(rs, x);
                for (int R = rs; R < n; R += 2 * RU) {
                    if (R + RU < n) fetch(R + RU, y);
                    apply_at(R, x);
                    if (R + 2 * RU < n) fetch(R + 2 * RU, x);
                    if (R + RU < n) apply_at(R + RU, y);
                }
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    s0 += __shfl_xor_sync(kAll, s0, o);
                    s1 += __shfl_xor_sync(kAll, s1, o);
                }
                if (g == 0 && !fin) {
                    if (in0) part[mc0] = s0;
                    if (in1) part[mc1] = s1;
                }
            }
            packed = false;
        } else {
            // three columns at a time in parts of 256 rows, 16-byte loads of row pairs, the next
            // part's loads in flight.  Pairs beyond the end repeat the last whole one against a
            // zero; the last row is taken by itself when it has no partner.
            const int pend = rs + 2 * ((n - rs) / 2);                  // end of the whole pairs
            for (int m0 = mw; m0 < cnt; m0 += 3 * kTriWarps) {
                const double* col[3];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    col[c] = src + (size_t)(rank + CL * min(m0 + kTriWarps * c, cnt - 1)) * lds + 2 * lane;
                auto fetch = [&](int R, double2 (&x)[3][4]) {
                    if (R + 256 <= pend) {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
#pragma unroll
                            for (int c = 0; c < 3; ++c) x[c][u] = *reinterpret_cast<const double2*>(col[c] + R + 64 * u);
                    } else {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int i = min(R + 64 * u, pend - 2 - 2 * lane);
#pragma unroll
                            for (int c = 0; c < 3; ++c) x[c][u] = *reinterpret_cast<const double2*>(col[c] + i);
                        }
                    }
                };
                double sum[4] = {0.0, 0.0, 0.0, 0.0};
                auto use = [&](int R, const double2 (&x)[3][4]) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int i = R + 64 * u + 2 * lane;
                        double2 xv = make_double2(0.0, 0.0);
                        if (i < pend) xv = *reinterpret_cast<const double2*>(xs + i);
#pragma unroll
                        for (int c = 0; c < 3; ++c) sum[c] = fma(x[c][u].y, xv.y, fma(x[c][u].x, xv.x, sum[c]));
                    }
                };
                double2 x[3][4], y[3][4];
                fetch(rs, x);
                if (lane == (r0 - rs) >> 1) {  // row k + 1 of these columns
#pragma unroll
                    for (int c = 0; c < 3; ++c)
                        if (m0 + kTriWarps * c < cnt) rowv[m0 + kTriWarps * c] = (r0 - rs) & 1 ? x[c][0].y : x[c][0].x;
                }
                if (lane == 0 && pend < n) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) sum[c] = col[c][n - 1] * xs[n - 1];
                }
                for (int R = rs; R < pend; R += 512) {
                    if (R + 256 < pend) fetch(R + 256, y);
                    use(R, x);
                    if (R + 512 < pend) fetch(R + 512, x);
                    if (R + 256 < pend) use(R + 256, y);
                }
                const double tot = sum4(sum, lane);
                const int mc = m0 + kTriWarps * ((lane >> 3) & 3);
                if ((lane & 7) == 0 && (lane >> 3) < 3 && mc < cnt) part[mc] = tot;
            }
        }
        if (!fin) {
            // the warp's part of u.y
            __syncwarp();
            double yv = 0.0;
            for (int m = mw + kTriWarps * lane; m < cnt; m += 32 * kTriWarps) yv = fma(part[m], xs[rank + CL * m], yv);
            yv = bfly(yv);
            if (lane == 0) pw[warp] = yv;
            // the kept updates' products with the new column: every block takes a run of rows
            if (warp < next) {
                const double *uq = U + warp * ld + par, *wq = W + warp * ld + par;
                double d1 = 0.0, d2 = 0.0;
                const int run = (n - k - 2 + CL - 1) / CL, end = min(n, k + 2 + (rank + 1) * run);
                for (int i = k + 2 + rank * run + lane; i < end; i += 32) {
                    const double x = xs[i];
                    d1 = fma(wq[i], x, d1);
                    d2 = fma(uq[i], x, d2);
                }
                d1 = bfly(d1);
                d2 = bfly(d2);
                if (lane == 0) tsum[8 * warp] = d1, tsum[8 * warp + 1] = d2;
            }
        }
        if (fin) break;
        step_sync();
        const double un = sc[kScale];
        if (un != 1.0) {
            // the rare normalised reflector: what was formed with the column takes the factor
            for (int i = k + 2 + tid; i < n; i += kTriRows) U[nw + i] *= un;
            for (int m = tid; m < cnt; m += kTriRows) part[m] *= un;
            if (tid < kTriWarps) pw[tid] *= un * un;
            if (tid < 2 * next) tsum[8 * (tid >> 1) + (tid & 1)] *= un;
            step_sync();
        }
        // ---- 3. sums, row k + 1 and the parts of the dot products to every block ----
        const unsigned bar = bar0 + 8 * (b ^ 1);
        // a warp sends 32 columns to one block at a time
        const int mB = first_own(k + 1);
        const int parts = (cnt - mB + 31) / 32;
        for (int e = warp; e < CL * parts; e += kTriWarps) {
            const int r = e % CL, m = mB + 32 * (e / CL) + lane;
            if (m >= cnt) continue;
            send16(map_rank(buf0 + 16 * ((b ^ 1) * lay.nr + rank * lay.cols + m), to0 + r), part[m], rowv[m],
                   map_rank(bar, to0 + r));
        }
        // after the updates went in, the new column is the first one kept
        if (apply)
            for (int i = k + 2 + tid; i < n; i += kTriRows) U[par + i] = U[nw + i];
        np = next;
    }
}

template <int CL>
__global__ void __launch_bounds__(kTriThreads, 1) k_tri_stream(const StreamTask* __restrict__ tasks, int* status) {
    extern __shared__ __align__(16) double tri_sm[];
    const StreamTask t = tasks[blockIdx.x];
    const int tid = threadIdx.x, warp = tid >> 5;
    double* sm = tri_sm;
    {
        const StreamLayout lay(t.n, CL, t.keep);
        for (int i = tid; i < lay.doubles(CL); i += kTriThreads) sm[i] = 0.0;
        __syncthreads();
        // step 0 reads y = 0 and column 0
        for (int i = tid; i < t.n; i += kTriThreads) sm[lay.buf() + 2 * ((i % CL) * lay.cols + i / CL) + 1] = t.A[i];
        if (tid == 0) {
            const unsigned bar = smem_addr(sm + lay.bar(CL));
            bar_init(bar);
            bar_init(bar + 8);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    __syncthreads();
    // no block stores a reflector before every block has read column 0
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
    unsigned cta;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(cta));
    const unsigned to0 = cta - (unsigned)t.rank;
    if (warp < kTriWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kMatrixRegs));
        stream_steps<CL>(t, sm, to0, status);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kNormRegs));
        if (warp == kTriWarps) stream_norm_steps<CL>(t, sm, to0);
    }
    // the blocks leave together: every message to one of them has been waited for, the last of
    // them at the step that only completes the last update
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// the sectors of order <= 128, one block each: D, E and tau go where k_syev reads them
__global__ void __launch_bounds__(kTriThreads, 1) k_tri_small(const SyevSector* __restrict__ secs, double* eigbuf,
                                                             double* wsd, int* status) {
    extern __shared__ __align__(16) double tri_sm[];
    const SyevSector sec = secs[blockIdx.x];
    if (sec.n < 2) return;
    TriTask t;
    t.A = eigbuf + sec.a_off;
    t.n = t.lda = sec.n;
    t.D = wsd + sec.w_off + syev_vec_off(sec.n);
    t.E = t.D + sec.n;
    t.TAU = t.E + sec.n;
    t.rank = 0;
    t.variant = 0;
    // a block holding NaN or Inf is left as it is: k_syev looks at the same entries and
    // reports it
    bool bad = false;
    for (int e = threadIdx.x; e < t.n * t.n; e += kTriThreads) bad |= !isfinite(t.A[e]);
    if (__syncthreads_or(bad)) return;
    if (t.n <= PlanS::NR) tri_run<PlanS, false>(t, tri_sm, 0, status);
    else tri_run<Plan0, false>(t, tri_sm, 0, status);
}

constexpr long long kSmemMax = 232448;   // 227 KB, the most one block may use
constexpr int kPlans = 6, kPlanCL[kPlans] = {1, 2, 4, 8, 8, 16};
constexpr int kPlanMax[kPlans] = {Plan0::kMax, Plan1::kMax, Plan2::kMax, Plan3::kMax, Plan4::kMax, Plan5::kMax};
constexpr size_t kPlanBytes[kPlans] = {Plan0::kBytes, Plan1::kBytes, Plan2::kBytes, Plan3::kBytes, Plan4::kBytes,
                                       Plan5::kBytes};

template <int MAXCL>
void cluster_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int blocks, size_t smem, cudaStream_t st) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3((unsigned)blocks);
    cfg->blockDim = dim3(kTriThreads);
    cfg->dynamicSmemBytes = smem;
    cfg->stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = MAXCL;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
}
template <int MAXCL>
int launch_clusters(nrg_context* ctx, const TriTask* d_tasks, int blocks, size_t smem, int* d_status) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    cluster_config<MAXCL>(&cfg, at, blocks, smem, ctx->stream);
    if (MAXCL > 8) NRG_CUDA_TRY(cudaFuncSetAttribute(k_tri_res<MAXCL>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    NRG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_tri_res<MAXCL>, d_tasks, d_status));
    ctx->launches++;
    return NRG_OK;
}

}  // namespace

namespace nrg {

// clusters of 16 blocks are beyond the portable size: where the device cannot place one,
// the plans of 8 blocks are the largest (NRG_TRI_CLUSTER=8 leaves 16 out: a test aid)
int tri_resident_max() {
    static const bool narrow = [] {
        const char* e = getenv("NRG_TRI_CLUSTER");
        return e && e[0] == '8' && e[1] == 0;
    }();
    if (narrow) return kPlanMax[kPlans - 2];
    static std::atomic<int> known[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return kPlanMax[kPlans - 2];
    int m = known[dev].load();
    if (m == 0) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        cluster_config<16>(&cfg, at, 16, kPlanBytes[kPlans - 1], nullptr);
        int clusters = 0;
        const bool ok =
            cudaFuncSetAttribute(k_tri_res<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, k_tri_res<16>, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) cudaGetLastError();
        m = kPlanMax[ok ? kPlans - 1 : kPlans - 2];
        known[dev].store(m);
    }
    return m;
}

// blocks of a streaming cluster: what fits in the shared memory of 8 is a little less than of 16
static int stream_cluster() { return tri_resident_max() == kPlanMax[kPlans - 1] ? 16 : 8; }

int tri_stream_max() {
    static const std::array<int, 2> most = [] {
        std::array<int, 2> m = {2, 2};
        for (int i = 0; i < 2; ++i)
            while (8LL * StreamLayout(m[i] + 1, 8 << i, 1).doubles(8 << i) <= kSmemMax) ++m[i];
        return m;
    }();
    return most[stream_cluster() / 16];
}

int tri_stream(nrg_context* ctx, const std::vector<TriItem>& items, DevBuf& buf) {
    if (items.empty()) return NRG_OK;
    const int CL = stream_cluster();
    std::vector<StreamTask> tasks;
    size_t smem = 0;
    for (const TriItem& it : items) {
        int keep = kStreamSlots;
        while (keep > 1 && 8LL * StreamLayout(it.n, CL, keep).doubles(CL) > kSmemMax) --keep;
        smem = std::max(smem, sizeof(double) * (size_t)StreamLayout(it.n, CL, keep).doubles(CL));
        for (int r = 0; r < CL; ++r) tasks.push_back(StreamTask{it.A, it.D, it.E, it.TAU, it.P, it.n, it.stop, r, keep});
    }
    if (smem > (size_t)kSmemMax) {
        nrg_set_error_message("order %d exceeds the streamed tridiagonalisation", items[0].n);
        return NRG_ERR_TOO_LARGE;
    }
    NRG_TRY(buf.ensure(sizeof(StreamTask) * tasks.size()));
    NRG_TRY(h2d_async(ctx, buf.p, tasks.data(), sizeof(StreamTask) * tasks.size()));
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    const int blocks = (int)tasks.size();
    if (CL == 16) {
        NRG_TRY(raise_smem_limit((const void*)k_tri_stream<16>, smem));
        NRG_CUDA_TRY(cudaFuncSetAttribute(k_tri_stream<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cluster_config<16>(&cfg, at, blocks, smem, ctx->stream);
        NRG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_tri_stream<16>, (const StreamTask*)buf.as<StreamTask>(), ctx->d_status.as<int>()));
    } else {
        NRG_TRY(raise_smem_limit((const void*)k_tri_stream<8>, smem));
        cluster_config<8>(&cfg, at, blocks, smem, ctx->stream);
        NRG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_tri_stream<8>, (const StreamTask*)buf.as<StreamTask>(), ctx->d_status.as<int>()));
    }
    ctx->launches++;
    return NRG_OK;
}

int tri_resident(nrg_context* ctx, const std::vector<TriItem>& items, DevBuf& buf) {
    if (items.empty()) return NRG_OK;
    // each item takes the fewest blocks that hold it; groups of one size follow one
    // another from the widest down, so a group never straddles two clusters
    std::vector<std::pair<int, int>> order;   // (plan, item)
    for (int i = 0; i < (int)items.size(); ++i) {
        int p = 0;
        while (p < kPlans && items[i].n > kPlanMax[p]) ++p;
        if (p == kPlans) {
            nrg_set_error_message("order %d exceeds the resident tridiagonalisation", items[i].n);
            return NRG_ERR_TOO_LARGE;
        }
        order.push_back({p, i});
    }
    std::stable_sort(order.begin(), order.end(), [&](const std::pair<int, int>& x, const std::pair<int, int>& y) {
        if (x.first != y.first) return x.first > y.first;
        return items[x.second].n > items[y.second].n;
    });
    std::vector<TriTask> tasks;
    size_t smem16 = 0, smem8 = 0;
    int n16 = 0;
    for (const auto& o : order) {
        const TriItem& it = items[o.second];
        const size_t need = kPlanBytes[o.first];
        (kPlanCL[o.first] == 16 ? smem16 : smem8) = std::max(kPlanCL[o.first] == 16 ? smem16 : smem8, need);
        for (int r = 0; r < kPlanCL[o.first]; ++r)
            tasks.push_back(TriTask{it.A, it.D, it.E, it.TAU, it.n, it.lda, o.first, r});
        if (kPlanCL[o.first] == 16) n16 = (int)tasks.size();
    }
    int n8 = (int)tasks.size() - n16;
    for (; n8 % 8; ++n8) tasks.push_back(TriTask{nullptr, nullptr, nullptr, nullptr, 0, 0, -1, 0});
    NRG_TRY(buf.ensure(sizeof(TriTask) * tasks.size()));
    NRG_TRY(h2d_async(ctx, buf.p, tasks.data(), sizeof(TriTask) * tasks.size()));
    const TriTask* d = buf.as<TriTask>();
    int* status = ctx->d_status.as<int>();
    if (n16) NRG_TRY(launch_clusters<16>(ctx, d, n16, smem16, status));
    if (n8) NRG_TRY(launch_clusters<8>(ctx, d + n16, n8, smem8, status));
    return NRG_OK;
}

}  // namespace nrg

int launch_tri_small(const SyevSector* d_secs, int nsec, double* eigbuf, double* wsd, int* d_status,
                     cudaStream_t st) {
    k_tri_small<<<nsec, kTriThreads, Plan0::kBytes, st>>>(d_secs, eigbuf, wsd, d_status);
    NRG_CUDA_TRY(cudaGetLastError());
    return NRG_OK;
}
