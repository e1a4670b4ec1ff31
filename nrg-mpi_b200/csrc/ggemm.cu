// Grouped FP64 GEMM with gathered operands: one launch runs every (sector pair, matrix
// type, local operation) product of a phase.  It replaces the per-pair dgemm calls of
// invariantMatrixDGEMM.F90:300,316, invariantMatrixForSpectrumDGEMM.F90:296,312,
// reducedDensityMatrixDGEMM.F90:280,296 and module.F90:1100,1113, without building the
// reference's dense coefficient matrices: rows of the eigenvector blocks are gathered
// through index lists instead.
//
//   C(i,j) = alpha * sum_k A(i,k) B(k,j) + beta * C(i,j)
//   A(i,k) = A[ri(i)*a_si + ki(k)*a_sk]          ri = a_ri ? a_ri[i] : i, ki likewise
//   B(k,j) = B[ki(k)*b_sk + ji(j)*b_sj]          ki = b_ki ? b_ki[k] : k, ji likewise
//   C(i,j) = C[ci(i)*c_si + cj(j)*c_sj]          ci = c_ri ? c_ri[i] : i, cj likewise
//
// A problem may be followed by further products of the same C (cont): they are summed in the
// accumulators of its tiles, one after another, and C is written once.
//
// FP64 tensor-core MMA (mma.sync m16n8k8 f64), k in slabs of 32 (16 on the larger tiles) that 8-byte
// asynchronous copies stage two ahead (every operand is only 8-byte aligned: odd leading dimensions, gathered
// rows).  Loads are coalesced along whichever index of each operand has unit stride, and a
// slab is laid out along that index.
// The tile shape of each launch is chosen by the context's tuner (GemmTuner below).
#include "cta_gemm.cuh"
#include "internal.hpp"

#include <algorithm>
#include <array>
#include <cstdlib>
#include <map>
#include <mutex>
#include <type_traits>

namespace nrg {
namespace {

// the 16 x 8 x 8 MMA on fragments held as [row half][k half]; 3-5% over twice m8n8k4 pairs
__device__ __forceinline__ void dmma16(double (&d)[2][2], const double (&a)[2][2], const double (&b)[2]) {
    nrg::cta_dmma16(d[0][0], d[0][1], d[1][0], d[1][1], make_double2(a[0][0], a[1][0]), make_double2(a[0][1], a[1][1]),
                    b[0], b[1]);
}

// (16 WM RM) x (8 WN RN) output tile of WM x WN warps with RM x RN MMA tiles each.  Every variant
// accumulates each output element over k in the same order (the k = 8 steps of the MMA), so all
// variants give bit-identical results and the tile choice is free to change between launches.
//
// What bounds it is the FP64 tensor rate (36 TFLOP/s): registers are kept to 128 so that two
// blocks of eight warps share an SM and one computes while the other waits for its slab.
// 64 products of 320 x 320 x 1310 run at 24.4 TFLOP/s on the 64 x 64 tile (slabs of 16: 20.4, of
// 32: 22.9, with the 16 x 8 x 8 MMA the rest), one of order 4096 at 28.3.  With the slabs staged
// through registers and 220-255 of them per thread, the products of a shell of N_keep = 4096
// ran at 8-11 TFLOP/s; 12-20 now, the sectors' ragged sizes taking the rest.
template <int WM_, int WN_, int RM_, int RN_, int TK_, int ST_, int BLK_>
struct Tile {
    static constexpr int WM = WM_, WN = WN_, RM = RM_, RN = RN_;
    static constexpr int TK = TK_, ST = ST_, BLK = BLK_;   // slab depth, slabs in shared memory, blocks per SM
    static constexpr int TM = 16 * WM * RM, TN = 8 * WN * RN, NT = 32 * WM * WN;
    static constexpr int LDK = TK + 4;   // leading dimension of a slab laid out along k
    static constexpr int SA = TM * LDK, SB = TN * LDK;
    static constexpr size_t smem_bytes() { return sizeof(double) * ST * (SA + SB); }
};

// One operand's slabs of TO rows (i of A, j of B) x TK.  A slab whose operand has unit stride
// along k is stored [row][k] with leading dimension TK + 4, otherwise [k][row] with TO + 4:
// both 4 mod 16 doubles, so that the copies (16 consecutive) and the MMA fragments (8 rows x 4 k)
// of a half warp fall on distinct bank pairs.
template <int TO, int TK, int NT>
struct Feed {
    static constexpr int E = TO * TK / NT;   // copies per thread and slab
    const double* base;
    const int* ki;
    long long sk, off[E];
    int K, k_of, idx[E];
    unsigned rows;   // copies whose row exists
    bool kf;
    __device__ __forceinline__ int row(int u) const {
        return kf ? (int)threadIdx.x / TK + u * (NT / TK) : (int)threadIdx.x % TO;
    }
    __device__ __forceinline__ int col(int u) const {
        return kf ? (int)threadIdx.x % TK : (int)threadIdx.x / TO + u * (NT / TO);
    }
    __device__ __forceinline__ void open(const double* p, long long so, long long sk_, const int* oi, const int* ki_,
                                         int o0, int extent, int K_) {
        base = p;
        ki = ki_;
        sk = sk_;
        K = K_;
        kf = sk_ == 1 && so != 1;
        rows = 0;
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int o = o0 + row(u);
            off[u] = 0;
            if (o < extent) {
                off[u] = (oi ? (long long)oi[o] : (long long)o) * so;
                rows |= 1u << u;
            }
            if (!kf) {   // one row per thread
                rows = o < extent ? ~0u : 0u;
                break;
            }
        }
        fetch_idx(0);
    }
    // the gathered k of the slab at k0, loaded one slab before it is used
    __device__ __forceinline__ void fetch_idx(int k0) {
        if (!ki) return;
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int k = k0 + col(u);
            idx[u] = k < K ? ki[k] : 0;
            if (kf) break;   // one k per thread
        }
    }
    __device__ __forceinline__ void issue(double* slab, int k0) {
        if (kf) {
            const int k = k0 + col(0);
            const long long ko = (ki ? idx[0] : k) * sk;
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const bool in = k < K && (rows >> u & 1u);
                nrg::cp_async8(slab + row(u) * (TK + 4) + col(u), in ? base + off[u] + ko : base, in ? 8 : 0);
            }
        } else {
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const int k = k0 + col(u);
                const bool in = k < K && rows;
                const long long ko = (ki ? idx[u] : k) * sk;
                nrg::cp_async8(slab + col(u) * (TO + 4) + row(u), in ? base + off[0] + ko : base, in ? 8 : 0);
            }
        }
        fetch_idx(k0 + TK);
    }
};

template <class T>
__global__ void __launch_bounds__(T::NT, T::BLK) k_ggemm(const GemmProblem* __restrict__ probs,
                                                    const int* __restrict__ tilePrefix, int nprob) {
    extern __shared__ double gsm[];
    const int bid = blockIdx.x;
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tilePrefix[mid] <= bid) lo = mid; else hi = mid - 1;
    }
    const GemmProblem& P = probs[lo];
    const int t = bid - tilePrefix[lo];
    const int tilesN = (P.N + T::TN - 1) / T::TN;
    const int i0 = (t / tilesN) * T::TM, j0 = (t % tilesN) * T::TN;
    const int M = P.M, N = P.dyn_n ? min(P.N, *P.dyn_n) : P.N;
    if (j0 >= N) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wi = (warp % T::WM) * 16 * T::RM, wj = (warp / T::WM) * 8 * T::RN;   // warp tile origin
    const int g = lane >> 2, q4 = lane & 3;
    // MMA tiles of the warp that hold any output: a tile at the edge leaves the tensor pipe to the
    // others (order 333 on 64 x 64: 27 tiles' work instead of 36)
    const int rl = min(T::RM, max(0, (M - i0 - wi + 15) / 16)), cl = min(T::RN, max(0, (N - j0 - wj + 7) / 8));
    double acc[T::RM][T::RN][2][2];
#pragma unroll
    for (int r = 0; r < T::RM; ++r)
#pragma unroll
        for (int c = 0; c < T::RN; ++c)
            acc[r][c][0][0] = acc[r][c][0][1] = acc[r][c][1][0] = acc[r][c][1][1] = 0.0;
    // the problem's slabs, then those of the problems added to it
    for (int x = lo; x == lo || (x < nprob && probs[x].cont); ++x) {
        const GemmProblem& Q = probs[x];
        Feed<T::TM, T::TK, T::NT> fa;
        Feed<T::TN, T::TK, T::NT> fb;
        fa.open(Q.A, Q.a_si, Q.a_sk, Q.a_ri, Q.a_ki, i0, M, Q.K);
        fb.open(Q.B, Q.b_sj, Q.b_sk, Q.b_ji, Q.b_ki, j0, N, Q.K);
        const int nslab = (Q.K + T::TK - 1) / T::TK;
        // strides of the fragments in a slab
        const int ai = fa.kf ? T::LDK : 1, ak = fa.kf ? 1 : T::TM + 4;
        const int bj = fb.kf ? T::LDK : 1, bk = fb.kf ? 1 : T::TN + 4;
        const int a_at = (wi + g) * ai + q4 * ak, b_at = (wj + g) * bj + q4 * bk;
#pragma unroll
        for (int s = 0; s < T::ST - 1; ++s) {
            if (s < nslab) {
                fa.issue(gsm + s * T::SA, s * T::TK);
                fb.issue(gsm + T::ST * T::SA + s * T::SB, s * T::TK);
            }
            nrg::cp_async_commit();
        }
        int cur = 0, ahead = T::ST - 1;
        for (int s = 0; s < nslab; ++s) {
            nrg::cp_async_wait<T::ST - 2>();
            __syncthreads();   // slab s has landed; every warp is through with slab s - 1
            if (s + T::ST - 1 < nslab) {
                fa.issue(gsm + ahead * T::SA, (s + T::ST - 1) * T::TK);
                fb.issue(gsm + T::ST * T::SA + ahead * T::SB, (s + T::ST - 1) * T::TK);
            }
            nrg::cp_async_commit();
            const double* as = gsm + cur * T::SA + a_at;
            const double* bs = gsm + T::ST * T::SA + cur * T::SB + b_at;
            auto multiply = [&](auto whole) {
#pragma unroll
                for (int ks = 0; ks < T::TK; ks += 8) {
                    double af[T::RM][2][2], bf[T::RN][2];
#pragma unroll
                    for (int r = 0; r < T::RM; ++r)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            af[r][h][0] = as[ks * ak + (16 * r + 8 * h) * ai];
                            af[r][h][1] = as[(ks + 4) * ak + (16 * r + 8 * h) * ai];
                        }
#pragma unroll
                    for (int c = 0; c < T::RN; ++c) {
                        bf[c][0] = bs[ks * bk + c * 8 * bj];
                        bf[c][1] = bs[(ks + 4) * bk + c * 8 * bj];
                    }
#pragma unroll
                    for (int r = 0; r < T::RM; ++r)
#pragma unroll
                        for (int c = 0; c < T::RN; ++c)
                            if (decltype(whole)::value || (r < rl && c < cl)) dmma16(acc[r][c], af[r], bf[c]);
                }
            };
            // (two copies of the loop are only worth their registers on the small warp tiles)
            if (T::RM * T::RN > 4 ? rl > 0 && cl > 0 : rl == T::RM && cl == T::RN) multiply(std::true_type());
            else if (T::RM * T::RN <= 4 && rl > 0 && cl > 0) multiply(std::false_type());
            ahead = cur;
            cur = cur + 1 == T::ST ? 0 : cur + 1;
        }
        nrg::cp_async_wait<0>();
        __syncthreads();   // the slabs may be overwritten
    }
#pragma unroll
    for (int r = 0; r < 2 * T::RM; ++r) {
        const int gi = i0 + wi + r * 8 + g;
        if (gi >= M) continue;
        const long long ci = P.c_ri ? P.c_ri[gi] : gi;
#pragma unroll
        for (int c = 0; c < T::RN; ++c) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gj = j0 + wj + c * 8 + 2 * q4 + h;
                if (gj >= N) continue;
                const long long cj = P.c_ji ? P.c_ji[gj] : gj;
                double* out = P.C + ci * P.c_si + cj * P.c_sj;
                const double v = P.alpha * acc[r / 2][c][r % 2][h];
                *out = (P.beta == 0.0) ? v : P.beta * *out + v;
            }
        }
    }
}

template <class T>
int launch_variant(nrg_context* ctx, const std::vector<GemmProblem>& live, DevBuf& buf) {
    const int np = (int)live.size();
    std::vector<int> prefix(np);
    long long total = 0;
    for (int i = 0; i < np; ++i) {
        prefix[i] = (int)total;   // an added product has no tiles of its own
        if (!live[i].cont) total += (long long)((live[i].M + T::TM - 1) / T::TM) * ((live[i].N + T::TN - 1) / T::TN);
    }
    if (total > 0x7fffffffLL) return NRG_ERR_TOO_LARGE;
    const GemmProblem* dp = nullptr;
    const int* dq = nullptr;
    NRG_TRY(h2d_pair(ctx, buf, live, prefix, &dp, &dq));
    NRG_TRY(raise_smem_limit((const void*)k_ggemm<T>, T::smem_bytes()));
    k_ggemm<T><<<(unsigned)total, T::NT, T::smem_bytes(), ctx->stream>>>(dp, dq, np);
    ctx->launches++;
    NRG_CUDA_TRY(cudaGetLastError());
    return NRG_OK;
}

// the tile variants, in the order of GemmTuner's slots: 64 x 64, 32 x 32, 128 x 64, 64 x 128
using Tile0 = Tile<2, 4, 2, 2, 32, 3, 2>;
using Tile1 = Tile<2, 2, 1, 2, 32, 3, 4>;
using Tile2 = Tile<4, 2, 2, 4, 16, 3, 2>;
using Tile3 = Tile<2, 4, 2, 4, 16, 3, 2>;

int log2_bucket(long long v) {
    int b = 0;
    while (v > 1 && b < 15) { v >>= 1; ++b; }
    return b;
}

}  // namespace

// Online tuning of the tile shape, per device.  Launches are keyed by their problem mix
// (log2 buckets of the median M, N, K and of the problem count); the first launches of a
// key try each tile variant in turn, timed by events on the launching stream, and later
// launches of the key take the variant with the least time per flop.  Timings are read without
// waiting: a pending measurement is collected by a later launch once its events have
// completed.  The variants give bit-identical results, so the choice never changes a
// result.  NRG_GGEMM_VARIANT=0..3 fixes one variant (no tuning).
int GemmTuner::pick(unsigned key) {
    static const int forced = [] {
        const char* e = getenv("NRG_GGEMM_VARIANT");
        if (!e || !*e) return -1;
        const int v = atoi(e);
        return (v >= 0 && v < kTunedVariants) ? v : -1;
    }();
    if (forced >= 0) return forced;
    Entry& e = table[key];
    for (int v = 0; v < kTunedVariants; ++v)
        if (e.samples[v] < kSamples && e.inflight[v] == 0) return v;
    int best = 0;
    for (int v = 1; v < kTunedVariants; ++v)
        if (e.samples[v] > 0 && (e.samples[best] == 0 || e.ms_per_gflop[v] < e.ms_per_gflop[best])) best = v;
    return best;
}

void GemmTuner::collect(bool wait) {
    for (size_t i = 0; i < pending.size();) {
        Pending& q = pending[i];
        cudaError_t st = wait ? cudaEventSynchronize(q.b) : cudaEventQuery(q.b);
        if (st == cudaErrorNotReady) { ++i; continue; }
        float ms = 0.0f;
        if (st == cudaSuccess && cudaEventElapsedTime(&ms, q.a, q.b) == cudaSuccess && q.gflop > 0.0) {
            Entry& e = table[q.key];
            const double r = ms / q.gflop;
            e.ms_per_gflop[q.variant] = e.samples[q.variant] == 0 ? r : std::min(e.ms_per_gflop[q.variant], r);
            e.samples[q.variant]++;
            e.inflight[q.variant]--;
        } else {
            cudaGetLastError();
            table[q.key].inflight[q.variant]--;
        }
        free_events.push_back(q.a);
        free_events.push_back(q.b);
        pending[i] = pending.back();
        pending.pop_back();
    }
}

// one tuner per device, shared by every context on it (independent instances side by side
// tune once between them); its state is guarded by its mutex
GemmTuner& tuner_for(int dev) {
    static std::mutex mu;
    static std::map<int, GemmTuner*> tuners;
    std::lock_guard<std::mutex> lk(mu);
    GemmTuner*& t = tuners[dev];
    if (!t) t = new GemmTuner();   // lives until the process exits
    return *t;
}

int launch_ggemm(nrg_context* ctx, std::vector<GemmProblem>& probs, int scratch_slot) {
    std::vector<GemmProblem> live;
    live.reserve(probs.size());
    // empty problems dropped, the others by decreasing length of their sums (a tile's time), those added to a product
    // behind it: a long tile that starts last runs alone
    std::vector<std::array<long long, 3>> sums;   // -K in total, first problem, end
    for (size_t x = 0; x < probs.size(); ++x) {
        if (!probs[x].cont || sums.empty()) sums.push_back({0, (long long)x, 0});
        if (probs[x].M > 0 && probs[x].N > 0 && probs[x].K > 0) sums.back()[0] -= probs[x].K;
        sums.back()[2] = (long long)x + 1;
    }
    std::stable_sort(sums.begin(), sums.end(), [](const auto& a, const auto& b) { return a[0] < b[0]; });
    for (const auto& q : sums) {
        bool added = false;
        for (long long x = q[1]; x < q[2]; ++x) {
            const GemmProblem& p = probs[x];
            if (p.M <= 0 || p.N <= 0 || p.K <= 0) continue;
            live.push_back(p);
            live.back().cont = added;
            added = true;
        }
    }
    const int np = (int)live.size();
    if (np == 0) return NRG_OK;
    // problem-mix key and algorithmic flops
    std::vector<int> ms(np), ns(np), ks(np);
    double gflop = 0.0;
    for (int i = 0; i < np; ++i) {
        ms[i] = live[i].M;
        ns[i] = live[i].N;
        ks[i] = live[i].K;
        gflop += 2e-9 * live[i].M * (double)live[i].N * live[i].K;
    }
    auto med = [](std::vector<int>& v) {
        std::nth_element(v.begin(), v.begin() + v.size() / 2, v.end());
        return (long long)v[v.size() / 2];
    };
    const unsigned key = (unsigned)(log2_bucket(med(ms)) | log2_bucket(med(ns)) << 4 | log2_bucket(med(ks)) << 8 |
                                    log2_bucket(np) << 12);
    int dev = 0;
    NRG_CUDA_TRY(cudaGetDevice(&dev));
    GemmTuner& tu = tuner_for(dev);
    std::unique_lock<std::mutex> lk(tu.mu);
    tu.collect(false);
    const int v = tu.pick(key);
    DevBuf& buf = ctx->scratch.b[scratch_slot];
    const bool timed = tu.table[key].samples[v] < GemmTuner::kSamples && tu.table[key].inflight[v] == 0;
    cudaEvent_t ea = nullptr, eb = nullptr;
    if (timed) {
        NRG_TRY(tu.event(&ea));
        NRG_TRY(tu.event(&eb));
        tu.table[key].inflight[v]++;   // claimed before the lock is released
    }
    lk.unlock();
    if (timed) NRG_CUDA_TRY(cudaEventRecord(ea, ctx->stream));
    int rc = NRG_OK;
    switch (v) {
        case 0: rc = launch_variant<Tile0>(ctx, live, buf); break;
        case 1: rc = launch_variant<Tile1>(ctx, live, buf); break;
        case 2: rc = launch_variant<Tile2>(ctx, live, buf); break;
        default: rc = launch_variant<Tile3>(ctx, live, buf); break;
    }
    if (timed) {
        const bool rec = rc == NRG_OK && cudaEventRecord(eb, ctx->stream) == cudaSuccess;
        lk.lock();
        if (rec) {
            tu.pending.push_back({key, v, ea, eb, gflop});
        } else {
            tu.table[key].inflight[v]--;
            tu.free_events.push_back(ea);
            tu.free_events.push_back(eb);
        }
    }
    return rc;
}

int GemmTuner::event(cudaEvent_t* e) {
    if (!free_events.empty()) {
        *e = free_events.back();
        free_events.pop_back();
        return NRG_OK;
    }
    NRG_CUDA_TRY(cudaEventCreate(e));
    return NRG_OK;
}

}  // namespace nrg
