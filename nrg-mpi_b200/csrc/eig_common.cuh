// Device building blocks of the FP64 symmetric eigensolver: block reductions and the vectors
// of the divide-and-conquer merges that are spread over the whole device (eig_large.cu).
#pragma once
#include "common.cuh"
#include "cta_gemm.cuh"

#include <math.h>

namespace {

constexpr double kEps = 1.1102230246251565e-16;

__device__ double block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    const int nw = blockDim.x >> 5;
    for (int i = 0; i < nw; ++i) s += red[i];   // same order in every thread
    return s;
}
__device__ double block_max(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    const int nw = blockDim.x >> 5;
    for (int i = 0; i < nw; ++i) s = fmax(s, red[i]);
    return s;
}

// v, or zero with the status flag set where v is not finite.  Every diagonal entry and merged
// value of the divide and conquer passes here: ranks among them are used as indexes, and with a
// NaN (a norm that overflowed in the reduction, a wait that ran out) two entries would share a
// rank and leave another unwritten.
__device__ __forceinline__ double finite_value(double v, int* status) {
    if (isfinite(v)) return v;
    atomicOr(status, NRG_DEV_NONFINITE);
    return 0.0;
}

// scratch arrays of one sector, each of length n, indexed by absolute row
struct Scratch {
    double *z, *ds, *zs, *dd, *zz, *tau, *zh, *vals, *rc, *rs;
    int *perm, *nd, *df, *org, *pos, *ra, *rb, *mk, *mr, *mf;
};

__device__ Scratch scratch_at(double* vec, int* I, int n) {
    // vec: D, E, TAU, then the merge arrays; I: the integer arrays
    Scratch S;
    S.z = vec + 3 * n; S.ds = vec + 4 * n; S.zs = vec + 5 * n; S.dd = vec + 6 * n;
    S.zz = vec + 7 * n; S.tau = vec + 8 * n; S.zh = vec + 9 * n; S.vals = vec + 10 * n;
    S.rc = vec + 11 * n; S.rs = vec + 12 * n;
    S.perm = I; S.nd = I + n; S.df = I + 2 * n; S.org = I + 3 * n; S.pos = I + 4 * n;
    S.ra = I + 5 * n; S.rb = I + 6 * n; S.mk = I + 7 * n; S.mr = I + 8 * n; S.mf = I + 9 * n;
    return S;
}

}  // namespace
