// One large sector (order > 128) of the eigensolver: its descriptor, its workspace and the
// views of it that the kernels of eig_large.cu and eig_panel.cu share.
#pragma once
#include "eig_common.cuh"

namespace nrg {

struct LSec {
    long long a_off, e_off, w_off, i_off;
    int n;
    int z_sel;   // where the divide and conquer leaves the eigenvectors: 0 Z, 2 Qt (in n x n)
};

}  // namespace nrg

namespace {

using nrg::LSec;

constexpr int NB = 32;        // tridiagonalisation panel
constexpr int NBB = 64;       // back-transformation panel
constexpr int DC_LOW = 128;   // merges of up to this many rows run inside one block
constexpr int TPB = 256;
constexpr int CB = 32;        // columns per block in the symmetric matrix-vector product

// workspace per sector: Z, U, Qt (n x n each), the panel V | W (n x 2 NB), y, the D&C
// vectors (16 n + 64), then the back-transformation's T factors and explicit reflector
// panels ((n + NBB)^2 bounds both)
long long lws_doubles(long long n) {
    return 3 * n * n + 2LL * NB * n + n + 16 * n + 64 + (n + NBB) * (n + NBB);
}
long long lws_ints(long long n) { return 12 * n + 64; }

struct LView {
    double *A, *Z, *U, *Qt, *ZV, *VW, *y, *vec, *D, *E, *TAU, *R;   // ZV: the eigenvectors of T
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
    v.ZV = W + s.z_sel * sq;
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

}  // namespace
