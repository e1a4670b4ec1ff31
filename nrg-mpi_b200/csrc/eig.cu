// Batched FP64 symmetric eigensolver for the symmetry-sector blocks of one NRG
// iteration (the dsyev('V','U') call of diagonalization.F90:267, one call per sector),
// one thread block per sector.  Used for blocks of order <= 128 of the runs that keep their
// eigenvectors on the device, and for nrg_block_eigh_noalloc (large blocks go through
// the multi-kernel pipeline of eig_large.cu, which reuses the pieces below; the eigenvectors
// that nrg_diagonalization returns come from eig_panel.cu):
//   1. Householder tridiagonalisation (H = Q T Q^T) by a launch of its own with the block in
//      registers (eig_tri.cu), reflectors kept in the block's own storage;
//   2. divide and conquer on T (eig_dc.cuh: Cuppen tearing down to 1x1 leaves, deflation of
//      small z components and of close pole pairs by Givens rotations, secular roots by a
//      safeguarded rational iteration in pole-shifted coordinates, Gu-Eisenstat
//      recomputation of z for orthogonal eigenvectors);
//   3. back-transformation V = Q Z with 32 reflectors at a time (compact WY form), the
//      columns of Z in registers.
// Eigenvalues come out ascending with their eigenvectors in the same column order, as
// dsyev returns them.
#include "eig_back.cuh"
#include "eig_dc.cuh"
#include "internal.hpp"

namespace {

constexpr int kThreads = kLeafThreads;
static_assert(kBtSmem <= kLeafSmem, "the back-transformation reuses the divide and conquer's shared memory");
static_assert(kThreads == kBtThreads, "the back-transformation's block");

template <bool MARK>
__global__ void __launch_bounds__(kThreads) k_syev(const SyevSector* __restrict__ secs,
                                                    double* __restrict__ eigbuf,
                                                    double* __restrict__ evals,
                                                    double* __restrict__ wsd, int* unsure, int* status) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int maybe;
    const SyevSector sec = secs[blockIdx.x];
    const int n = sec.n;
    const int tid = threadIdx.x, T = blockDim.x;
    double* A = eigbuf + sec.a_off;
    double* ev = evals + sec.e_off;
    {
        // a block holding NaN or Inf is reported and left undiagonalised (its eigenvalues
        // become NaN): the iterations below have fixed bounds, but their results would
        // be meaningless
        bool bad = false;
        for (long long e = tid; e < (long long)n * n; e += T) bad |= !isfinite(A[e]);
        if (__syncthreads_or(bad)) {
            if (tid == 0) atomicOr(status, NRG_DEV_NONFINITE);
            for (int i = tid; i < n; i += T) ev[i] = __longlong_as_double(0x7ff8000000000000LL);
            if (MARK && tid == 0) *unsure = 0;
            return;
        }
    }
    if (n == 1) {
        if (tid == 0) { ev[0] = A[0]; A[0] = 1.0; if (MARK) *unsure = 0; }
        return;
    }
    double* W = wsd + sec.w_off;
    double* Z = W;
    double* vec = W + syev_vec_off(n);
    double* Dd = vec;
    double* Ee = vec + n;
    double* TAU = vec + 2 * n;

    // ---- 2. divide and conquer on (Dd, Ee) -> eigenvalues in Dd, vectors in Z ----
    if (tid == 0) maybe = 0;
    dc_leaf<MARK>(0, n, n, Dd, Ee, Z, sm, status, &maybe);   // (a barrier before its first merge)
    __syncthreads();
    if (MARK) {
        const double gap = kUnsureGap * fmax(fabs(Dd[0]), fabs(Dd[n - 1]));
        for (int i = tid; i < n - 1; i += T)
            if (Dd[i + 1] - Dd[i] <= gap) maybe = 1;
    }

    // ---- 3. back-transformation, straight to the output ----
    back_transform(A, n, TAU, Z, sm);
    for (int i = tid; i < n; i += T) ev[i] = Dd[i];
    if (MARK && tid == 0) *unsure = maybe;   // (back_transform has barriers before this)
}

}  // namespace

int launch_syev(const SyevSector* d_secs, int nsec, double* eigbuf, double* evals, double* wsd, int* unsure, int* d_status, cudaStream_t st) {
    if (nsec == 0) return NRG_OK;
    NRG_TRY(launch_tri_small(d_secs, nsec, eigbuf, wsd, d_status, st));
    auto kernel = unsure ? k_syev<true> : k_syev<false>;
    NRG_TRY(nrg::raise_smem_limit((const void*)kernel, kLeafSmem));
    kernel<<<nsec, kThreads, kLeafSmem, st>>>(d_secs, eigbuf, evals, wsd, unsure, d_status);
    NRG_CUDA_TRY(cudaGetLastError());
    return NRG_OK;
}
