// Shared definitions for the NRG hot-path kernels (sm_100a, FP64).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <cstdio>

#include "../../include/nrg_b200.h"

#define NRG_CUDA_TRY(expr)                                                        \
    do {                                                                          \
        cudaError_t _e = (expr);                                                  \
        if (_e != cudaSuccess) {                                                  \
            nrg_set_error_message("%s:%d %s -> %s", __FILE__, __LINE__, #expr,    \
                                  cudaGetErrorString(_e));                        \
            return NRG_ERR_CUDA;                                                  \
        }                                                                         \
    } while (0)

#define NRG_TRY(expr)                       \
    do {                                    \
        int _s = (expr);                    \
        if (_s != NRG_OK) return _s;        \
    } while (0)

void nrg_set_error_message(const char* fmt, ...);

// device status flags written by kernels (bit set; read back by the host)
enum : int {
    NRG_DEV_OK = 0,
    NRG_DEV_BAD_INDEX = 1,       // a gathered index fell outside its array
    NRG_DEV_SMEM = 2,            // a block did not fit the configured shared memory
    NRG_DEV_SECULAR = 4,         // a secular root did not bracket
    NRG_DEV_NONFINITE = 8,       // NaN/Inf met in an input block
    NRG_DEV_TIMEOUT = 16,        // a bounded wait between blocks expired
};

// the status a call returns for these flags.  A wait that ran out comes first: what else is set
// may be its consequence.
inline int device_status_code(int flags) {
    if (flags == NRG_DEV_OK) return NRG_OK;
    if (flags & NRG_DEV_TIMEOUT) return NRG_ERR_TIMEOUT;
    return (flags & (NRG_DEV_SECULAR | NRG_DEV_NONFINITE)) ? NRG_ERR_NUMERIC : NRG_ERR_INVALID;
}

// --------------------------------------------------------------------------------------
// eigensolver work description (one entry per symmetry sector)
// --------------------------------------------------------------------------------------
struct SyevSector {
    long long a_off;    // offset of the d x d block in the eigenvector buffer
    long long w_off;    // offset of the double workspace
    long long e_off;    // offset of the eigenvalues (start_input - 1)
    int n;
    int pad;
};

// workspace of a sector of order n <= 128, in doubles: the eigenvectors of T, two more n x n
// arrays for the panel solver's merges, then D | E | tau (n each)
__host__ __device__ constexpr long long syev_vec_off(long long n) { return 3 * n * n; }
__host__ __device__ constexpr long long syev_ws_doubles(long long n) { return syev_vec_off(n) + 3 * n; }

// launch helpers implemented in the .cu files (return NRG status)
int launch_tri_small(const SyevSector* d_secs, int nsec, double* eigbuf, double* wsd, int* d_status, cudaStream_t st);
// orders <= 128, one block each.  unsure (one sector; may be null): set to 1 where the signs or
// the mixing of eigenvectors hang on the last bits, otherwise to 0.  launch_syev_panel
// (eig_panel.cu) given it solves the sector only where it is set, from the block at `from`
// (n x n, not overwritten here; null: in eigbuf as usual).
int launch_syev(const SyevSector* d_secs, int nsec, double* eigbuf, double* evals, double* wsd, int* unsure, int* d_status, cudaStream_t st);
int launch_syev_panel(const SyevSector* d_secs, int nsec, double* eigbuf, double* evals, double* wsd, const int* unsure,
                      const double* from, int* d_status, cudaStream_t st);
