// nrg_block_eigh_noalloc: the per-sector FP64 eigensolvers (eig.cu, eig_panel.cu) for one
// symmetric block, for callers that cannot allocate device memory.  Its workspace lives in
// the file-scope device array below (allocated when the library is loaded on a device and
// held until the process exits); the call itself allocates nothing.
#include "common.cuh"

#include <cuda.h>   // CUcontext and CUresult only: driver calls go through cudaGetDriverEntryPoint

#include <mutex>

namespace {

// largest block order the static workspace covers
constexpr long long kMaxN = NRG_NOALLOC_MAX_ORDER;
constexpr int kPanelOnly = 5;   // see the call
// [0, 8): sector descriptor, [8, 16): status word and the mark of a close decision, then the
// workspace
constexpr long long kDescOff = 0, kStatusOff = 8, kDblOff = 16;
constexpr long long kTotalDoubles = kDblOff + syev_ws_doubles(kMaxN);
static_assert(sizeof(SyevSector) <= 8 * sizeof(double), "descriptor slot too small");

}  // namespace

// the workspace: one copy per device that loads the library (~396 KB), kept until exit
static __device__ __align__(256) double g_noalloc_scratch[kTotalDoubles];

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_mu;

// The array's device address, looked up once per device and CUDA context.  The address
// belongs to the context the library's device code was loaded into: after the application
// resets the device (cudaDeviceReset) a new primary context loads the module again, and
// the old address is stale.  The context is told apart by its process-unique id
// (cuCtxGetId, through the runtime's driver entry points: no link against libcuda).
struct ScratchEntry {
    unsigned long long ctx_id;   // 0: unknown, look up again on the next call
    double* ptr;
};
ScratchEntry g_scratch[kMaxDevices] = {};

typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long*);

// id of the calling thread's current context; 0 when there is none or it cannot be told
unsigned long long current_context_id() {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static bool resolved = false;
    if (!resolved) {   // under g_mu
        resolved = true;
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<CtxGetCurrentFn>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<CtxGetIdFn>(f);
        cudaGetLastError();
    }
    if (!get_current || !get_id) return 0;
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (get_current(&c) != CUDA_SUCCESS || !c || get_id(c, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// device address of the static array on the current device
int scratch_address(int device, double** out) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (device < 0 || device >= kMaxDevices) return NRG_ERR_DEVICE;
    ScratchEntry& e = g_scratch[device];
    unsigned long long id = current_context_id();
    if (e.ptr && id != 0 && id == e.ctx_id) {
        *out = e.ptr;
        return NRG_OK;
    }
    void* p = nullptr;
    const cudaError_t err = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (err != cudaSuccess) {
        nrg_set_error_message("cudaGetSymbolAddress of the static workspace failed: %s", cudaGetErrorString(err));
        return NRG_ERR_CUDA;
    }
    if (id == 0) id = current_context_id();   // the lookup made the primary context current
    e.ptr = static_cast<double*>(p);
    e.ctx_id = id;
    *out = e.ptr;
    return NRG_OK;
}

// memory this device's kernels may read and write: device memory of the current device,
// or managed memory; a device pointer of another GPU is refused (no peer access is set up)
bool on_device(const void* p, int device) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type == cudaMemoryTypeManaged) return true;
    return a.type == cudaMemoryTypeDevice && a.device == device;
}

}  // namespace

extern "C" int nrg_block_eigh_noalloc(const double* H, int32_t n, double* eigenvalues,
                                      double* eigenvectors, void* stream) {
    if (n < 1 || n > kMaxN) {
        nrg_set_error_message("nrg_block_eigh_noalloc: order %d outside 1..%lld (the static workspace limit)",
                              n, kMaxN);
        return NRG_ERR_TOO_LARGE;
    }
    int device = 0;
    NRG_CUDA_TRY(cudaGetDevice(&device));
    if (!H || !eigenvalues || !eigenvectors || !on_device(H, device) || !on_device(eigenvalues, device) ||
        !on_device(eigenvectors, device)) {
        nrg_set_error_message("nrg_block_eigh_noalloc: H, eigenvalues and eigenvectors must be device arrays "
                              "of the current device (%d) or managed memory", device);
        return NRG_ERR_INVALID;
    }
    double* base = nullptr;
    NRG_TRY(scratch_address(device, &base));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    SyevSector sec;
    sec.a_off = 0;
    sec.w_off = 0;
    sec.e_off = 0;
    sec.n = n;
    sec.pad = 0;
    SyevSector* d_sec = reinterpret_cast<SyevSector*>(base + kDescOff);
    int* d_status = reinterpret_cast<int*>(base + kStatusOff);
    int* d_unsure = d_status + 1;
    double* d_ws = base + kDblOff;
    // the workspace keeps the previous call's contents: the status word must start at zero;
    // the eigensolver writes every other workspace entry before reading it
    NRG_CUDA_TRY(cudaMemsetAsync(d_status, 0, sizeof(int), st));
    NRG_CUDA_TRY(cudaMemcpyAsync(d_sec, &sec, sizeof(sec), cudaMemcpyHostToDevice, st));
    if (eigenvectors != H)
        NRG_CUDA_TRY(cudaMemcpyAsync(eigenvectors, H, sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToDevice, st));
    // Up to order 5 the panel solver alone, one launch instead of three: order 2 takes 51 us for 56,
    // 3 64 for 61, 4 64 for 68, 5 76 for 81, 6 80..88 for 81, 8 89 for 81.  Above it the fast solver,
    // and where that decides so close to a tolerance that a column's sign hangs on its last bits the
    // panel solver, whose signs stay what they are (eig_panel.cu).  Order 128: 0.45 ms, 1.9 ms for
    // the 10% that are solved twice; the panel solver alone takes 1.5.
    if (n <= kPanelOnly) {
        NRG_TRY(launch_syev_panel(d_sec, 1, eigenvectors, eigenvalues, d_ws, nullptr, nullptr, d_status, st));
    } else {
        // the block, for the panel solver, where the results are written over it
        const bool over = eigenvectors == H || (eigenvalues < H + (size_t)n * n && H < eigenvalues + n);
        double* kept = d_ws + (long long)n * n;   // where only the panel solver works
        if (over)
            NRG_CUDA_TRY(cudaMemcpyAsync(kept, H, sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToDevice, st));
        NRG_TRY(launch_syev(d_sec, 1, eigenvectors, eigenvalues, d_ws, d_unsure, d_status, st));
        NRG_TRY(launch_syev_panel(d_sec, 1, eigenvectors, eigenvalues, d_ws, d_unsure, over ? kept : H, d_status, st));
    }
    int flags = 0;
    NRG_CUDA_TRY(cudaMemcpyAsync(&flags, d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
    NRG_CUDA_TRY(cudaStreamSynchronize(st));
    if (flags != 0) {
        nrg_set_error_message("nrg_block_eigh_noalloc: device status flags 0x%x", flags);
        return device_status_code(flags);
    }
    return NRG_OK;
}
