// FP64 tensor-core MMA (mma.sync m8n8k4 f64) and 8-byte asynchronous copies for the products in
// shared memory.
#pragma once
#include <cuda_runtime.h>

namespace nrg {

// d (8 x 8) += a (8 x 4) b (4 x 8): lane l holds a(l / 4, l % 4), b(l % 4, l / 4) and
// d(l / 4, 2 (l % 4) + {0, 1})
__device__ __forceinline__ void cta_dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// d (16 x 8) += a (16 x 8) b (8 x 8): lane l holds a(l / 4 + {0, 8}, l % 4) in lo, a(l / 4 + {0, 8},
// l % 4 + 4) in hi, b(l % 4 + {0, 4}, l / 4), and d(l / 4, 2 (l % 4) + {0, 1}), then d(l / 4 + 8, ...)
__device__ __forceinline__ void cta_dmma16(double& d0, double& d1, double& d2, double& d3, double2 lo, double2 hi,
                                           double b0, double b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};\n"
        : "+d"(d0), "+d"(d1), "+d"(d2), "+d"(d3)
        : "d"(lo.x), "d"(lo.y), "d"(hi.x), "d"(hi.y), "d"(b0), "d"(b1));
}

// 8-byte asynchronous global-to-shared copies (zero-filled when bytes is 0)
__device__ __forceinline__ void cp_async8(double* dst, const double* src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

}  // namespace nrg
