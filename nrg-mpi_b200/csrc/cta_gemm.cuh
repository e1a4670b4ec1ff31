// FP64 tensor-core MMA (mma.sync m8n8k4 f64) for the products inside the eigensolver's blocks.
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

}  // namespace nrg
