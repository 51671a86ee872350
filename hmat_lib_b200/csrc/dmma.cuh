// One FP64 tensor-core product: C (8 x 8) += A (8 x 4) B (4 x 8) by a warp.
// Lane l holds A[l / 4][l % 4], B[l % 4][l / 4] and C[l / 4][2 (l % 4) + {0, 1}].
#pragma once

namespace hb {

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

}  // namespace hb
