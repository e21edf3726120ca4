// FP64 matrix instruction: c (8 x 8) += a (8 x 4) b (4 x 8) over a warp.
#pragma once

namespace plx {
namespace {

// Lane l holds a[l / 4][l % 4], b[l % 4][l / 4] and c[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

}  // namespace
}  // namespace plx
