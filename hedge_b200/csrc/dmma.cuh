// Warp-level FP64 matrix product (mma.sync m8n8k4).
#pragma once

namespace hb {

// c += A B for one 8 x 8 tile and 4 k: lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and C[l / 4][2 (l % 4)], C[l / 4][2 (l % 4) + 1].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

}  // namespace hb
