// Warp-level FP64 matrix product (mma.sync m8n8k4).
#pragma once

#include <cstddef>
#include <cstdint>

namespace hb {

// c += A B for one 8 x 8 tile and 4 k: lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and C[l / 4][2 (l % 4)], C[l / 4][2 (l % 4) + 1].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// acc += A B over `steps` steps of 8 k, MT tiles of 8 rows by RN tiles of 8
// columns.  A in fragment order, [step][MT][32] double2, `ap` at this lane's
// entry of the first step: lane (g, t) = (l / 4, l % 4) holds row 8 m + g,
// columns 8 s + 2 t and 8 s + 2 t + 1 (the k of a step's two MMAs is permuted
// so that both values of a lane are adjacent in A and in B).  B in shared
// memory, [column][ldz] with k contiguous, `zp` at column g and k = 2 t of the
// first step.  A row tile's fragment of the next step is requested as soon as
// its last product of this step is issued.
template <int MT, int RN, int LDZ, int UNROLL = 1>
__device__ __forceinline__ void dmma_steps(double (&acc)[MT][RN][2], const double2* __restrict__ ap,
                                           const double* zp, int steps) {
  if (steps <= 0) return;
  double2 af[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) af[m] = __ldg(ap + m * 32);
#pragma unroll UNROLL
  for (int s = 0; s < steps; ++s) {
    double2 b[RN];
#pragma unroll
    for (int c = 0; c < RN; ++c) b[c] = *reinterpret_cast<const double2*>(zp + c * 8 * LDZ);
    ap += s + 1 < steps ? MT * 32 : 0;   // the last step reloads its own
    zp += 8;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int c = 0; c < RN; ++c) dmma(acc[m][c], af[m].x, b[c].x);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
#pragma unroll
      for (int c = 0; c < RN; ++c) dmma(acc[m][c], af[m].y, b[c].y);
      af[m] = __ldg(ap + m * 32);
    }
  }
}

// Entry of row i, column k of an operator with mt row tiles in that order.
__host__ __device__ constexpr size_t dmma_afrag(int i, int k, int mt) {
  return (((size_t)(k / 8) * mt + i / 8) * 32 + (i % 8) * 4 + (k % 8) / 2) * 2 + (k & 1);
}

__device__ __forceinline__ void cp_async8(void* smem, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(smem)),
               "l"(g)
               : "memory");
}
template <typename T>
__device__ __forceinline__ void cp_async_word(T* smem, const T* g) {
  if constexpr (sizeof(T) == 8)
    cp_async8(smem, g);
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(smem)),
                 "l"(g)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Elements per batch of a launch over n elements: EB, evened out over whole
// rounds of the grid; on a mesh smaller than one round fewer, down to one tile
// of 8 columns, so that every SM has work (684 triangles of N = 3: 228 CTAs
// and 4.2 us a stage, where batches of 25 made 28 CTAs and 8.3 us)
inline int dmma_batch(int64_t n, int eb, int columns, int64_t slots) {
  const int64_t rounds = (n + eb * slots - 1) / (eb * slots);
  const int64_t even = (n + rounds * slots - 1) / (rounds * slots);
  const int64_t least = (8 + columns - 1) / columns;
  return (int)(even < least ? (least < eb ? least : eb) : even < eb ? even : eb);
}

}  // namespace hb
