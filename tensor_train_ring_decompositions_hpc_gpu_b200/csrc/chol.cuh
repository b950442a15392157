// Cholesky factor of a small symmetric matrix in shared memory, by one block.
#pragma once
#include <math.h>

namespace ttr {

constexpr int CQ_P = 8;  // panel width

// Packed upper triangle by rows: element (k, j), j >= k, at cq_row(k, N) + j.
__device__ __forceinline__ int cq_row(int k, int N) { return k * N - ((k * (k - 1)) >> 1) - k; }

// R of W = R^T R over W (packed upper triangle), by the whole block.  A pivot at or below rel_tol * max
// diag marks a dependent column: its row of R is zero and so is inv[k], the reciprocal of R's
// diagonal.  pan: cq_pan(N) doubles.  Ends with a block barrier.
constexpr int cq_pstride(int N) { return (N + 4) & ~1; }  // the last four-row group reads past N
constexpr int cq_pan(int N) { return CQ_P * cq_pstride(N); }
__device__ inline void chol_panels(double* W, int N, double rel_tol, double* inv, double* pan) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  const int PS = cq_pstride(N);
  double dmax = 0.0;
  for (int i = lane; i < N; i += 32) dmax = fmax(dmax, W[cq_row(i, N) + i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
  const double tol = rel_tol * dmax;
  for (int k0 = 0; k0 < N; k0 += CQ_P) {
    const int j = k0 + tid;                   // this thread's column of the panel
    const bool active = k0 + 32 * warp < N;  // warps without one go straight to the barriers
    double D[CQ_P][CQ_P], v[CQ_P];
    if (active) {
#pragma unroll
      for (int i = 0; i < CQ_P; ++i) {
        const double* row = W + cq_row(min(k0 + i, N - 1), N);
#pragma unroll
        for (int c = i; c < CQ_P; ++c) D[i][c] = k0 + c < N ? row[k0 + c] : 0.0;
        v[i] = (j < N && j >= k0 + i) ? row[j] : 0.0;
      }
    }
    __syncthreads();  // the panel is read
    if (active) {
#pragma unroll
      for (int i = 0; i < CQ_P; ++i) {
        const double d = D[i][i];
        const double rs = (d > tol && dmax > 0.0) ? rsqrt(d) : 0.0;
#pragma unroll
        for (int c = i + 1; c < CQ_P; ++c) D[i][c] *= rs;
#pragma unroll
        for (int p = i + 1; p < CQ_P; ++p)
#pragma unroll
          for (int c = p; c < CQ_P; ++c) D[p][c] = fma(-D[i][p], D[i][c], D[p][c]);
        v[i] *= rs;
#pragma unroll
        for (int p = i + 1; p < CQ_P; ++p) v[p] = fma(-D[i][p], v[i], v[p]);
        if (tid == 0 && k0 + i < N) inv[k0 + i] = rs;
      }
      if (j < N) {
#pragma unroll
        for (int i = 0; i < CQ_P; ++i) {
          pan[i * PS + tid] = v[i];
          if (j >= k0 + i) W[cq_row(k0 + i, N) + j] = v[i];
        }
      }
    }
    __syncthreads();
    // the rest: four rows i0 .. i0 + 3 per warp, a column per lane
    for (int i0 = k0 + CQ_P + 4 * warp; i0 < N; i0 += 4 * nw) {
      double m[CQ_P][4];
      double* row[4];
#pragma unroll
      for (int p = 0; p < CQ_P; ++p) {
        const double2 m0 = *reinterpret_cast<const double2*>(pan + p * PS + (i0 - k0));
        const double2 m1 = *reinterpret_cast<const double2*>(pan + p * PS + (i0 - k0) + 2);
        m[p][0] = m0.x; m[p][1] = m0.y; m[p][2] = m1.x; m[p][3] = m1.y;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) row[e] = W + cq_row(min(i0 + e, N - 1), N);
      for (int c = i0 + lane; c < N; c += 32) {
        double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int p = 0; p < CQ_P; ++p) {
          const double x = pan[p * PS + (c - k0)];
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] = fma(m[p][e], x, a[e]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (i0 + e <= c) row[e][c] -= a[e];
      }
    }
    __syncthreads();
  }
}

}  // namespace ttr
