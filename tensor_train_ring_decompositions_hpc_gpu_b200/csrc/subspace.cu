// Leading eigenpairs of a symmetric positive semidefinite matrix, 64 < N <= 128, of which only the first few are
// used: orthogonal (subspace) iteration on a block of kSubDim columns, then Rayleigh-Ritz.  One CTA holds W (FP64)
// and two blocks of kSubDim columns in shared memory (column-major, rows padded to a multiple of 8 with zeros).
// The start block is Philox Gaussian; every second multiplication by W the block is orthonormalised by one
// CholeskyQR pass, and the last basis gets a second one (CholeskyQR2).  The projected matrix H = Y^T W Y
// (kSubDim x kSubDim) goes to the N <= 32 Jacobi solver and the Ritz vectors are Y times its eigenvectors.  The
// span of the first k Ritz vectors converges to W's leading k-dimensional invariant subspace as
// (lambda_{kSubDim+1} / lambda_k)^kSubMults.
//
// Bound by latency and the FP64 rate of one SM: 17 products W Y (N^2 x 32 FMAs, 1.7 us each at N = 80), 10 Gram
// matrices, Cholesky factors and row solves.  All products are on the FP64 matrix instructions, fragments straight
// from shared memory: a leading dimension of 4 or 12 modulo 16 puts the 4 x 4 values of a half warp in distinct
// banks.  N = 80: 165 us.
#include "chol.cuh"
#include "kernels.cuh"
#include "philox.cuh"

namespace ttr {
namespace {

constexpr int kSubDim = 32;
constexpr int kSubMults = 16;
constexpr int SU_T = 512;

constexpr int su_rows(int N) { return (N + 7) & ~7; }
constexpr int su_ld(int N) { return su_rows(N) + 4; }
constexpr int kSubPacked = kSubDim * (kSubDim + 1) / 2;

// Upper tile (p, q) of the kSubDim / 8 x kSubDim / 8 tiles, in rows.
__device__ __forceinline__ void su_tile(int e, int& p, int& q) {
  constexpr int T = kSubDim / 8;
  p = 0;
  while (e >= T - p) {
    e -= T - p;
    ++p;
  }
  q = p + e;
}

// Y = an orthonormal basis of span(Y), in place.  Columns whose pivot is below 1e-28 of the largest diagonal of
// Y^T Y (directions W annihilates) come out zero.
__device__ __noinline__ void sub_cholqr(double* Y, int rows, int LD, double* G, double* inv, double* pan) {
  constexpr int B = kSubDim;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lk = lane & 3, lr = lane >> 2;
  if (warp < 10) {
    int p, q;
    su_tile(warp, p, q);
    double c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
    const double* a = Y + (8 * p + lr) * LD + lk;
    const double* b = Y + (8 * q + lr) * LD + lk;
#pragma unroll 2
    for (int k = 0; k < rows; k += 8) {
      mma_f64(c0, a[k], b[k]);
      mma_f64(c1, a[k + 4], b[k + 4]);
    }
    const int i = 8 * p + lr;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int j = 8 * q + 2 * lk + e;
      if (i <= j) G[cq_row(i, B) + j] = c0[e] + c1[e];
    }
  }
  __syncthreads();
  chol_panels(G, B, 1e-28, inv, pan);
  // row i: q R = y, every later column updated as soon as one is known
  for (int i = tid; i < rows; i += SU_T) {
    double y[B];
#pragma unroll
    for (int c = 0; c < B; ++c) y[c] = Y[c * LD + i];
#pragma unroll
    for (int c = 0; c < B; ++c) {
      y[c] *= inv[c];
      const double* R = G + cq_row(c, B);
#pragma unroll
      for (int c2 = c + 1; c2 < B; ++c2) y[c2] = fma(-y[c], R[c2], y[c2]);
    }
#pragma unroll
    for (int c = 0; c < B; ++c) Y[c * LD + i] = y[c];
  }
  __syncthreads();
}

// Z = W Y: a warp forms 8 rows of 16 columns.
__device__ __noinline__ void sub_mult(const double* W, const double* Y, double* Z, int rows, int LD) {
  const int lane = threadIdx.x & 31, lk = lane & 3, lr = lane >> 2;
  for (int u = threadIdx.x >> 5; u < rows / 8 * 2; u += SU_T / 32) {
    const int i0 = 8 * (u >> 1), q0 = 16 * (u & 1);
    double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    const double* a = W + lk * LD + i0 + lr;  // W is symmetric: its rows are its columns
    const double* b = Y + (q0 + lr) * LD + lk;
#pragma unroll 4
    for (int k = 0; k < rows; k += 4) {
      const double av = a[k * LD];
      mma_f64(c[0], av, b[k]);
      mma_f64(c[1], av, b[8 * LD + k]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) Z[(q0 + 8 * h + 2 * lk + e) * LD + i0 + lr] = c[h][e];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(SU_T, 1) k_subspace_iter(const double* __restrict__ w_in, int N,
                                                           unsigned long long seed, double* __restrict__ y_out,
                                                           double* __restrict__ h_out) {
  extern __shared__ __align__(16) double sm_sub[];
  constexpr int B = kSubDim;
  const int rows = su_rows(N), LD = su_ld(N);
  double* Ws = sm_sub;              // rows x rows
  double* Ys = Ws + rows * LD;      // rows x B
  double* Zs = Ys + B * LD;         // rows x B
  double* pan = Zs + B * LD;        // cq_pan(B)
  double* G = pan + cq_pan(B);      // packed B x B
  double* inv = G + kSubPacked;     // B
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lk = lane & 3, lr = lane >> 2;
  for (int k = warp; k < rows; k += SU_T / 32)
    for (int i = lane; i < rows; i += 32)
      Ws[k * LD + i] = (i < N && k < N) ? 0.5 * (w_in[i + (long long)N * k] + w_in[k + (long long)N * i]) : 0.0;
  const int NP = N + (N & 1);  // the Gaussian calls go by this many rows
  for (int q = tid; q < NP * (B / 4); q += SU_T) {
    const int i = q % NP, c4 = 4 * (q / NP);
    const float4 g = philox_normal4((unsigned long long)q, 0x5ab5u, seed);
    const bool live = i < N;
    Ys[(c4 + 0) * LD + i] = live ? g.x : 0.0;
    Ys[(c4 + 1) * LD + i] = live ? g.y : 0.0;
    Ys[(c4 + 2) * LD + i] = live ? g.z : 0.0;
    Ys[(c4 + 3) * LD + i] = live ? g.w : 0.0;
  }
  for (int q = tid; q < (rows - NP) * B; q += SU_T) Ys[q / (rows - NP) * LD + NP + q % (rows - NP)] = 0.0;
  __syncthreads();
  sub_cholqr(Ys, rows, LD, G, inv, pan);
  for (int it = 0; it < kSubMults / 2; ++it) {
    sub_mult(Ws, Ys, Zs, rows, LD);
    sub_mult(Ws, Zs, Ys, rows, LD);
    sub_cholqr(Ys, rows, LD, G, inv, pan);
  }
  sub_cholqr(Ys, rows, LD, G, inv, pan);
  sub_mult(Ws, Ys, Zs, rows, LD);
  // H = (Y^T Z + Z^T Y) / 2, Y out column-major N x B
  if (warp < 10) {
    int p, q;
    su_tile(warp, p, q);
    double c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
    const int pa = (8 * p + lr) * LD + lk, qb = (8 * q + lr) * LD + lk;
    for (int k = 0; k < rows; k += 4) {
      mma_f64(c0, Ys[pa + k], Zs[qb + k]);
      mma_f64(c1, Zs[pa + k], Ys[qb + k]);
    }
    const int i = 8 * p + lr;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int j = 8 * q + 2 * lk + e;
      if (i <= j) {
        h_out[i + B * j] = 0.5 * (c0[e] + c1[e]);
        h_out[j + B * i] = 0.5 * (c0[e] + c1[e]);
      }
    }
  }
  for (int c = warp; c < B; c += SU_T / 32)
    for (int i = lane; i < N; i += 32) y_out[i + (long long)N * c] = Ys[c * LD + i];
}

// evecs (N x N) = [Y E, 0], evals = [lambda(H), 0]: the kSubDim Ritz pairs, zero beyond them.
__global__ void k_ritz(const double* __restrict__ y, const double* __restrict__ eh, const double* __restrict__ lh,
                       int N, double* __restrict__ evals, double* __restrict__ evecs) {
  constexpr int B = kSubDim;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < (long long)N * N;
       idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx % N), j = (int)(idx / N);
    double v = 0.0;
    if (j < B)
      for (int c = 0; c < B; ++c) v = fma(y[i + (long long)N * c], eh[c + B * j], v);
    evecs[idx] = v;
    if (i == 0) evals[j] = j < B ? lh[j] : 0.0;
  }
}

size_t syev_top_smem(int N) {
  return ((size_t)su_ld(N) * (su_rows(N) + 2 * kSubDim) + cq_pan(kSubDim) + kSubPacked + kSubDim) * sizeof(double);
}

}  // namespace

int launch_syev_top(const double* w, int N, double* evals, double* evecs, int max_sweeps, Arena& ws,
                    DevStatus* st, cudaStream_t s) {
  if (N <= 64 || N > TT_MAX_SMALL) return launch_syev(w, N, evals, evecs, max_sweeps, ws, st, s);
  const size_t mk = ws.mark();
  double* y = ws.take<double>((size_t)N * kSubDim);
  double* h = ws.take<double>((size_t)kSubDim * kSubDim);
  double* eh = ws.take<double>((size_t)kSubDim * kSubDim);
  double* lh = ws.take<double>(kSubDim);
  if (!y || !h || !eh || !lh) {
    set_error(TT_ERR_NOMEM, "subspace eigen-solver workspace");
    return TT_ERR_NOMEM;
  }
  const size_t shm = syev_top_smem(N);
  TT_TRY(smem_optin_k(k_subspace_iter, shm));
  k_subspace_iter<<<1, SU_T, shm, s>>>(w, N, 0x7c3a9e15ull, y, h);
  count_launch();
  TT_LAUNCH_CHECK();
  TT_TRY(launch_syev(h, kSubDim, lh, eh, max_sweeps, ws, st, s));
  k_ritz<<<ceil_div(N * N, 256), 256, 0, s>>>(y, eh, lh, N, evals, evecs);
  count_launch();
  TT_LAUNCH_CHECK();
  ws.reset(mk);
  return TT_OK;
}

}  // namespace ttr
