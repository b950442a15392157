// CholeskyQR of tall FP32 matrices (n x N column-major, N <= 128): FP64 Gram, FP64 Cholesky, rows
// solved against R in FP32.  Replaces basicQR = geqrf + orgqr (TT3O:85-159).
//
// What bounds it is latency: a sketch is a few hundred rows of a few dozen columns, and the
// factorisation is a chain of N pivots.  So:
//  * Cholesky by panels of 8 rows of R.  Every thread factors the panel's 8 x 8 diagonal block for
//    itself in registers (a chain of 8 FP64 reciprocal square roots, 55 cycles each, no shuffle, no
//    division) and finishes one column of the panel; the block then applies the panel to the rest:
//    three barriers per 8 pivots.
//  * The Gram converts each row to FP64 once, 32 rows at a time (conversions run at ~8 per clock and
//    SM, an eighth of the FP64 FMAs), into 8 x 8 tiles whose components are interleaved, so that the
//    loads of a warp are consecutive words; row groups are summed from shared memory.
//  * Rows are solved in panels of 8 columns: 32 independent sums per row instead of 4 per column, the
//    row itself in shared memory, so one code serves every N and stays in the instruction cache.
//    Above 64 columns (80 for few rows), and where the rows are too many for one launch, the rows are
//    multiplied by R^-1 (FP64, rounded once): no chain at all per row.
//  * `exact` rows (the decompositions on the FP32 engine): the first pass divides in FP64 and rounds each entry
//    once.  An FP32 reciprocal pivot makes a whole column of Q longer or shorter by up to 2^-24, which the second
//    pass cannot mend (its factor 1 + 3e-8 rounds back), and close eigenvectors of B B^T tilt by that over their
//    gap: interior bases of a 24^6 tensor at ranks 24 come out 3 to 5 times closer to their 64-bit values.
//    The second pass then finds R = I to 1e-9 and has nothing to round.  256^3, ranks 16: 680 us (678 without).
// CholeskyQR2 of 384 x 24: 32 us; 1024 x 40: 49; 256 x 80: 118; 640 x 96: 187.  What is left is the chain: at
// 1024 x 40, per pass, 14k cycles of Cholesky, 8.5k of Gram, 6k for the cluster's sum, 6k of row solves.
// Small matrices take one launch, a cluster of up to 8 CTAs (kCqRows and cholqr_passes below have the rule).
#include <algorithm>

#include "chol.cuh"
#include "kernels.cuh"

namespace ttr {
namespace {

constexpr int CQ_T = 256;   // threads per CTA
constexpr int CQ_RC = 32;   // rows converted to FP64 at a time

int cq_packed(int N) { return N * (N + 1) / 2; }
int cq_rstride(int N) { return (N + 7) & ~7; }  // row stride of the FP32 copy of R

// Cluster helpers: rank in the cluster, cluster size, cluster-wide barrier (release / acquire),
// and an FP64 load from the same shared-memory offset in another CTA of the cluster.
__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ double ld_peer_f64(const double* p, unsigned rank) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  unsigned ra;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(ra) : "memory");
  return v;
}

// W (packed R) <- R^-1, in place, by the whole block: 8 rows at a time from the bottom.  A thread
// pair holds a column j of those rows (the pair splits the sum over k), T[i][j] = -(sum_{k > i} R[i][k]
// T[k][j]) / R[i][i], T[j][j] = 1 / R[j][j]; a dependent column (inv 0) comes out zero.  rt: the rows'
// R staged k-major (N x 8, at least 8 x 8: the bottom rows' triangle is read whole, zero past N), red: 8 x 128
// partial sums.  Ends with a block barrier.
constexpr int cq_rt(int N) { return (N > CQ_P ? N : CQ_P) * CQ_P; }
constexpr int cq_inv(int N) { return cq_rt(N) + CQ_P * 128; }  // doubles of both
__device__ void invert_upper(double* W, int N, const double* inv, double* rt, double* red) {
  const int tid = threadIdx.x, j = tid & 127, h = tid >> 7;
  for (int k0 = ((N - 1) / CQ_P) * CQ_P; k0 >= 0; k0 -= CQ_P) {
    const int k1 = min(k0 + CQ_P, N);
    for (int idx = tid; idx < max(N - k0, CQ_P) * CQ_P; idx += CQ_T) {
      const int k = k0 + idx / CQ_P, i = k0 + idx % CQ_P;
      rt[(k - k0) * CQ_P + (i - k0)] = (k < N && k > i) ? W[cq_row(i, N) + k] : 0.0;
    }
    __syncthreads();
    double a[CQ_P];
#pragma unroll
    for (int i = 0; i < CQ_P; ++i) a[i] = 0.0;
    if (j < N) {
#pragma unroll 2
      for (int k = k1 + h; k <= j; k += 2) {
        const double t = W[cq_row(k, N) + j];
        const double2* r = reinterpret_cast<const double2*>(rt + (k - k0) * CQ_P);
#pragma unroll
        for (int i = 0; i < CQ_P / 2; ++i) {
          const double2 v = r[i];
          a[2 * i] = fma(v.x, t, a[2 * i]);
          a[2 * i + 1] = fma(v.y, t, a[2 * i + 1]);
        }
      }
    }
    if (h == 1) {
#pragma unroll
      for (int i = 0; i < CQ_P; ++i) red[i * 128 + j] = a[i];
    }
    __syncthreads();
    if (h == 0 && j >= k0 && j < N) {
#pragma unroll
      for (int i = CQ_P - 1; i >= 0; --i) {
        double x = a[i] + red[i * 128 + j];
#pragma unroll
        for (int k = i + 1; k < CQ_P; ++k) x = fma(rt[k * CQ_P + i], a[k], x);  // rows of this block
        const int gi = k0 + i;
        a[i] = gi > j || gi >= N ? 0.0 : gi == j ? inv[gi] : -x * inv[gi];
        if (gi <= j) W[cq_row(gi, N) + j] = a[i];
      }
    }
    __syncthreads();
  }
}

// q R = y for one row, in place (row in shared memory): panels of 8 columns, R's rows as FP32
// (stride RS), inv the reciprocals of its diagonal (0: the column is dependent and comes out 0).
// Each column sums its products in four chains (k mod 4).
__device__ __forceinline__ void solve_row(float* row, int N, const float* Rf, int RS, const float* inv) {
  for (int p = 0; p < N; p += CQ_P) {
    uint64_t acc[4][4];  // chain, column pair
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float lo = p + 2 * c < N ? row[p + 2 * c] : 0.f, hi = p + 2 * c + 1 < N ? row[p + 2 * c + 1] : 0.f;
      acc[0][c] = f2_pack(lo, hi);
      acc[1][c] = acc[2][c] = acc[3][c] = 0ull;
    }
    for (int k = 0; k < p; k += 4) {
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint64_t q = f2_dup(-row[k + m]);
        const ulonglong2 r0 = *reinterpret_cast<const ulonglong2*>(Rf + (k + m) * RS + p);
        const ulonglong2 r1 = *reinterpret_cast<const ulonglong2*>(Rf + (k + m) * RS + p + 4);
        ffma2(acc[m][0], q, r0.x);
        ffma2(acc[m][1], q, r0.y);
        ffma2(acc[m][2], q, r1.x);
        ffma2(acc[m][3], q, r1.y);
      }
    }
    float a[4][CQ_P];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int c = 0; c < 4; ++c) f2_unpack(acc[m][c], a[m][2 * c], a[m][2 * c + 1]);
#pragma unroll
    for (int k = 0; k < CQ_P; ++k) {
      if (p + k < N) {
        const float q = ((a[0][k] + a[1][k]) + (a[2][k] + a[3][k])) * inv[p + k];
        row[p + k] = q;
        const float* R = Rf + (p + k) * RS + p;
#pragma unroll
        for (int c = k + 1; c < CQ_P; ++c) a[k & 3][c] = fmaf(-q, R[c], a[k & 3][c]);
      }
    }
  }
}

// The same with FP64 products, sums and reciprocals against R in FP64 (packed).
__device__ __forceinline__ void solve_row64(float* row, int N, const double* W, const double* inv) {
  for (int p = 0; p < N; p += CQ_P) {
    double a[CQ_P];
#pragma unroll
    for (int c = 0; c < CQ_P; ++c) a[c] = p + c < N ? (double)row[p + c] : 0.0;
    const int last = N - 1 - p;  // columns past the end repeat the last one
#pragma unroll 2
    for (int k = 0; k < p; ++k) {
      const double q = -(double)row[k];
      const double* R = W + cq_row(k, N) + p;
#pragma unroll
      for (int c = 0; c < CQ_P; ++c) a[c] = fma(q, R[min(c, last)], a[c]);
    }
#pragma unroll
    for (int k = 0; k < CQ_P; ++k) {
      if (p + k < N) {
        const float qf = (float)(a[k] * inv[p + k]);
        row[p + k] = qf;
        const double q = -(double)qf;
        const double* R = W + cq_row(p + k, N) + p;
#pragma unroll
        for (int c = k + 1; c < CQ_P; ++c) a[c] = fma(q, R[min(c, last)], a[c]);
      }
    }
  }
}

// q = y T for one row, in place, T upper triangular (FP32 or FP64 rows of stride RS; products and sums in its
// type): panels of 8 columns from the last one down, so that a panel overwrites what no later one reads.
__device__ __forceinline__ void mul_row(float* row, int N, const float* Tf, int RS) {
  for (int p = ((N - 1) / CQ_P) * CQ_P; p >= 0; p -= CQ_P) {
    uint64_t acc[4] = {0ull, 0ull, 0ull, 0ull};
    const int kend = min(p + CQ_P, N);
#pragma unroll 4
    for (int k = 0; k < kend; ++k) {
      const uint64_t q = f2_dup(row[k]);
      const ulonglong2 t0 = *reinterpret_cast<const ulonglong2*>(Tf + k * RS + p);
      const ulonglong2 t1 = *reinterpret_cast<const ulonglong2*>(Tf + k * RS + p + 4);
      ffma2(acc[0], q, t0.x);
      ffma2(acc[1], q, t0.y);
      ffma2(acc[2], q, t1.x);
      ffma2(acc[3], q, t1.y);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float lo, hi;
      f2_unpack(acc[c], lo, hi);
      if (p + 2 * c < N) row[p + 2 * c] = lo;
      if (p + 2 * c + 1 < N) row[p + 2 * c + 1] = hi;
    }
  }
}

__device__ __forceinline__ void mul_row(float* row, int N, const double* T, int RS) {
  for (int p = ((N - 1) / CQ_P) * CQ_P; p >= 0; p -= CQ_P) {
    double a[CQ_P];
#pragma unroll
    for (int c = 0; c < CQ_P; ++c) a[c] = 0.0;
    const int kend = min(p + CQ_P, N);
#pragma unroll 2
    for (int k = 0; k < kend; ++k) {
      const double q = (double)row[k];
      const double2* t = reinterpret_cast<const double2*>(T + k * RS + p);
#pragma unroll
      for (int c = 0; c < CQ_P / 2; ++c) {
        const double2 v = t[c];
        a[2 * c] = fma(q, v.x, a[2 * c]);
        a[2 * c + 1] = fma(q, v.y, a[2 * c + 1]);
      }
    }
#pragma unroll
    for (int c = 0; c < CQ_P; ++c)
      if (p + c < N) row[p + c] = (float)a[c];
  }
}

// Copy of the packed triangle W (FP32 or FP64 rows of stride RS, zero outside it; `diag`: with its diagonal).
template <typename T>
__device__ void write_tri(const double* W, int N, bool diag, T* Rf, int RS) {
  for (int k = threadIdx.x >> 5; k < N; k += CQ_T / 32)
    for (int c = threadIdx.x & 31; c < RS; c += 32)
      Rf[k * RS + c] = (c > k - (diag ? 1 : 0) && c < N) ? (T)W[cq_row(k, N) + c] : T(0);
}

// Whether k_cholqr_cluster solves its rows against R (four partial sums an entry) or multiplies them by R^-1 (one
// chain of FP32 products with a rounded inverse).  Solving is the more exact form and, up to 80 columns, the faster
// one (CholeskyQR2 of 256 x 80: 118 us, 151 with the inverse; 448 x 72: 107, 135; 1024 x 80: 132, 170).  Above 64
// columns it ends all the same where the rows (odd multiples of 16 bytes) and W no longer fit 206,528 bytes of one
// CTA: a TF32 decomposition without power iterations follows the rounding of its noise columns (3e-5 of a core when
// the form changes), so the sizes keep the form that they have always had.
__host__ __device__ constexpr bool cq_solves(long long n, int N) {
  return N <= 64 || (N <= 80 && 16 * n * (((N + 3) / 4) | 1) + 8 * ((N * N + 1) & ~1) <= 206528);
}
constexpr int cq_tile(int N) { return N <= 56 ? 4 : 8; }  // Gram tile: 4 x 4 keeps the threads busy (N = 56: 69 against 83 us)

// Shared memory of k_cholqr_cluster (bytes), `rpc` rows per CTA.
struct CqSmem {
  size_t ys, work, part, w, slice, total;
};
CqSmem cq_smem(long long n, int N, int rpc, int cl) {
  auto up = [](size_t b) { return (b + 15) & ~size_t(15); };
  CqSmem s;
  const size_t E = (size_t)cq_packed(N), rf = (size_t)N * cq_rstride(N) * 4;
  const int ts = cq_tile(N), tt = (N + ts - 1) / ts;
  s.ys = up((size_t)rpc * (N | 1) * 4);
  s.work = up(8 * (size_t)std::max({CQ_RC * tt * ts, CQ_T * 16, cq_pan(N), cq_solves(n, N) ? 0 : cq_inv(N)}));
  s.part = up(std::max(E * 8, rf));
  s.w = up(E * 8);
  s.slice = up((E + cl - 1) / cl * 8);
  s.total = s.ys + s.work + s.part + s.w + s.slice + up((size_t)N * 8) + up((size_t)N * 4);
  return s;
}

// CholeskyQR2 of Y in one launch: a cluster of CTAs, `rpc` consecutive rows each in
// shared memory.  Per pass: partial Gram of the CTA's rows, summed over the cluster through
// distributed shared memory (each rank sums one slice in rank order, then all gather the slices: the
// same bits everywhere, so the redundant factorisations agree), Cholesky, row solves.  y64 (or null):
// Y in FP64, rounded on the way in.  r (or null): R2 R1 (r1: N x N scratch).  exact: see above.
template <int TS>
__global__ void __launch_bounds__(CQ_T, 1) k_cholqr_cluster(const double* __restrict__ y64, float* __restrict__ y,
                                                            int n, int N, long long ld, int rpc, CqSmem lay,
                                                            double* __restrict__ r, double* __restrict__ r1,
                                                            double rel_tol, bool exact) {
  extern __shared__ __align__(16) unsigned char sm_cq[];
  float* const Ys = reinterpret_cast<float*>(sm_cq);                       // rpc x SN
  double* const Yd = reinterpret_cast<double*>(sm_cq + lay.ys);            // FP64 rows / group sums / panel
  double* const P = reinterpret_cast<double*>(sm_cq + lay.ys + lay.work);  // partial Gram, then R (R^-1) in FP32
  double* const W = P + lay.part / 8;
  double* const S = W + lay.w / 8;
  double* const inv = S + lay.slice / 8;
  float* const invf = reinterpret_cast<float*>(inv + ((N + 1) & ~1));
  float* const Rf = reinterpret_cast<float*>(P);
  const unsigned crank = cl_rank(), csize = cl_size();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int TT = (N + TS - 1) / TS;  // component ta + TT p of the rows is component p of tile index ta
  const int SN = N | 1, LD = TT * TS, RS = (N + 7) & ~7, E = N * (N + 1) / 2;
  const long long row0 = (long long)crank * rpc;
  const int nl = (int)max(0LL, min((long long)rpc, n - row0));
  for (int i0 = lane; i0 < nl; i0 += 128) {
#pragma unroll 2
    for (int c = warp; c < N; c += CQ_T / 32) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + 32 * u;
        v[u] = i >= nl ? 0.f : y64 ? (float)y64[row0 + i + (long long)n * c] : y[row0 + i + ld * c];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + 32 * u < nl) Ys[(i0 + 32 * u) * SN + c] = v[u];
    }
  }
  // Gram tile (ta, tb), ta <= tb, of this thread, for the rows of its group
  const int nt = TT * (TT + 1) / 2;
  const int groups = min(CQ_RC, max(1, CQ_T / nt));
  const int t = tid % nt, g = tid / nt;
  int ta = 0, rem = t;
  while (rem >= TT - ta) {
    rem -= TT - ta;
    ++ta;
  }
  const int tb = ta + rem;
  for (int pass = 0; pass < 2; ++pass) {
    double acc[TS][TS];
#pragma unroll
    for (int p = 0; p < TS; ++p)
#pragma unroll
      for (int q = 0; q < TS; ++q) acc[p][q] = 0.0;
    for (int c0 = 0; c0 < nl; c0 += CQ_RC) {
      const int nr = min(CQ_RC, nl - c0);
      __syncthreads();  // the rows (or the previous pass's) are written, the last chunk is consumed
      for (int c = lane; c < LD; c += 32) {
        float x[CQ_RC / 8];  // a column of this warp's rows: loads, conversions and stores overlap
#pragma unroll
        for (int u = 0; u < CQ_RC / 8; ++u)
          x[u] = (c < N && warp + 8 * u < nr) ? Ys[(c0 + warp + 8 * u) * SN + c] : 0.f;
#pragma unroll
        for (int u = 0; u < CQ_RC / 8; ++u)
          if (warp + 8 * u < nr) Yd[(warp + 8 * u) * LD + c] = (double)x[u];
      }
      __syncthreads();
      if (g < groups) {
        for (int v = g; v < nr; v += groups) {
          double av[TS], bv[TS];
#pragma unroll
          for (int p = 0; p < TS; ++p) {
            av[p] = Yd[v * LD + ta + TT * p];
            bv[p] = Yd[v * LD + tb + TT * p];
          }
#pragma unroll
          for (int p = 0; p < TS; ++p)
#pragma unroll
            for (int q = 0; q < TS; ++q) acc[p][q] = fma(av[p], bv[q], acc[p][q]);
        }
      }
    }
    // group sums, 16 entries of the tiles at a time: 16 threads an entry, a tile each
#pragma unroll
    for (int h = 0; h < TS * TS / 16; ++h) {
      __syncthreads();
#pragma unroll
      for (int e = 0; e < 16; ++e) Yd[e * CQ_T + tid] = acc[(16 * h + e) / TS][(16 * h + e) % TS];
      __syncthreads();
      const int e = tid >> 4, p = (16 * h + e) / TS, q = (16 * h + e) % TS;
      int a = 0, off = tid & 15;  // tile u = (a, a + off)
      for (int u = tid & 15; u < nt; u += 16, off += 16) {
        while (off >= TT - a) {
          off -= TT - a;
          ++a;
        }
        const int i = a + TT * p, j = a + off + TT * q;
        if (i >= N || j >= N || (off == 0 && p > q)) continue;
        double sum = 0.0;
        for (int z = 0; z < groups; ++z) sum += Yd[e * CQ_T + z * nt + u];
        P[cq_row(min(i, j), N) + max(i, j)] = sum;
      }
    }
    if (csize > 1) {
      const int sl = (E + (int)csize - 1) / (int)csize;
      cl_sync();
      for (int e = tid; e < sl; e += CQ_T) {
        const int idx = (int)crank * sl + e;
        if (idx >= E) break;
        double v[8];
#pragma unroll
        for (unsigned q = 0; q < 8; ++q) v[q] = q < csize ? ld_peer_f64(P + idx, q) : 0.0;
        double sum = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) sum += v[q];
        S[e] = sum;
      }
      cl_sync();  // slices complete; no peer reads this CTA's partial any more
      for (unsigned q = 0; q < csize; ++q)
        for (int e = tid; e < sl; e += CQ_T)
          if ((int)q * sl + e < E) W[q * sl + e] = ld_peer_f64(S + e, q);
    } else {
      __syncthreads();
      for (int idx = tid; idx < E; idx += CQ_T) W[idx] = P[idx];
    }
    __syncthreads();
    chol_panels(W, N, rel_tol, inv, Yd);
    if (r && crank == 0) {
      for (int idx = tid; idx < N * N; idx += CQ_T) {
        const int c = idx / N, k = idx - c * N;
        if (pass == 0) {
          r1[idx] = k <= c ? W[cq_row(k, N) + c] : 0.0;
        } else {
          double a = 0.0;
          for (int j = k; j <= c; ++j) a = fma(W[cq_row(k, N) + j], r1[j + N * c], a);
          r[idx] = a;
        }
      }
    }
    if (exact && pass == 0) {
      for (int i = tid; i < nl; i += CQ_T) solve_row64(Ys + i * SN, N, W, inv);
    } else if (cq_solves(n, N)) {
      write_tri(W, N, false, Rf, RS);
      for (int k = tid; k < N; k += CQ_T) invf[k] = (float)inv[k];
      __syncthreads();
      for (int i = tid; i < nl; i += CQ_T) solve_row(Ys + i * SN, N, Rf, RS, invf);
    } else {
      __syncthreads();  // R is out
      invert_upper(W, N, inv, Yd, Yd + cq_rt(N));
      write_tri(W, N, true, Rf, RS);
      __syncthreads();
      for (int i = tid; i < nl; i += CQ_T) mul_row(Ys + i * SN, N, Rf, RS);
    }
  }
  __syncthreads();
  for (int c = warp; c < N; c += CQ_T / 32)
    for (int i = lane; i < nl; i += 32) y[row0 + i + ld * c] = Ys[i * SN + c];
  if (csize > 1) cl_sync();  // peers may still be gathering this CTA's slice
}

// W (N x N, column-major) -> R^-1 (rows of stride RS) for k_apply_t; R in FP64 (or null).
template <typename T>
__global__ void __launch_bounds__(CQ_T, 1) k_chol_inv(const double* __restrict__ w, int N, double rel_tol,
                                                      T* __restrict__ tf, double* __restrict__ r_out) {
  extern __shared__ __align__(16) double sm_ch[];
  double* const work = sm_ch;  // panel, then the inversion's scratch
  double* const W = work + cq_inv(N);
  double* const inv = W + N * (N + 1) / 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int j = warp; j < N; j += CQ_T / 32)  // column j, rows 0..j
    for (int i = lane; i <= j; i += 32) W[cq_row(i, N) + j] = w[i + (long long)N * j];
  __syncthreads();
  chol_panels(W, N, rel_tol, inv, work);
  if (r_out) {
    for (int idx = tid; idx < N * N; idx += CQ_T) {
      const int c = idx / N, k = idx - c * N;
      r_out[idx] = k <= c ? W[cq_row(k, N) + c] : 0.0;
    }
    __syncthreads();
  }
  invert_upper(W, N, inv, work, work + cq_rt(N));
  write_tri(W, N, true, tf, (N + 7) & ~7);
}

// Y (n x N, column-major) <- Y T, T = R^-1.  A thread owns a row: the loads and stores of a warp are
// runs of 32 rows of a column, the row waits in the thread's own line of shared memory (odd stride),
// so nothing but T is shared and tiles need no barrier.  HBM / FP32 FMA bound: N (N + 1) / 2 FMAs per
// 8 N bytes (262144 x 80: 128 us).  An FP64 T takes twice the shared memory, so half the rows.
template <typename T>
constexpr int cq_apply_rows() { return sizeof(T) == 8 ? CQ_T / 2 : CQ_T; }
template <typename T>
__global__ void __launch_bounds__(CQ_T) k_apply_t(float* __restrict__ y, long long n, int N, long long ld,
                                                  const T* __restrict__ tf) {
  constexpr int ROWS = cq_apply_rows<T>();
  extern __shared__ __align__(16) unsigned char sm_ar[];
  const int RS = (N + 7) & ~7, SN = N | 1, tid = threadIdx.x;
  T* const Ts = reinterpret_cast<T*>(sm_ar);
  float* const row = reinterpret_cast<float*>(Ts + N * RS) + tid * SN;
  for (int idx = tid; idx < N * RS; idx += ROWS) Ts[idx] = tf[idx];
  __syncthreads();
  for (long long j = (long long)blockIdx.x * ROWS + tid; j < n; j += (long long)gridDim.x * ROWS) {
    float* src = y + j;
#pragma unroll 16
    for (int c = 0; c < N; ++c) row[c] = src[ld * c];
    mul_row(row, N, Ts, RS);
#pragma unroll 8
    for (int c = 0; c < N; ++c) src[ld * c] = row[c];
  }
}

// R = R2 * R1 (upper triangular, FP64).
__global__ void k_mul_upper(const double* __restrict__ r2, const double* __restrict__ r1, int N,
                            double* __restrict__ r) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= N * N) return;
  const int i = idx % N, j = idx / N;
  double acc = 0.0;
  for (int k = i; k <= j; ++k) acc += r2[i + (long long)N * k] * r1[k + (long long)N * j];
  r[idx] = (j >= i) ? acc : 0.0;
}

// Rows up to which the eight SMs of a cluster are as fast as the whole GPU in seven launches.  One launch against
// several, us: 7,000 x 2 61 / 63, 10,000 x 2 72 / 63, 100,000 x 2 334 / 62; 7,000 x 16 87 / 75, 15,000 x 16 123 / 75;
// 15,000 x 24 144 / 87.
constexpr long long kCqRows = 8192;
constexpr double kCqTol = 1e-12;  // pivots below this share of the largest diagonal: dependent columns

// The pass Y <- Y R^-1 of the Gram w, R^-1 through `tf` (N rows of stride RS), R to r (or null).
template <typename T>
int apply_inverse(float* y, long long n, int N, long long ld, const double* w, T* tf, double* r, cudaStream_t s) {
  constexpr int ROWS = cq_apply_rows<T>();
  const size_t csm = ((size_t)cq_inv(N) + cq_packed(N) + N) * sizeof(double);
  const size_t asm_ = (size_t)N * cq_rstride(N) * sizeof(T) + (size_t)ROWS * (N | 1) * sizeof(float);
  TT_TRY(smem_optin_k(k_chol_inv<T>, csm));
  TT_TRY(smem_optin_k(k_apply_t<T>, asm_));
  // persistent blocks (T staged once per block), as many as fit on the SMs
  const int per_sm = std::max(1, std::min(8, (int)((size_t)dev_smem_max() / (asm_ + 1024))));
  const int grid = (int)std::min<long long>(ceil_div_ll(n, ROWS), (long long)per_sm * dev_sms());
  k_chol_inv<T><<<1, CQ_T, csm, s>>>(w, N, kCqTol, tf, r);
  count_launch();
  TT_LAUNCH_CHECK();
  k_apply_t<T><<<grid, ROWS, asm_, s>>>(y, n, N, ld, tf);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

int cholqr_passes(const double* y64, float* y, long long n, int N, long long ld, double* r, Arena& ws,
                  cudaStream_t s, int passes, bool exact) {
  if (N <= 0 || n <= 0) return TT_OK;
  if (N > TT_MAX_SMALL) {
    set_error(TT_ERR_UNSUPPORTED, "cholqr2 width %d > %d", N, TT_MAX_SMALL);
    return TT_ERR_UNSUPPORTED;
  }
  const size_t mk = ws.mark();
  double* r1 = ws.take<double>((size_t)N * N);
  if (!r1) {
    set_error(TT_ERR_NOMEM, "cholqr2 workspace");
    return TT_ERR_NOMEM;
  }
  // One launch up to kCqRows rows where they fit the shared memory of 8 CTAs (at N = 40 1,130 rows each): CTAs of
  // at least 64 rows, as few as fit.
  if (n <= (1LL << 20)) {
    for (int cl = (int)std::min<long long>(8, ceil_div_ll(n, 64)); cl <= 8; ++cl) {
      const int rpc = (int)ceil_div_ll(n, cl);
      const CqSmem lay = cq_smem(n, N, rpc, cl);
      if (lay.total > (size_t)dev_smem_max()) continue;
      if (n > kCqRows) {
        passes = 2;  // as in one launch
        break;
      }
      TT_TRY(smem_optin_k(k_cholqr_cluster<4>, dev_smem_max()));
      TT_TRY(smem_optin_k(k_cholqr_cluster<8>, dev_smem_max()));
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(cl, 1, 1);
      cfg.blockDim = dim3(CQ_T, 1, 1);
      cfg.dynamicSmemBytes = lay.total;
      cfg.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = cl;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      const cudaError_t e =
          cq_tile(N) == 4 ? cudaLaunchKernelEx(&cfg, k_cholqr_cluster<4>, y64, y, (int)n, N, ld, rpc, lay, r, r1, kCqTol, exact)
                          : cudaLaunchKernelEx(&cfg, k_cholqr_cluster<8>, y64, y, (int)n, N, ld, rpc, lay, r, r1, kCqTol, exact);
      if (e == cudaSuccess) {
        count_launch();
        TT_LAUNCH_CHECK();
        ws.reset(mk);
        return TT_OK;
      }
      // A cluster that cannot be placed (its CTAs' shared memory on one GPC) takes the launches below.
      (void)cudaGetLastError();
      break;
    }
  }
  if (y64) TT_TRY(launch_f64_to_f32_cols(y64, n, n, N, y, ld, N, s));
  double* w = ws.take<double>((size_t)N * N);
  double* r2 = ws.take<double>((size_t)N * N);
  double* tf = ws.take<double>((size_t)N * cq_rstride(N));
  if (!w || !r2 || !tf) {
    set_error(TT_ERR_NOMEM, "cholqr2 workspace");
    return TT_ERR_NOMEM;
  }
  for (int pass = 0; pass < passes; ++pass) {
    TT_TRY(launch_gram(y, n, N, 1, ld, w, ws, s));
    double* rp = !r ? nullptr : pass == 0 ? r1 : r2;
    if (exact && pass == 0) TT_TRY(apply_inverse(y, n, N, ld, w, tf, rp, s));
    else TT_TRY(apply_inverse(y, n, N, ld, w, reinterpret_cast<float*>(tf), rp, s));
  }
  if (r && passes == 2) {
    k_mul_upper<<<ceil_div(N * N, 256), 256, 0, s>>>(r2, r1, N, r);
    count_launch();
    TT_LAUNCH_CHECK();
  }
  ws.reset(mk);
  return TT_OK;
}

}  // namespace

int launch_cholqr2(const double* y64, float* y, long long n, int N, long long ld, double* r, Arena& ws,
                   cudaStream_t s, bool exact) {
  return cholqr_passes(y64, y, n, N, ld, r, ws, s, 2, exact);
}

// One CholeskyQR pass: the orthonormalisation between power iterations, which only has to keep
// the basis well conditioned (the sketch that follows is orthonormalised by CholeskyQR2): a basis whose
// columns span a graded spectrum (condition kappa) comes out with orthogonality ~kappa * 2^-24.  A
// basis that fits one launch gets both passes there.
int launch_orth_power(float* y, long long n, int N, long long ld, Arena& ws, cudaStream_t s) {
  return cholqr_passes(nullptr, y, n, N, ld, nullptr, ws, s, 1, false);
}

}  // namespace ttr
