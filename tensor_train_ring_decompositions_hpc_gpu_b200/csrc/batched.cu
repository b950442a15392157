// Batched TT-SVD of many small tensors in one persistent launch.
//
// One CTA decomposes one tensor at a time and takes the next tensor index from a global work
// counter, so the SMs stay busy whatever the size mix.  Every step of a tensor runs inside the
// CTA: the exact Gram-eigen step when the small side of the unfolding is <= 32 (Gram in FP64,
// Jacobi in shared memory), otherwise EDrSVD (Philox Gaussian sketch generated on the fly, both
// CholeskyQR passes in shared memory, projection B = Q^T A with the Gram B B^T accumulated
// alongside, Jacobi).  Ranks follow the delta-truncation rule of tt_svd (eps > 0) or are the
// largest allowed (eps = 0), capped by rmax.  The unfoldings of the tensor being processed
// live in a per-CTA scratch (ping-pong), cores are written compactly in the caller's buffer.
// The reference decomposes one tensor per call (ttdec_gpu_float, ttdec_half_lu_device_6) and
// has no batched path.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "kernels.cuh"
#include "philox.cuh"
#include "bl_solver.cuh"

namespace ttr {
namespace {

constexpr int BT = 384;       // threads per CTA: the eigen-solver's 12 warps
constexpr int BSLOTS = 512;   // (tile, group of vectors) pairs of a Gram matrix
constexpr int BMAXM = 512;    // largest row count of a randomized unfolding
constexpr int BSMALL = 32;    // largest exact small side / sketch width
constexpr int BMAXD = 8;      // largest order
// Tunable: columns of the Gaussian test matrix generated per chunk of the sketch (BCH, a
// template parameter) and the order in which the work counter hands out tensors.
constexpr int kChunks[3] = {16, 32, 64};
enum { SCHED_NATURAL = 0, SCHED_LARGEST_FIRST = 1 };

struct BatchShape {
  int d;
  int n[BMAXD];
  long long size;
  long long x_off;
  long long core_off;
};

// Shared memory of the kernel: two CTAs share an SM (one waits at a barrier or in the eigen-solver's
// chain of rotations while the other works), so each has half of it and 80 registers per thread.
// 4096 tensors of order 4, 8-32 per mode: 18.2 ms with one CTA per SM, 14.9 with two.
constexpr int YQ_PAD = 4;                                                   // rows of Y, Q: W + 4 floats
constexpr size_t SM_STAGE = 9216 * sizeof(float);                             // least size of yq
constexpr size_t SM_W = (size_t)BSMALL * BSMALL * sizeof(double);             // Gram
constexpr size_t SM_JAC = 2 * (size_t)BSMALL * BSMALL * sizeof(double);       // Jacobi buffers
constexpr size_t SM_RED = (size_t)(BT / 32) * sizeof(double);                 // reductions
inline size_t sm_yq(int mrows) {  // mrows: rows of the tallest sketched step
  return std::max(SM_STAGE, (size_t)mrows * (BSMALL + YQ_PAD) * sizeof(float));
}
inline size_t sm_total(int mrows) { return sm_yq(mrows) + SM_W + SM_JAC + SM_RED; }

struct Smem {
  float* yq;      // Y, Q, U of a sketched step (rows of W + 4 floats); vectors of an exact step's Gram
  int yq_floats;
  double* w;      // BSMALL x BSMALL (row-major)
  double* jac;    // 2 x BSMALL^2: the eigen-solver's W; between solves Omega chunks, Gram partials, R, E_r
  double* red;    // BT / 32
};

__device__ double cta_sum(double v, double* red) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < BT / 32; ++w) t += red[w];
  __syncthreads();
  return t;
}

// Gram matrices W (N x N, row-major, stride N) = sum of v v^T over vectors of N <= BSMALL floats that lie as
// rows of 16-byte words (padded past N with anything finite or not: those products are dropped).  4 x 4
// register tiles of the upper triangle, vectors split into groups of threads, every `groups`-th vector to a
// group, groups added in order.  F32P: products summed in FP32 over 64 vectors of a thread, then in FP64
// (the Grams that feed an eigen-solve: relative errors ~1e-8 of the entries, and no FP64 conversion per
// product); otherwise FP64 products (CholeskyQR of a sketch, whose condition number the Gram squares).
// The groups number BSLOTS / tiles; a thread serves slot tid and, where there are more than BT of them, slot
// tid + BT after it.
struct GramTile {
  int nt, groups;
  int t[2], g[2], ta[2], tb[2];  // tile, group of the thread's slots
  __device__ explicit GramTile(int N) {
    const int TT = (N + 3) / 4;
    nt = TT * (TT + 1) / 2;
    groups = min(32, max(1, BSLOTS / nt));
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int s = (int)threadIdx.x + BT * u;
      t[u] = s % nt;
      g[u] = s / nt;
      tile(N, t[u], ta[u], tb[u]);
    }
  }
  static __device__ void tile(int N, int t, int& ta, int& tb) {
    const int TT = (N + 3) / 4;
    ta = 0;
    while (t >= TT - ta) {
      t -= TT - ta;
      ++ta;
    }
    tb = ta + t;
  }
  // vectors of slot u among nvec
  __device__ int rows(int u, int nvec) const {
    return g[u] < groups && nvec > g[u] ? (nvec - g[u] + groups - 1) / groups : 0;
  }
};

template <bool F32P>
struct GramAcc {
  double acc[16];
  float accf[F32P ? 16 : 1];
  int cnt = 0;
  __device__ GramAcc() {
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] = 0.0;
    if constexpr (F32P) {
#pragma unroll
      for (int e = 0; e < 16; ++e) accf[e] = 0.f;
    }
  }
  __device__ void flush() {
    if constexpr (F32P) {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        acc[e] += (double)accf[e];
        accf[e] = 0.f;
      }
      cnt = 0;
    }
  }
  // `rows` vectors of this thread's group, `step` floats apart
  __device__ void add(const float* row, long long step, int rows, int ta, int tb) {
    while (rows > 0) {
      const int k = F32P ? min(rows, 64 - cnt) : rows;
#pragma unroll 2
      for (int i = 0; i < k; ++i, row += step) {
        const float4 av = *reinterpret_cast<const float4*>(row + 4 * ta);
        const float4 bv = *reinterpret_cast<const float4*>(row + 4 * tb);
        const float a[4] = {av.x, av.y, av.z, av.w}, b[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if constexpr (F32P) accf[p * 4 + q] = fmaf(a[p], b[q], accf[p * 4 + q]);
            else acc[p * 4 + q] = fma((double)a[p], (double)b[q], acc[p * 4 + q]);
          }
      }
      rows -= k;
      if constexpr (F32P) {
        cnt += k;
        if (cnt == 64) flush();
      }
    }
  }
};

// Groups' sums to W: as many groups at a time as `stage` (2 BSMALL^2 doubles) holds, entries dealt to the
// threads.  (One group after the other through W, a barrier each, took as long as the products.)
template <bool F32P>
__device__ __forceinline__ void gram_finish(const GramAcc<F32P> (&A)[2], const GramTile& T, int N, double* stage,
                                            double* W) {
  const int tid = threadIdx.x, E = 16 * T.nt, per = 2 * BSMALL * BSMALL / E;
  double v[2] = {0.0, 0.0};  // entries tid and tid + BT (E <= 576)
  for (int g0 = 0; g0 < T.groups; g0 += per) {
    const int ng = min(per, T.groups - g0);
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (T.g[u] >= g0 && T.g[u] < g0 + ng) {
#pragma unroll
        for (int e = 0; e < 16; ++e) stage[(T.g[u] - g0) * E + e * T.nt + T.t[u]] = A[u].acc[e];
      }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (tid + BT * u < E)
        for (int g = 0; g < ng; ++g) v[u] += stage[g * E + tid + BT * u];
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int q = tid + BT * u;
    if (q >= E) continue;
    const int e = q / T.nt, t = q - e * T.nt;
    int ta, tb;
    GramTile::tile(N, t, ta, tb);
    const int i = 4 * ta + (e >> 2), j = 4 * tb + (e & 3);
    if (i < N && j < N && i <= j) {  // upper triangle, mirrored (diagonal tiles hold both halves)
      W[i * N + j] = v[u];
      W[j * N + i] = v[u];
    }
  }
  __syncthreads();
}

// Vectors already in such rows (`vs` floats apart, a multiple of 4), in shared or global memory.
template <bool F32P>
__device__ __noinline__ void cta_gram(const float* base, int vs, int N, int nvec, double* stage, double* W) {
  const GramTile T(N);
  GramAcc<F32P> A[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    A[u].add(base + (long long)T.g[u] * vs, (long long)vs * T.groups, T.rows(u, nvec), T.ta[u], T.tb[u]);
    A[u].flush();
  }
  gram_finish(A, T, N, stage, W);
}

// Component p of vector j at a[p + N j] (COLS: the columns of an N x nvec matrix) or a[j + nvec p] (its
// transpose's), any alignment: brought into rows of shared memory a chunk at a time, every value once and
// coalesced (a tile read straight from global memory takes each value TT + 1 times, one by one).
template <bool COLS>
__device__ __noinline__ void cta_gram_staged(const float* a, int N, long long nvec, float* rows, int cap,
                                             double* stage, double* W) {
  const GramTile T(N);
  GramAcc<true> A[2];
  const int tid = threadIdx.x, S = (N + 3) & ~3;
  const int chunk = cap / S / T.groups * T.groups;  // a whole number of vectors per group
  const float inv_n = 1.0f / (float)N;              // quotients of f < 2^15 by N: exact (error far below 0.5 / N)
  for (long long j0 = 0; j0 < nvec; j0 += chunk) {
    const int nj = (int)min((long long)chunk, nvec - j0);
    __syncthreads();  // the chunk before is consumed
    if (COLS) {
      const float* src = a + j0 * N;
#pragma unroll 4
      for (int f = tid; f < nj * N; f += BT) {
        const int j = (int)(((float)f + 0.5f) * inv_n);
        cp_async4(rows + j * S + (f - j * N), src + f, true);
      }
    } else {
      for (int p = tid >> 5; p < N; p += BT / 32) {
        const float* src = a + j0 + nvec * p;
#pragma unroll 4
        for (int j = tid & 31; j < nj; j += 32) cp_async4(rows + j * S + p, src + j, true);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u)
      A[u].add(rows + T.g[u] * S, (long long)S * T.groups, T.rows(u, nj), T.ta[u], T.tb[u]);
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) A[u].flush();
  gram_finish(A, T, N, stage, W);
}

template <int W>
struct Width {
  static constexpr int value = W;
};

// Calls f(Width<W>{}) with W = n rounded up to a multiple of 8 (n <= BSMALL).  The per-column
// register loops of a step (a rank or sketch width of 2..32) then run over W columns rather than
// all BSMALL with most of them predicated off; columns beyond n are computed on zeros or ignored
// and never stored, so every kept column's FMA sequence is the same whatever W is.
template <class F>
__device__ __forceinline__ void by_width(int n, F&& f) {
  if (n <= 8) f(Width<8>{});
  else if (n <= 16) f(Width<16>{});
  else if (n <= 24) f(Width<24>{});
  else f(Width<32>{});
}

// Largest-|entry| of each of the first r columns of U (entry (i, c) at U[i rs + c cs]) made positive;
// the sign is recorded in sgn[c] (+1/-1) and applied to U; `out` (rows x r, column-major) gets a copy.
__device__ __noinline__ void cta_canon(float* U, int rows, int rs, int cs, int r, float* sgn, float* out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int c = warp; c < r; c += BT / 32) {
    float* u = U + (long long)cs * c;
    float best = 0.f;
    int bi = rows;
    for (int i = lane; i < rows; i += 32) {
      const float v = fabsf(u[(long long)i * rs]);
      if (v > best || (v == best && i < bi)) {
        best = v;
        bi = i;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    const float s = (bi < rows && u[(long long)bi * rs] < 0.f) ? -1.f : 1.f;
    __syncwarp();
    for (int i = lane; i < rows; i += 32) {
      const float v = u[(long long)i * rs] * s;
      u[(long long)i * rs] = v;
      if (out) out[i + (long long)rows * c] = v;
    }
    if (lane == 0) sgn[c] = s;
  }
  __syncthreads();
}

// Rank from eigenvalues (descending) of an unfolding whose energy is `energy`: the smallest r
// (<= cap) whose discarded energy is <= delta2; eps = 0 keeps cap.  Returns r and updates the
// energy carried and the discarded total.
__device__ int pick_rank(const double* lam, int nev, int cap, double delta2, bool adaptive, double energy,
                         double* kept_out, double* tail_out) {
  int r = 0;
  double kept = 0.0;
  if (!adaptive) {
    for (; r < cap; ++r) kept += fmax(lam[r], 0.0);
  } else {
    while (r < cap && (r == 0 || energy - kept > delta2)) kept += fmax(lam[r++], 0.0);
  }
  (void)nev;
  *kept_out = kept;
  *tail_out = fmax(energy - kept, 0.0);
  return r;
}

// The phases of a step, each a call of its own width with its own registers.  4096 tensors of order 4 (8-32 per
// mode, 2.6 GB read, floor 0.41 ms): 13.0 ms.  It is bound by chains, not by memory: 39 % of the time are
// the eigen-solves (8 sweeps of one barrier per round), 15 % the Gram matrices of exact steps, 22 % the products
// with the bases.  The order of every FP32 sum is fixed per tensor, whatever the batch and the schedule.

// A warp's 32 columns (one per lane) of a column-major matrix, eight rows at a time through a tile of shared
// memory: read by the lanes that use them, the values lie a column apart (32 lines per load, and the little L1
// that the shared memory leaves does not hold them until the next row).
constexpr int TILE_LD = 9;                 // odd: a lane's row of the tile in its own bank
constexpr int TILE = 32 * TILE_LD;         // floats per warp
static_assert((BT / 32) * TILE * sizeof(float) <= SM_JAC, "the warps' tiles lie in the eigen-solver's buffer");

// f(i, a_i) for i = 0 .. m - 1 in order, a_i the lane's entry of row i; src: the warp's first column, nj of them.
template <class F>
__device__ __forceinline__ void each_row(const float* src, int m, int nj, float* tile, F&& f) {
  const int lane = threadIdx.x & 31, lr = lane & 7, lc = lane >> 3;
  float next[8];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int c = lc + 4 * u;
      next[u] = i0 + lr < m && c < nj ? src[(long long)m * c + i0 + lr] : 0.f;
    }
  };
  fetch(0);
  for (int i0 = 0; i0 < m; i0 += 8) {
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 8; ++u) tile[(lc + 4 * u) * TILE_LD + lr] = next[u];
    __syncwarp();
    fetch(i0 + 8);
    const float* row = tile + lane * TILE_LD;
    if (i0 + 8 <= m) {
#pragma unroll
      for (int e = 0; e < 8; ++e) f(i0 + e, row[e]);
    } else {
      for (int e = 0; i0 + e < m; ++e) f(i0 + e, row[e]);
    }
  }
  __syncwarp();
}

// Exact step, m <= cols: next = U^T A (r x cols, column-major), U (m x r) column-major (where the tiles go
// afterwards), Ut: m x W scratch.
template <int W>
__device__ __noinline__ void rotate_short(const float* src, int m, long long cols, int r, float* U, float* Ut,
                                          float* dst) {
  const int tid = threadIdx.x, lane = tid & 31, lr = lane & 7, lc = lane >> 3;
  // U row-major (m x W, zero beyond r): a row's columns in W/4 float4 loads
  for (int idx = tid; idx < m * W; idx += BT) {
    const int i = idx / W, c = idx - i * W;
    Ut[idx] = c < r ? U[i + m * c] : 0.f;
  }
  __syncthreads();
  float* const tile = U + (tid >> 5) * TILE;
  for (long long j0 = (tid >> 5) * 32; j0 < cols; j0 += BT) {
    const int nj = (int)min(32LL, cols - j0);
    uint64_t acc2[W / 2];  // columns (2c, 2c+1) as FP32 pairs (fma.rn.f32x2 per pair)
#pragma unroll
    for (int c = 0; c < W / 2; ++c) acc2[c] = 0ull;
    each_row(src + j0 * m, m, nj, tile, [&](int i, float av) {
      const uint64_t av2 = f2_dup(av);
      const ulonglong2* u2 = reinterpret_cast<const ulonglong2*>(Ut + i * W);
#pragma unroll
      for (int c4 = 0; c4 < W / 4; ++c4) {
        const ulonglong2 u = u2[c4];
        ffma2(acc2[2 * c4 + 0], av2, u.x);
        ffma2(acc2[2 * c4 + 1], av2, u.y);
      }
    });
#pragma unroll
    for (int c8 = 0; c8 < W; c8 += 8) {  // out the same way, eight outputs of 32 columns
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        float lo, hi;
        f2_unpack(acc2[(c8 + c) / 2], lo, hi);
        tile[lane * TILE_LD + c] = lo;
        tile[lane * TILE_LD + c + 1] = hi;
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int c = lc + 4 * u;
        if (c8 + lr < r && c < nj) dst[(j0 + c) * r + c8 + lr] = tile[c * TILE_LD + lr];
      }
      __syncwarp();
    }
  }
}

// Exact step, nc = cols <= 32 < m: core U = A V_r / sigma (m x r), Vf: r x W scratch.
template <int W>
__device__ __noinline__ void rotate_tall(const float* src, long long m, int nc, int r, const double* evec,
                                         const float* sig_inv, float* Vf, float* cp) {
  const int tid = threadIdx.x;
  // Vf[c W + q] = V[q][c] in FP32 (zero beyond nc)
  for (int idx = tid; idx < r * W; idx += BT) {
    const int c = idx / W, q = idx - c * W;
    Vf[idx] = q < nc ? (float)evec[q + nc * c] : 0.f;
  }
  __syncthreads();
  for (long long i = tid; i < m; i += BT) {
    float arow[W];
#pragma unroll
    for (int q = 0; q < W; ++q) arow[q] = q < nc ? src[i + m * q] : 0.f;
    for (int c = 0; c < r; ++c) {
      const float4* v4 = reinterpret_cast<const float4*>(Vf + c * W);
      float acc = 0.f;
#pragma unroll
      for (int q4 = 0; q4 < W / 4; ++q4) {
        const float4 v = v4[q4];
        if (4 * q4 + 0 < nc) acc = fmaf(arow[4 * q4 + 0], v.x, acc);
        if (4 * q4 + 1 < nc) acc = fmaf(arow[4 * q4 + 1], v.y, acc);
        if (4 * q4 + 2 < nc) acc = fmaf(arow[4 * q4 + 2], v.z, acc);
        if (4 * q4 + 3 < nc) acc = fmaf(arow[4 * q4 + 3], v.w, acc);
      }
      cp[i + m * c] = acc * sig_inv[c];
    }
  }
}

// Y = A Omega for rows of yq (W + YQ_PAD floats, zero in columns ks..W-1), Omega (cols x ks) N(0,1) from
// Philox: element (j, c) is component j & 3 of call (c * cols4 + (j & ~3)) / 4, cols4 = cols rounded up to a
// multiple of 4.  A thread sums CW columns of one row: all of them, or half (up to BT / 2 rows: a step
// has some 200, and the sum over the columns of A is one chain per entry).
template <int BCH, int W, int CW>
__device__ __noinline__ void sketch_rows(const float* src, int m, long long cols, int ks, unsigned stream,
                                         unsigned long long seed, float* om, float* yq) {
  constexpr int RB = BT / (W / CW);  // rows per pass
  const int tid = threadIdx.x, rt = tid % RB, c0 = tid / RB * CW;
  const long long cols4 = (cols + 3) & ~3LL;
  for (int row0 = 0; row0 < m; row0 += RB) {
    const int row = row0 + rt;
    uint64_t yacc2[CW / 2];  // sketch columns (2c, 2c+1) as FP32 pairs
#pragma unroll
    for (int c = 0; c < CW / 2; ++c) yacc2[c] = 0ull;
    for (long long j0 = 0; j0 < cols; j0 += BCH) {
      const int nj = (int)min((long long)BCH, cols - j0);
      __syncthreads();
      for (int q = tid; q < (BCH / 4) * W; q += BT) {
        const int c = q / (BCH / 4), j4 = 4 * (q % (BCH / 4));
        // columns ks..W-1 of the chunk are zero
        const float4 g = c < ks ? philox_normal4((unsigned long long)((c * cols4 + j0 + j4) >> 2), stream, seed)
                                : make_float4(0.f, 0.f, 0.f, 0.f);
        om[(j4 + 0) * W + c] = g.x;
        om[(j4 + 1) * W + c] = g.y;
        om[(j4 + 2) * W + c] = g.z;
        om[(j4 + 3) * W + c] = g.w;
      }
      __syncthreads();
      if (row < m) {
        const float* a = src + row + m * j0;
#pragma unroll 8
        for (int jj = 0; jj < nj; ++jj) {
          const uint64_t av2 = f2_dup(a[(long long)m * jj]);
          const ulonglong2* o2 = reinterpret_cast<const ulonglong2*>(om + jj * W + c0);
#pragma unroll
          for (int c4 = 0; c4 < CW / 4; ++c4) {
            const ulonglong2 o = o2[c4];
            ffma2(yacc2[2 * c4 + 0], av2, o.x);
            ffma2(yacc2[2 * c4 + 1], av2, o.y);
          }
        }
      }
    }
    if (row < m)
#pragma unroll
      for (int c4 = 0; c4 < CW / 4; ++c4)
        *reinterpret_cast<ulonglong2*>(yq + row * (W + YQ_PAD) + c0 + 4 * c4) =
            make_ulonglong2(yacc2[2 * c4], yacc2[2 * c4 + 1]);
  }
  __syncthreads();
}

// Q = Y R^-1 from the factored Gram matrix Wc (D of its L D L^T on the diagonal).  R in FP32 once:
// rf[k W + c] = W[k][c] / sqrt(W[k][k]) for live rows k < c (0 elsewhere), rf[W W + c] = 1 / sqrt(W[c][c])
// (0: dead column), so the substitution is FMAs only.  Row i: q R = y by forward substitution in registers,
// every later column updated as soon as one is known (a dead column's entry is 0, so it adds nothing).
template <int W>
__device__ __noinline__ void solve_rows(const double* Wc, int ks, double tol, bool any, float* rf, float* yq, int m) {
  const int tid = threadIdx.x;
  for (int idx = tid; idx < W * W + W; idx += BT) {
    const int kk = idx / W, c = idx - kk * W;
    float v = 0.f;
    if (kk < W) {
      const double dk = kk < ks ? Wc[kk * ks + kk] : 0.0;
      if (kk < c && c < ks && dk > tol && any) v = (float)(Wc[kk * ks + c] / sqrt(dk));
    } else if (c < ks) {
      const double dc = Wc[c * (ks + 1)];
      if (dc > tol && any) v = (float)(1.0 / sqrt(dc));
    }
    rf[idx] = v;
  }
  __syncthreads();
  for (int i = tid; i < m; i += BT) {
    float4* yr = reinterpret_cast<float4*>(yq + i * (W + YQ_PAD));
    float y[W];
#pragma unroll
    for (int c4 = 0; c4 < W / 4; ++c4) {
      const float4 v = yr[c4];
      y[4 * c4] = v.x;
      y[4 * c4 + 1] = v.y;
      y[4 * c4 + 2] = v.z;
      y[4 * c4 + 3] = v.w;
    }
#pragma unroll
    for (int c = 0; c < W; ++c) {
      const float dv = rf[W * W + c];
      y[c] = dv == 0.f ? 0.f : y[c] * dv;
#pragma unroll
      for (int c2 = c + 1; c2 < W; ++c2) y[c2] = fmaf(-y[c], rf[c * W + c2], y[c2]);
    }
#pragma unroll
    for (int c4 = 0; c4 < W / 4; ++c4)
      yr[c4] = make_float4(y[4 * c4], y[4 * c4 + 1], y[4 * c4 + 2], y[4 * c4 + 3]);
  }
  __syncthreads();
}

// B = Q^T A: columns of SB floats in Bg, zero past ks.  A thread forms half the rows of one column.
template <int W>
__device__ __noinline__ void project_cols(const float* src, int m, int cols, int SB, const float* yq, float* tiles,
                                          float* Bg) {
  constexpr int CW = W / 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, blocks = (cols + 31) / 32;
  float* const tile = tiles + warp * TILE;
  for (int q = warp; q < 2 * blocks; q += BT / 32) {
    const int h = q >= blocks, j0 = (q - h * blocks) * 32, c0 = h * CW, nj = min(32, cols - j0);
    uint64_t b2[CW / 2];  // rows (c0 + 2c, c0 + 2c+1) of B as FP32 pairs
#pragma unroll
    for (int c = 0; c < CW / 2; ++c) b2[c] = 0ull;
    each_row(src + (long long)j0 * m, m, nj, tile, [&](int i, float av) {
      const uint64_t av2 = f2_dup(av);
      const ulonglong2* q2 = reinterpret_cast<const ulonglong2*>(yq + c0 + i * (W + YQ_PAD));
#pragma unroll
      for (int c4 = 0; c4 < CW / 4; ++c4) {
        const ulonglong2 v = q2[c4];
        ffma2(b2[2 * c4 + 0], av2, v.x);
        ffma2(b2[2 * c4 + 1], av2, v.y);
      }
    });
    if (lane < nj) {
#pragma unroll
      for (int c4 = 0; c4 < CW / 4; ++c4)
        if (c0 + 4 * c4 < SB)
          *reinterpret_cast<ulonglong2*>(Bg + (long long)(j0 + lane) * SB + c0 + 4 * c4) =
              make_ulonglong2(b2[2 * c4], b2[2 * c4 + 1]);
    }
  }
  __syncthreads();
}

// acc[c] over the entries q < ks of a row in registers with column c of E (Ef[c W + q]), in order.
template <int W>
__device__ __forceinline__ float row_dot(const float (&y)[W], const float* e, int ks) {
  const float4* e4 = reinterpret_cast<const float4*>(e);
  float acc = 0.f;
#pragma unroll
  for (int q4 = 0; q4 < W / 4; ++q4) {
    const float4 v = e4[q4];
    if (4 * q4 + 0 < ks) acc = fmaf(y[4 * q4 + 0], v.x, acc);
    if (4 * q4 + 1 < ks) acc = fmaf(y[4 * q4 + 1], v.y, acc);
    if (4 * q4 + 2 < ks) acc = fmaf(y[4 * q4 + 2], v.z, acc);
    if (4 * q4 + 3 < ks) acc = fmaf(y[4 * q4 + 3], v.w, acc);
  }
  return acc;
}

// U = Q E_r over Q, row by row -> canonical signs -> core; next = E_r^T B with the same signs.
template <int W>
__device__ __noinline__ void rotate_sketched(float* yq, int m, long long cols, int ks, int SB, int r,
                                             const double* evec, float* Ef, float* sgn, const float* Bg, float* cp,
                                             float* dst) {
  const int tid = threadIdx.x;
  // E_r in FP32, Ef[c W + q] = E[q][c] (zero beyond ks)
  for (int idx = tid; idx < r * W; idx += BT) {
    const int c = idx / W, q = idx - c * W;
    Ef[idx] = q < ks ? (float)evec[q + ks * c] : 0.f;
  }
  __syncthreads();
  float y[W];
  for (int i = tid; i < m; i += BT) {
    float* yr = yq + i * (W + YQ_PAD);
#pragma unroll
    for (int c4 = 0; c4 < W / 4; ++c4) {
      const float4 v = *reinterpret_cast<const float4*>(yr + 4 * c4);
      y[4 * c4] = v.x;
      y[4 * c4 + 1] = v.y;
      y[4 * c4 + 2] = v.z;
      y[4 * c4 + 3] = v.w;
    }
    for (int c = 0; c < r; ++c) yr[c] = row_dot<W>(y, Ef + c * W, ks);
  }
  __syncthreads();
  cta_canon(yq, m, W + YQ_PAD, 1, r, sgn, cp);
  for (long long j = tid; j < cols; j += BT) {
#pragma unroll
    for (int c4 = 0; c4 < W / 4; ++c4) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (4 * c4 < SB) v = *reinterpret_cast<const float4*>(Bg + j * SB + 4 * c4);
      y[4 * c4] = v.x;
      y[4 * c4 + 1] = v.y;
      y[4 * c4 + 2] = v.z;
      y[4 * c4 + 3] = v.w;
    }
    for (int c = 0; c < r; ++c) dst[j * r + c] = sgn[c] * row_dot<W>(y, Ef + c * W, ks);
  }
}

template <int BCH, int PER_SM>
__global__ void __launch_bounds__(BT, PER_SM)
    k_tt_batched(const BatchShape* __restrict__ shp, const int* __restrict__ order, int count,
                 const float* __restrict__ x,
                 float* __restrict__ cores, int* __restrict__ ranks_out, double* __restrict__ err_out,
                 float* __restrict__ scratch, long long scratch_per_cta, long long half, double eps, int rmax,
                 int oversample, unsigned long long seed, int max_sweeps, int* __restrict__ counter,
                 int yq_floats, DevStatus* st) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Smem S;
  {
    unsigned char* p = smraw;
    S.yq = reinterpret_cast<float*>(p);
    S.yq_floats = yq_floats;
    p += (size_t)yq_floats * sizeof(float);
    S.w = reinterpret_cast<double*>(p);
    p += SM_W;
    S.jac = reinterpret_cast<double*>(p);
    p += SM_JAC;
    S.red = reinterpret_cast<double*>(p);
  }
  float* const om = reinterpret_cast<float*>(S.jac);  // BCH x BSMALL
  __shared__ double lam[BSMALL], evec[BSMALL * BSMALL];
  __shared__ float sgn[BSMALL], sig_inv[BSMALL];
  __shared__ int sh_i[4];
  const int tid = threadIdx.x;
  float* buf0 = scratch + (long long)blockIdx.x * scratch_per_cta;
  float* buf1 = buf0 + half;
  float* Bg = buf1 + half;  // ks x cols of the randomized steps

  for (;;) {
    if (tid == 0) sh_i[0] = atomicAdd(counter, 1);
    __syncthreads();
    const int slot = sh_i[0];
    __syncthreads();
    if (slot >= count) break;
    const int t = order ? order[slot] : slot;
    const BatchShape sh = shp[t];
    const int d = sh.d;
    const float* src = x + sh.x_off;
    float* cp = cores + sh.core_off;
    long long size = sh.size;
    // ||X||^2
    double s2 = 0.0;
#pragma unroll 8
    for (long long i = tid; i < size; i += BT) s2 = fma((double)src[i], (double)src[i], s2);
    const double xn2 = cta_sum(s2, S.red);
    const bool adaptive = eps > 0.0;
    const double delta2 = eps * eps * xn2 / (double)max(d - 1, 1);
    double energy = xn2, tails = 0.0;
    int r_prev = 1;
    if (tid == 0) ranks_out[(long long)t * (BMAXD + 1)] = 1;
    bool fail = false;
    for (int k = 0; k < d - 1 && !fail; ++k) {
      const long long m = (long long)r_prev * sh.n[k];
      const long long cols = size / m;
      const long long small = m < cols ? m : cols;
      const int cap = (int)min((long long)rmax, small);
      float* dst = (k & 1) ? buf0 : buf1;
      const bool exact = small <= BSMALL;
      if (!exact && m > BMAXM) {
        fail = true;
        if (tid == 0 && st) dev_fail(st, TT_ERR_UNSUPPORTED, t);
        break;
      }
      const int N = exact ? (int)small : (int)min((long long)min(cap + oversample, BSMALL), small);
      const int SB = (N + 3) & ~3;  // row stride of B^T
      const int mi = (int)m;        // sketched steps, and exact ones with m <= cols
      if (exact) {
        // ---- exact Gram-eigen step ----
        if (m <= cols) cta_gram_staged<true>(src, N, cols, S.yq, S.yq_floats, S.jac, S.w);  // W = A A^T
        else cta_gram_staged<false>(src, N, m, S.yq, S.yq_floats, S.jac, S.w);              // W = A^T A
      } else {
        // ---- randomized step (EDrSVD) ----
        const int ks = N;
        const int SY = (ks + 7) / 8 * 8 + YQ_PAD;  // row stride of Y, Q, U: an odd number of 16-byte words
        const unsigned stream = (unsigned)(t * BMAXD + k);
        by_width(ks, [&](auto w) {
          constexpr int W = decltype(w)::value;
          if (2 * mi <= BT) sketch_rows<BCH, W, W / 2>(src, mi, cols, ks, stream, seed, om, S.yq);
          else sketch_rows<BCH, W, W>(src, mi, cols, ks, stream, seed, om, S.yq);
        });
        // CholeskyQR2 on Y (rows x ks in shared memory): Gram in FP64, Cholesky, substitution
        for (int pass = 0; pass < 2; ++pass) {
          cta_gram<false>(S.yq, SY, ks, mi, S.jac, S.w);
          double* Wc = S.w;
          double dmax = 0.0;
          for (int i = 0; i < ks; ++i) dmax = fmax(dmax, Wc[i * ks + i]);
          const double tol = 1e-12 * dmax;
          __syncthreads();  // every thread has read the diagonal before the first update changes it
          for (int kk = 0; kk < ks; ++kk) {
            const double dk = Wc[kk * ks + kk];
            if (dk > tol && dmax > 0.0) {
              const double inv = 1.0 / dk;
              const int j = kk + 1 + (tid & 31);
              if (j < ks) {
                const double wkj = Wc[kk * ks + j] * inv;
                for (int i = kk + 1 + (tid >> 5); i <= j; i += BT / 32) Wc[i * ks + j] -= Wc[kk * ks + i] * wkj;
              }
            }
            __syncthreads();
          }
          // R in the eigen-solver's buffer
          by_width(ks, [&](auto w) {
            solve_rows<decltype(w)::value>(Wc, ks, tol, dmax > 0.0, reinterpret_cast<float*>(S.jac), S.yq, mi);
          });
        }
        // B = Q^T A, then W = B B^T
        by_width(ks, [&](auto w) { 
          project_cols<decltype(w)::value>(src, mi, (int)cols, SB, S.yq, reinterpret_cast<float*>(S.jac), Bg);
        });
        cta_gram<true>(Bg, SB, ks, (int)cols, S.jac, S.w);  // W = B B^T (vectors = columns of B)
      }
      const int sw = bl_solve<32>(S.w, N, lam, evec, max_sweeps, S.jac);
      if (tid == 0 && st) {
        atomicMax(&st->sweeps, sw);
        if (sw > max_sweeps) dev_fail(st, TT_ERR_NOCONV, t);
      }
      double kept, tail, full = energy;
      if (exact && adaptive) {
        full = 0.0;
        for (int i = 0; i < N; ++i) full += fmax(lam[i], 0.0);
      }
      const int r = pick_rank(lam, N, min(cap, N), delta2, adaptive, full, &kept, &tail);
      tails += tail;
      energy = kept;
      if (!exact) {
        by_width(N, [&](auto w) {
          rotate_sketched<decltype(w)::value>(S.yq, mi, cols, N, SB, r, evec, reinterpret_cast<float*>(S.jac), sgn, Bg,
                                              cp, dst);
        });
      } else if (m <= cols) {
        // U = E_r (m x r): canonical signs, core, next = U^T A (r x cols, column-major)
        float* U = reinterpret_cast<float*>(S.jac);  // m x r
        for (int idx = tid; idx < mi * r; idx += BT) U[idx] = (float)evec[idx];
        __syncthreads();
        cta_canon(U, mi, 1, mi, r, sgn, cp);
        by_width(r, [&](auto w) { rotate_short<decltype(w)::value>(src, mi, cols, r, U, S.yq, dst); });
      } else {
        // cols <= 32 < m: V (cols x cols), U = A V_r / sigma (m x r), next = sigma V_r^T
        for (int c = tid; c < r; c += BT) sig_inv[c] = lam[c] > 0.0 ? (float)(1.0 / sqrt(lam[c])) : 0.f;
        by_width(N, [&](auto w) {
          rotate_tall<decltype(w)::value>(src, m, N, r, evec, sig_inv, reinterpret_cast<float*>(S.jac), cp);
        });
        __syncthreads();
        // canonical signs on the core columns (global memory), mirrored on the rows of sigma V^T
        cta_canon(cp, (int)m, 1, (int)m, r, sgn, nullptr);
        for (int idx = tid; idx < r * N; idx += BT) {
          const int c = idx % r, q = idx / r;  // dst column-major r x cols: dst[c + r q]
          dst[idx] = sgn[c] * (float)(sqrt(fmax(lam[c], 0.0)) * evec[q + N * c]);
        }
      }
      __syncthreads();
      cp += m * r;
      src = dst;
      size = (long long)r * cols;
      r_prev = r;
      if (tid == 0) ranks_out[(long long)t * (BMAXD + 1) + k + 1] = r;
    }
    if (!fail) {
      // last core = the remaining data (r_{d-1}, n_d, 1)
      for (long long i = tid; i < size; i += BT) cp[i] = src[i];
      if (tid == 0) {
        ranks_out[(long long)t * (BMAXD + 1) + d] = 1;
        err_out[t] = xn2 > 0.0 ? sqrt(tails / xn2) : 0.0;
      }
    }
    __syncthreads();
  }
}

// Shape table of a batch: validation and the per-CTA scratch the kernel needs.
struct BatchLayout {
  std::vector<BatchShape> hs;
  long long half = 0, per_cta = 0;
  int mrows = 0;  // rows of the tallest sketched step
};

int batch_layout(int count, int d, const int* n, const long long* x_off, const long long* core_off, int rmax,
                 BatchLayout& L) {
  L.hs.assign((size_t)count, BatchShape{});
  long long maxdata = 0, maxbg = 0;
  for (int t = 0; t < count; ++t) {
    BatchShape& b = L.hs[(size_t)t];
    b.d = d;
    b.size = 1;
    for (int k = 0; k < BMAXD; ++k) b.n[k] = k < d ? n[(size_t)t * d + k] : 1;
    for (int k = 0; k < d; ++k) {
      if (b.n[k] < 1) {
        set_error(TT_ERR_SHAPE, "batched: tensor %d mode %d size %d", t, k, b.n[k]);
        return TT_ERR_SHAPE;
      }
      b.size *= b.n[k];
    }
    b.x_off = x_off[t];
    b.core_off = core_off[t];
    // randomized steps keep B (ks x cols) and need rows <= BMAXM
    long long rp = 1, sz = b.size;
    for (int k = 0; k < d - 1; ++k) {
      const long long m = rp * b.n[k], cols = sz / m, small = std::min(m, cols);
      if (small > BSMALL) {
        if (m > BMAXM) {
          set_error(TT_ERR_UNSUPPORTED, "batched: tensor %d step %d has %lld rows (> %d) on a sketched step", t, k, m,
                    BMAXM);
          return TT_ERR_UNSUPPORTED;
        }
        maxbg = std::max(maxbg, (long long)BSMALL * cols);
        L.mrows = std::max(L.mrows, (int)m);
      }
      const long long rn = std::min<long long>((long long)rmax, small);
      sz = rn * cols;
      rp = rn;
      maxdata = std::max(maxdata, sz);  // what a step leaves for the next one
    }
  }
  L.half = (maxdata + 63) & ~63LL;
  L.per_cta = 2 * L.half + ((maxbg + 63) & ~63LL);
  return TT_OK;
}

int check_batch_args(int count, int d, int rmax, double eps, int oversample) {
  if (count < 0 || d < 2 || d > BMAXD || rmax < 1 || rmax > BSMALL || !(eps >= 0.0) || oversample < 0) {
    set_error(TT_ERR_SHAPE, "batched: count %d, order %d (2..%d), rmax %d (1..%d), eps %g, oversample %d", count, d,
              BMAXD, rmax, BSMALL, eps, oversample);
    return TT_ERR_SHAPE;
  }
  return TT_OK;
}

template <int BCH>
int set_smem_attr() {
  TT_TRY((smem_optin_k(k_tt_batched<BCH, 1>, sm_total(BMAXM))));
  return smem_optin_k(k_tt_batched<BCH, 2>, sm_total(BMAXM));
}

struct BatchArgs {
  const BatchShape* shp;
  const int* order;
  int count;
  const float* x;
  float* cores;
  int* ranks;
  double* err;
  float* scratch;
  long long per_cta, half;
  double eps;
  int rmax, oversample;
  unsigned long long seed;
  int* counter;
  int mrows;
  DevStatus* st;
};

template <int BCH>
int launch_bch(int grid, cudaStream_t s, const BatchArgs& a) {
  TT_TRY(set_smem_attr<BCH>());
  // Alone on its SM a CTA may have 168 registers a thread instead of 80: a round of the eigen-solver is shorter
  // and the Gram matrices do not spill (69 tensors of order 3: 326 us, 410 at 80 registers).
  auto* kernel = grid <= dev_sms() ? k_tt_batched<BCH, 1> : k_tt_batched<BCH, 2>;
  kernel<<<grid, BT, sm_total(a.mrows), s>>>(a.shp, a.order, a.count, a.x, a.cores, a.ranks, a.err, a.scratch,
                                             a.per_cta, a.half, a.eps, a.rmax, a.oversample, a.seed, 40, a.counter,
                                             (int)(sm_yq(a.mrows) / sizeof(float)), a.st);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

int launch_batched(int bch, int grid, cudaStream_t s, const BatchArgs& a) {
  switch (bch) {
    case 16: return launch_bch<16>(grid, s, a);
    case 32: return launch_bch<32>(grid, s, a);
    case 64: return launch_bch<64>(grid, s, a);
    default:
      set_error(TT_ERR_ARG, "batched: chunk width %d", bch);
      return TT_ERR_ARG;
  }
}

// CTAs of a batch, `per_sm` (1 or 2) to an SM.  Up to kOneWave tensors per SM one is better: the batch is then
// about as long as its slowest tensors, and those run faster alone.  One against two, us: order 4 of 8-32 per mode,
// 310 tensors 1168 / 1708, 440 1542 / 1740, 580 1933 / 1848; of 12-20, 200 tensors 566 / 645, 310 821 / 775, 440 994 /
// 994, 580 1284 / 1119; order 3 of 20-28, 440 728 / 702, 580 925 / 773.
constexpr int kOneWave = 3;
int best_per_sm(int count) { return count <= kOneWave * dev_sms() ? 1 : 2; }
int persistent_grid(int count, int per_sm) { return std::max(1, std::min(count, per_sm * dev_sms())); }

}  // namespace
}  // namespace ttr

using namespace ttr;

extern "C" long long tt_batch_core_capacity(int d, const int* n, int rmax) {
  if (d < 2 || d > BMAXD || !n || rmax < 1) return -1;
  long long total = 0, left = 1, right = 1;
  for (int k = 0; k < d; ++k) right *= n[k];
  long long rp = 1;
  for (int k = 0; k < d; ++k) {
    left *= n[k];
    right /= n[k];
    const long long rn = (k == d - 1) ? 1 : std::min<long long>({(long long)rmax, left, right});
    total += rp * n[k] * rn;
    rp = rn;
  }
  return total;
}

extern "C" int tt_svd_batched(tt_ctx* ctx, int count, int d, const int* n, const float* x,
                              const long long* x_off, double eps, int rmax, int oversample,
                              unsigned long long seed, float* cores, const long long* core_off, int* ranks,
                              double* err_est) {
  if (!ctx || !n || !x || !x_off || !cores || !core_off || !ranks || count < 0) {
    set_error(TT_ERR_ARG, "null argument");
    return TT_ERR_ARG;
  }
  TT_TRY(check_batch_args(count, d, rmax, eps, oversample));
  if (count == 0) return TT_OK;
  BatchLayout L;
  TT_TRY(batch_layout(count, d, n, x_off, core_off, rmax, L));
  // two CTAs per SM where that is better; one where the scratch of two does not fit
  int grid = 0, rc = TT_OK;
  Arena ws;
  for (int per_sm = best_per_sm(count); per_sm >= 1; --per_sm) {
    grid = persistent_grid(count, per_sm);
    const size_t bytes = sizeof(BatchShape) * (size_t)count + sizeof(int) * (size_t)count * (BMAXD + 1) +
                         sizeof(double) * (size_t)count + sizeof(float) * (size_t)L.per_cta * grid + 4096;
    rc = ctx_arena(ctx, bytes, &ws);
    if (rc != TT_ERR_NOMEM) break;
  }
  TT_TRY(rc);
  BatchShape* dshp = ws.take<BatchShape>((size_t)count);
  int* dranks = ws.take<int>((size_t)count * (BMAXD + 1));
  double* derr = ws.take<double>((size_t)count);
  int* dcounter = ws.take<int>(1);
  float* scratch = ws.take<float>((size_t)L.per_cta * grid);
  if (!dshp || !dranks || !derr || !dcounter || !scratch) {
    set_error(TT_ERR_NOMEM, "batched workspace");
    return TT_ERR_NOMEM;
  }
  cudaStream_t s = ctx_stream(ctx);
  DevStatus* dst = ctx_status(ctx);
  TT_CUDA(cudaMemsetAsync(dst, 0, sizeof(DevStatus), s));
  TT_CUDA(cudaMemcpyAsync(dshp, L.hs.data(), sizeof(BatchShape) * (size_t)count, cudaMemcpyHostToDevice, s));
  TT_CUDA(cudaMemsetAsync(dcounter, 0, sizeof(int), s));
  const BatchArgs args{dshp, nullptr, count, x, cores, dranks, derr, scratch, L.per_cta, L.half,
                       eps, rmax, oversample, seed, dcounter, L.mrows, dst};
  TT_TRY(launch_batched(32, grid, s, args));
  std::vector<int> hr((size_t)count * (BMAXD + 1));
  TT_CUDA(cudaMemcpyAsync(hr.data(), dranks, sizeof(int) * hr.size(), cudaMemcpyDeviceToHost, s));
  if (err_est) TT_CUDA(cudaMemcpyAsync(err_est, derr, sizeof(double) * (size_t)count, cudaMemcpyDeviceToHost, s));
  DevStatus hst;
  TT_CUDA(cudaMemcpyAsync(&hst, dst, sizeof(hst), cudaMemcpyDeviceToHost, s));
  TT_CUDA(cudaStreamSynchronize(s));
  for (int t = 0; t < count; ++t)
    for (int k = 0; k <= d; ++k) ranks[(size_t)t * (d + 1) + k] = hr[(size_t)t * (BMAXD + 1) + k];
  if (hst.code) {
    set_error(hst.code, "batched: device status %d (tensor %d)", hst.code, hst.detail);
    return hst.code;
  }
  return TT_OK;
}

// ---------------------------------------------------------------------------------------
// Batch plans: the batch's shape table, work orders and scratch allocated once, a variant
// (chunk width x work order) picked by timing every candidate on the batch, and the launch
// sequence (status reset, counter reset, persistent kernel, result read-back) captured in a
// CUDA graph that every later run replays with one cudaGraphLaunch.
// ---------------------------------------------------------------------------------------
struct tt_batch_plan {
  tt_ctx* ctx = nullptr;
  int count = 0, d = 0, rmax = 0, oversample = 0, grid = 1;
  double eps = 0.0;
  unsigned long long seed = 0;
  long long per_cta = 0, half = 0;
  int mrows = 0;
  char* dmem = nullptr;
  BatchShape* dshp = nullptr;
  int* dorder = nullptr;  // largest-first order
  int* dranks = nullptr;
  double* derr = nullptr;
  int* dcounter = nullptr;
  DevStatus* dst = nullptr;
  float* scratch = nullptr;
  int* hranks = nullptr;  // pinned
  double* herr = nullptr;
  DevStatus* hst = nullptr;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev_in = nullptr, e0 = nullptr, e1 = nullptr;
  int bch = 32, sched = SCHED_LARGEST_FIRST;
  float tune_ms[6] = {0, 0, 0, 0, 0, 0};
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  const float* gx = nullptr;
  float* gcores = nullptr;
  int gbch = 0, gsched = -1;
};

namespace {
BatchArgs plan_args(tt_batch_plan* p, const float* x, float* cores, int sched) {
  return BatchArgs{p->dshp, sched == SCHED_LARGEST_FIRST ? p->dorder : nullptr, p->count, x, cores, p->dranks,
                   p->derr, p->scratch, p->per_cta, p->half, p->eps, p->rmax, p->oversample, p->seed, p->dcounter,
                   p->mrows, p->dst};
}

// The launch sequence of one run, on the plan's stream (also what the graph records).
int plan_enqueue(tt_batch_plan* p, const float* x, float* cores, int bch, int sched, bool readback) {
  cudaStream_t s = p->stream;
  TT_CUDA(cudaMemsetAsync(p->dst, 0, sizeof(DevStatus), s));
  TT_CUDA(cudaMemsetAsync(p->dcounter, 0, sizeof(int), s));
  TT_TRY(launch_batched(bch, p->grid, s, plan_args(p, x, cores, sched)));
  if (readback) {
    TT_CUDA(cudaMemcpyAsync(p->hranks, p->dranks, sizeof(int) * (size_t)p->count * (BMAXD + 1),
                            cudaMemcpyDeviceToHost, s));
    TT_CUDA(cudaMemcpyAsync(p->herr, p->derr, sizeof(double) * (size_t)p->count, cudaMemcpyDeviceToHost, s));
    TT_CUDA(cudaMemcpyAsync(p->hst, p->dst, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
  }
  return TT_OK;
}

void plan_drop_graph(tt_batch_plan* p) {
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  p->exec = nullptr;
  p->graph = nullptr;
  p->gx = nullptr;
  p->gcores = nullptr;
  p->gsched = -1;
}

int plan_capture(tt_batch_plan* p, const float* x, float* cores) {
  plan_drop_graph(p);
  TT_TRY(set_smem_attr<16>());
  TT_TRY(set_smem_attr<32>());
  TT_TRY(set_smem_attr<64>());
  TT_CUDA(cudaStreamBeginCapture(p->stream, cudaStreamCaptureModeThreadLocal));
  const int rc = plan_enqueue(p, x, cores, p->bch, p->sched, true);
  cudaGraph_t g = nullptr;
  const cudaError_t ec = cudaStreamEndCapture(p->stream, &g);
  if (rc != TT_OK) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (ec != cudaSuccess || !g) {
    set_error(TT_ERR_CUDA, "batched: graph capture: %s", cudaGetErrorString(ec));
    return TT_ERR_CUDA;
  }
  p->graph = g;
  if (cudaGraphInstantiate(&p->exec, g, 0) != cudaSuccess) {
    p->exec = nullptr;
    plan_drop_graph(p);
    set_error(TT_ERR_CUDA, "batched: graph instantiation");
    return TT_ERR_CUDA;
  }
  p->gx = x;
  p->gcores = cores;
  p->gbch = p->bch;
  p->gsched = p->sched;
  return TT_OK;
}
}  // namespace

extern "C" int tt_batch_plan_destroy(tt_batch_plan* p) {
  if (!p) return TT_OK;
  if (p->stream) cudaStreamSynchronize(p->stream);
  plan_drop_graph(p);
  if (p->dmem) cudaFree(p->dmem);
  if (p->hranks) cudaFreeHost(p->hranks);
  if (p->herr) cudaFreeHost(p->herr);
  if (p->hst) cudaFreeHost(p->hst);
  if (p->ev_in) cudaEventDestroy(p->ev_in);
  if (p->e0) cudaEventDestroy(p->e0);
  if (p->e1) cudaEventDestroy(p->e1);
  if (p->stream) cudaStreamDestroy(p->stream);
  delete p;
  return TT_OK;
}

extern "C" int tt_batch_plan_create(tt_ctx* ctx, int count, int d, const int* n, const long long* x_off, double eps,
                                    int rmax, int oversample, unsigned long long seed, const long long* core_off,
                                    tt_batch_plan** out) {
  if (!ctx || !n || !x_off || !core_off || !out || count < 1) {
    set_error(TT_ERR_ARG, "batch plan: null argument or empty batch");
    return TT_ERR_ARG;
  }
  *out = nullptr;
  TT_TRY(check_batch_args(count, d, rmax, eps, oversample));
  BatchLayout L;
  TT_TRY(batch_layout(count, d, n, x_off, core_off, rmax, L));
  tt_batch_plan* p = new tt_batch_plan();
  p->ctx = ctx;
  p->count = count;
  p->d = d;
  p->rmax = rmax;
  p->oversample = oversample;
  p->eps = eps;
  p->seed = seed;
  p->per_cta = L.per_cta;
  p->half = L.half;
  p->mrows = L.mrows;
  size_t off = 0;
  auto carve = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 255) & ~size_t(255);
    return o;
  };
  const size_t o_shp = carve(sizeof(BatchShape) * (size_t)count);
  const size_t o_ord = carve(sizeof(int) * (size_t)count);
  const size_t o_rk = carve(sizeof(int) * (size_t)count * (BMAXD + 1));
  const size_t o_err = carve(sizeof(double) * (size_t)count);
  const size_t o_cnt = carve(sizeof(int));
  const size_t o_st = carve(sizeof(DevStatus));
  const size_t o_scr = off;
  cudaError_t mem = cudaErrorMemoryAllocation;
  for (int per_sm = best_per_sm(count); per_sm >= 1 && mem != cudaSuccess; --per_sm) {  // one per SM where two do not fit
    p->grid = persistent_grid(count, per_sm);
    mem = cudaMalloc(&p->dmem, o_scr + sizeof(float) * (size_t)L.per_cta * p->grid);
    if (mem != cudaSuccess) {
      p->dmem = nullptr;
      (void)cudaGetLastError();  // reported below
    }
  }
  if (mem != cudaSuccess ||
      cudaMallocHost(&p->hranks, sizeof(int) * (size_t)count * (BMAXD + 1)) != cudaSuccess ||
      cudaMallocHost(&p->herr, sizeof(double) * (size_t)count) != cudaSuccess ||
      cudaMallocHost(&p->hst, sizeof(DevStatus)) != cudaSuccess ||
      cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&p->ev_in, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreate(&p->e0) != cudaSuccess || cudaEventCreate(&p->e1) != cudaSuccess) {
    tt_batch_plan_destroy(p);
    set_error(TT_ERR_NOMEM, "batch plan allocation");
    return TT_ERR_NOMEM;
  }
  p->dshp = reinterpret_cast<BatchShape*>(p->dmem + o_shp);
  p->dorder = reinterpret_cast<int*>(p->dmem + o_ord);
  p->dranks = reinterpret_cast<int*>(p->dmem + o_rk);
  p->derr = reinterpret_cast<double*>(p->dmem + o_err);
  p->dcounter = reinterpret_cast<int*>(p->dmem + o_cnt);
  p->dst = reinterpret_cast<DevStatus*>(p->dmem + o_st);
  p->scratch = reinterpret_cast<float*>(p->dmem + o_scr);
  // largest-first order: the longest tensors start first, so the work counter's tail holds
  // only small ones (longest-processing-time rule for the SM makespan)
  std::vector<int> ord((size_t)count);
  for (int t = 0; t < count; ++t) ord[(size_t)t] = t;
  std::stable_sort(ord.begin(), ord.end(),
                   [&](int a, int b) { return L.hs[(size_t)a].size > L.hs[(size_t)b].size; });
  if (cudaMemcpyAsync(p->dshp, L.hs.data(), sizeof(BatchShape) * (size_t)count, cudaMemcpyHostToDevice, p->stream) !=
          cudaSuccess ||
      cudaMemcpyAsync(p->dorder, ord.data(), sizeof(int) * (size_t)count, cudaMemcpyHostToDevice, p->stream) !=
          cudaSuccess ||
      cudaStreamSynchronize(p->stream) != cudaSuccess) {
    tt_batch_plan_destroy(p);
    set_error(TT_ERR_CUDA, "batch plan upload");
    return TT_ERR_CUDA;
  }
  *out = p;
  return TT_OK;
}

extern "C" int tt_batch_plan_tune(tt_batch_plan* p, const float* x, float* cores, int reps, float* ms_out) {
  if (!p || !x || !cores) {
    set_error(TT_ERR_ARG, "batch plan tune: null argument");
    return TT_ERR_ARG;
  }
  reps = std::max(1, reps);
  TT_CUDA(cudaEventRecord(p->ev_in, ctx_stream(p->ctx)));
  TT_CUDA(cudaStreamWaitEvent(p->stream, p->ev_in, 0));
  float best = 0.f;
  int vi = 0;
  for (int sched = 0; sched < 2; ++sched)
    for (int c = 0; c < 3; ++c, ++vi) {
      TT_TRY(plan_enqueue(p, x, cores, kChunks[c], sched, false));  // warm-up
      TT_CUDA(cudaEventRecord(p->e0, p->stream));
      for (int r = 0; r < reps; ++r) TT_TRY(plan_enqueue(p, x, cores, kChunks[c], sched, false));
      TT_CUDA(cudaEventRecord(p->e1, p->stream));
      TT_CUDA(cudaEventSynchronize(p->e1));
      float ms = 0.f;
      TT_CUDA(cudaEventElapsedTime(&ms, p->e0, p->e1));
      ms /= (float)reps;
      p->tune_ms[vi] = ms;
      if (vi == 0 || ms < best) {
        best = ms;
        p->bch = kChunks[c];
        p->sched = sched;
      }
    }
  DevStatus h;
  TT_CUDA(cudaMemcpyAsync(&h, p->dst, sizeof(h), cudaMemcpyDeviceToHost, p->stream));
  TT_CUDA(cudaStreamSynchronize(p->stream));
  if (h.code) {
    set_error(h.code, "batched: device status %d (tensor %d)", h.code, h.detail);
    return h.code;
  }
  if (ms_out)
    for (int i = 0; i < 6; ++i) ms_out[i] = p->tune_ms[i];
  return TT_OK;
}

extern "C" int tt_batch_plan_variant(const tt_batch_plan* p, int* chunk, int* largest_first) {
  if (!p) {
    set_error(TT_ERR_ARG, "batch plan: null");
    return TT_ERR_ARG;
  }
  if (chunk) *chunk = p->bch;
  if (largest_first) *largest_first = p->sched == SCHED_LARGEST_FIRST;
  return TT_OK;
}

extern "C" int tt_batch_plan_run(tt_batch_plan* p, const float* x, float* cores, int* ranks, double* err_est) {
  if (!p || !x || !cores) {
    set_error(TT_ERR_ARG, "batch plan run: null argument");
    return TT_ERR_ARG;
  }
  if (!p->exec || p->gx != x || p->gcores != cores || p->gbch != p->bch || p->gsched != p->sched)
    TT_TRY(plan_capture(p, x, cores));
  TT_CUDA(cudaEventRecord(p->ev_in, ctx_stream(p->ctx)));
  TT_CUDA(cudaStreamWaitEvent(p->stream, p->ev_in, 0));
  TT_CUDA(cudaGraphLaunch(p->exec, p->stream));
  count_launch();
  TT_CUDA(cudaStreamSynchronize(p->stream));
  if (ranks)
    for (int t = 0; t < p->count; ++t)
      for (int k = 0; k <= p->d; ++k)
        ranks[(size_t)t * (p->d + 1) + k] = p->hranks[(size_t)t * (BMAXD + 1) + k];
  if (err_est) memcpy(err_est, p->herr, sizeof(double) * (size_t)p->count);
  if (p->hst->code) {
    set_error(p->hst->code, "batched: device status %d (tensor %d)", p->hst->code, p->hst->detail);
    return p->hst->code;
  }
  return TT_OK;
}
