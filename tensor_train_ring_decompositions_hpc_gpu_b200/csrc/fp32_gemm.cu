// The plain-FP32 GEMM engine (CUDA cores): sketch Y = A W, projection out = A^T Q, and the projection of
// short columns (the rotation of a small factor).  A is a column-major m x n unfolding, W / Q are narrow.
// Replaces the GemmEx calls of TT3O:601-708.
//
// Bound by the FP32 FMAs from about 24 output columns on (128 per clock and SM, issued as pairs by
// fma.rn.f32x2), by HBM below.  Hence wide tiles per thread (at 8 x 4 or 8 x 5, loads and operand copies take as
// many issue slots as the FMAs: 35-49 % of their rate) and row tiles of 64, which hang little over the end of an
// unfolding.  576 x 331776 at 32 columns (floor 164 us of FMAs): sketch 328 us, projection 330.  Sketches of
// 600 x 950k: 565 us at 16 columns, 2480 at 96 (59 % of the FMA rate).  384 x 320: 6 us each.
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"

namespace ttr {
namespace {

// ---------------------------------------------------------------------------------------
// sketch
// ---------------------------------------------------------------------------------------
// A block owns 64 rows of A and NT = 4 RC columns of W; its 8 warps take every eighth chunk of 8 columns
// of A, each through a 4-deep cp.async ring of its own (no barrier until the end), so the running FP32
// sums are an eighth as long as the block's range.  A lane holds 8 rows x RC columns: pairs of columns
// with A's values duplicated (RC >= 8), or pairs of rows with W's (fewer copies for narrow sketches).
// The warps' sums are added in FP64.
constexpr int SK_ROWS = 64, SK_JC = 8, SK_ST = 4, SK_W = 8;
constexpr int sk_ws(int NT) { return NT + 4; }  // row stride of W's chunk: an odd number of 16-byte words
constexpr int sk_slot(int NT) { return SK_JC * (SK_ROWS + sk_ws(NT)); }
constexpr size_t sk_smem(int NT) {
  const size_t ring = (size_t)SK_W * SK_ST * sk_slot(NT) * sizeof(float);
  const size_t red = (size_t)SK_W * NT * (SK_ROWS + 4) * sizeof(float);
  return ring > red ? ring : red;
}
constexpr int sk_blocks(int NT) { return NT <= 32 ? 2 : 1; }  // per SM

template <int RC>
__global__ void __launch_bounds__(32 * SK_W, RC <= 8 ? 2 : 1)
    k_sketch32(const float* __restrict__ a, long long m, long long n, const float* __restrict__ w, int N,
               long long wj, long long wc, long long jchunk, double* __restrict__ part) {
  constexpr int NT = 4 * RC, WS = sk_ws(NT), SLOT = sk_slot(NT);
  constexpr bool DUPA = RC >= 8;
  constexpr int P0 = DUPA ? 8 : 4, P1 = DUPA ? RC / 2 : RC;  // accumulator pairs: rows x column pairs, or row pairs x columns
  extern __shared__ __align__(16) float sm_sk[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane & 7, cg = lane >> 3;
  float* const ring = sm_sk + (size_t)warp * SK_ST * SLOT;
  const long long i0 = (long long)blockIdx.x * SK_ROWS;
  const int c0 = blockIdx.z * NT;
  const long long jb = blockIdx.y * jchunk, je = min(jb + jchunk, n);
  const long long nch = je > jb ? (je - jb + SK_JC - 1) / SK_JC : 0;
  const int my = warp < nch ? (int)((nch - 1 - warp) / SK_W + 1) : 0;
  const bool vec = (m & 3) == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
  // this lane's part of a chunk: rows 4 (lane & 15).. of columns lane / 16 + 2 u; W rows lane & 7
  const int li = 4 * (lane & 15), lj = lane >> 4;
  const bool inr = i0 + li < m;  // vec: m % 4 == 0, so four rows or none
  auto load = [&](int k) {
    if (k < my) {
      const long long j0 = jb + (warp + (long long)SK_W * k) * SK_JC;
      const int nj = (int)min((long long)SK_JC, je - j0);
      float* const as = ring + (k % SK_ST) * SLOT;
      float* const ws = as + SK_JC * SK_ROWS;
      const float* src = a + (j0 + lj) * m + i0 + li;
#pragma unroll
      for (int u = 0; u < SK_JC / 2; ++u) {
        const int jj = lj + 2 * u;
        float* dst = as + jj * SK_ROWS + li;
        if (vec) {
          const bool ok = inr && jj < nj;
          cp_async16z(dst, ok ? src + 2 * u * m : a, ok);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const bool ok = jj < nj && i0 + li + e < m;
            cp_async4(dst + e, ok ? src + 2 * u * m + e : a, ok);
          }
        }
      }
      const int jw = lane & 7, cw = lane >> 3;
      const float* wsrc = w + (j0 + jw) * wj + (c0 + cw) * wc;
#pragma unroll
      for (int u = 0; u < RC; ++u) {
        const bool ok = jw < nj && c0 + cw + 4 * u < N;
        cp_async4(ws + jw * WS + cw + 4 * u, ok ? wsrc + 4 * u * wc : w, ok);
      }
    }
    cp_async_commit();
  };
  uint64_t acc[P0][P1];
#pragma unroll
  for (int p = 0; p < P0; ++p)
#pragma unroll
    for (int q = 0; q < P1; ++q) acc[p][q] = 0ull;
#pragma unroll
  for (int s = 0; s < SK_ST - 1; ++s) load(s);
  for (int k = 0; k < my; ++k) {
    cp_async_wait<SK_ST - 2>();
    __syncwarp();  // chunk k landed for every lane; the chunk before it is consumed
    load(k + SK_ST - 1);
    const float* as = ring + (k % SK_ST) * SLOT;
    const float* ws = as + SK_JC * SK_ROWS;
#pragma unroll
    for (int jj = 0; jj < SK_JC; ++jj) {
      // rows 4 rg .. 4 rg + 3 and 32 + 4 rg ..; column pairs cg + 4 q (columns 2 (cg + 4 q) and the next)
      const float* ar = as + jj * SK_ROWS + 4 * rg;
      const float* wr = ws + jj * WS;
      if constexpr (DUPA) {
        const float4 x0 = *reinterpret_cast<const float4*>(ar);
        const float4 x1 = *reinterpret_cast<const float4*>(ar + 32);
        const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
        uint64_t wp[P1];
#pragma unroll
        for (int q = 0; q < P1; ++q) wp[q] = *reinterpret_cast<const uint64_t*>(wr + 2 * (cg + 4 * q));
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          const uint64_t xd = f2_dup(x[p]);
#pragma unroll
          for (int q = 0; q < P1; ++q) ffma2(acc[p][q], xd, wp[q]);
        }
      } else {
        const ulonglong2 x0 = *reinterpret_cast<const ulonglong2*>(ar);
        const ulonglong2 x1 = *reinterpret_cast<const ulonglong2*>(ar + 32);
        const uint64_t xp[4] = {x0.x, x0.y, x1.x, x1.y};
#pragma unroll
        for (int q = 0; q < P1; ++q) {
          const uint64_t wd = f2_dup(wr[2 * (cg + 4 * (q / 2)) + (q & 1)]);
#pragma unroll
          for (int p = 0; p < 4; ++p) ffma2(acc[p][q], xp[p], wd);
        }
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();  // rings free: they take the warps' sums, column-major, rows padded to 68
  constexpr int RS = SK_ROWS + 4;
  float* const red = sm_sk + (size_t)warp * NT * RS;
#pragma unroll
  for (int q = 0; q < RC; ++q) {
    float v[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      float lo, hi;
      if (DUPA) {
        f2_unpack(acc[p % P0][(q / 2) % P1], lo, hi);
        v[p] = (q & 1) ? hi : lo;
      } else {
        f2_unpack(acc[(p / 2) % P0][q % P1], lo, hi);
        v[p] = (p & 1) ? hi : lo;
      }
    }
    float* dst = red + (2 * (cg + 4 * (q / 2)) + (q & 1)) * RS + 4 * rg;
    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(dst + 32) = make_float4(v[4], v[5], v[6], v[7]);
  }
  __syncthreads();
  for (int f = threadIdx.x; f < NT * SK_ROWS; f += 32 * SK_W) {
    const int c = f / SK_ROWS, i = f % SK_ROWS;
    if (i0 + i >= m || c0 + c >= N) continue;
    double sum = 0.0;
#pragma unroll
    for (int v = 0; v < SK_W; ++v) sum += (double)sm_sk[((size_t)v * NT + c) * RS + i];
    part[((long long)blockIdx.y * N + c0 + c) * m + i0 + i] = sum;
  }
}

// Sum of nsplit partial blocks: each 256-thread block owns 32 consecutive outputs, its 8 warps
// read interleaved splits (coalesced 256-byte rows, several loads in flight per lane) and the
// 8 warp sums are added in a fixed order, so the result does not depend on scheduling.
__global__ void __launch_bounds__(256) k_reduce_splits(const double* __restrict__ part, long long count,
                                                       int nsplit, double* __restrict__ y) {
  __shared__ double red[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long base = (long long)blockIdx.x * 32; base < count; base += (long long)gridDim.x * 32) {
    const long long idx = base + lane;
    double s0 = 0.0, s1 = 0.0;
    if (idx < count) {
      int k = warp;
#pragma unroll 4
      for (; k + 8 < nsplit; k += 16) {
        s0 += part[(long long)k * count + idx];
        s1 += part[(long long)(k + 8) * count + idx];
      }
      if (k < nsplit) s0 += part[(long long)k * count + idx];
    }
    red[warp][lane] = s0 + s1;
    __syncthreads();
    if (warp == 0 && idx < count) {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < 8; ++w) t += red[w][lane];
      y[idx] = t;
    }
    __syncthreads();
  }
}

// Tile width NT (a multiple of 8 up to 64) and column blocks covering N columns evenly.
int sk_width(int N, int* blocks) {
  *blocks = ceil_div(N, 64);
  const int per = ceil_div(N, *blocks);
  return std::max(16, (per + 7) / 8 * 8);
}

// Splits of the long dimension: as many blocks as fill the SMs twice, each a whole chunk per warp at
// least (8 warps x 8 columns; a 384 x 320 unfolding then takes 30 blocks and 7 us instead of 2 and 39).  More
// often than twice where a warp's FP32 chain, an eighth of a split, would be longer than that of splits that fill
// the SMs four times with blocks of 256 rows (and 256 columns): sketches above 64 columns, which take two blocks of
// columns (600 x 950k, 96 columns: chains of 8,488 -> 4,096 columns in the same 2.5 ms).
long long sketch_chain(long long m, long long n) {
  return std::max(256LL, ceil_div_ll(n, std::max(1LL, 4LL * dev_sms() / ceil_div_ll(m, 256))));
}
void sketch_split_plan(long long m, long long n, int N, long long* jchunk, int* nsplit) {
  int cb;
  const int NT = sk_width(N, &cb);
  const long long tiles = ceil_div_ll(m, SK_ROWS) * cb;
  constexpr long long unit = SK_W * SK_JC;
  const long long chain = sketch_chain(m, n);
  long long jc = unit;
  for (int waves = 2;; ++waves) {
    const long long splits = std::max<long long>(1, (long long)waves * sk_blocks(NT) * dev_sms() / tiles);
    jc = ceil_div_ll(ceil_div_ll(n, splits), unit) * unit;
    if (jc <= SK_W * chain) break;
  }
  *jchunk = jc;
  *nsplit = (int)ceil_div_ll(n, jc);
}

// Lowers the split count until the partial sums fit `cap` doubles.
int sketch_split_fit(long long m, long long n, int N, size_t cap, long long* jchunk, int* nsplit) {
  const long long max_ns = (long long)(cap / ((size_t)N * (size_t)m));
  if (max_ns < 1) {
    set_error(TT_ERR_NOMEM, "sketch workspace");
    return TT_ERR_NOMEM;
  }
  if (*nsplit > max_ns) {
    *jchunk = (ceil_div_ll(n, max_ns) + 31) / 32 * 32;
    *nsplit = (int)ceil_div_ll(n, *jchunk);
  }
  return TT_OK;
}

template <int RC>
int run_sketch32(const float* a, long long m, long long n, const float* w, int N, long long wj, long long wc,
                 long long jchunk, int nsplit, int cb, double* part, cudaStream_t s) {
  TT_TRY(smem_optin_k(k_sketch32<RC>, sk_smem(4 * RC)));
  const dim3 grid(ceil_div(m, SK_ROWS), nsplit, cb);
  k_sketch32<RC><<<grid, 32 * SK_W, sk_smem(4 * RC), s>>>(a, m, n, w, N, wj, wc, jchunk, part);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

int sketch32(const float* a, long long m, long long n, const float* w, int N, long long wj, long long wc,
             long long jchunk, int nsplit, double* part, cudaStream_t s) {
  int cb;
  switch (sk_width(N, &cb)) {
    case 16: return run_sketch32<4>(a, m, n, w, N, wj, wc, jchunk, nsplit, cb, part, s);
    case 24: return run_sketch32<6>(a, m, n, w, N, wj, wc, jchunk, nsplit, cb, part, s);
    case 32: return run_sketch32<8>(a, m, n, w, N, wj, wc, jchunk, nsplit, cb, part, s);
    case 40: return run_sketch32<10>(a, m, n, w, N, wj, wc, jchunk, nsplit, cb, part, s);
    case 48: return run_sketch32<12>(a, m, n, w, N, wj, wc, jchunk, nsplit, cb, part, s);
    case 56: return run_sketch32<14>(a, m, n, w, N, wj, wc, jchunk, nsplit, cb, part, s);
    default: return run_sketch32<16>(a, m, n, w, N, wj, wc, jchunk, nsplit, cb, part, s);
  }
}

// ---------------------------------------------------------------------------------------
// projection
// ---------------------------------------------------------------------------------------
// out = A^T Q, contraction along A's contiguous dimension, so both operands are paired along it: an
// accumulator holds the sums over even and odd k, nothing is transposed or copied (8 x RC pairs take
// 8 + RC 16-byte loads per 4 k, 16 RC paired FMAs).  128 columns of A x NT = 8 RC outputs per block of 4
// warps, chunks of 32 k through a 3-deep cp.async ring, rows padded to 36 floats (the 16-byte loads of
// 4 columns of A and of 8 columns of Q then fall in distinct banks).
constexpr int PJ_T = 128, PJ_KC = 32, PJ_LD = PJ_KC + 4, PJ_ST = 3;
constexpr size_t pj_smem(int NT) { return (size_t)PJ_ST * (PJ_T + NT) * PJ_LD * sizeof(float); }

template <int RC>
__global__ void __launch_bounds__(PJ_T) k_project32(const float* __restrict__ a, long long m, long long n,
                                                    const float* __restrict__ q, int N, long long ldq,
                                                    float* __restrict__ out, long long ldo, int mode, int r0,
                                                    int r1, long long kchunk) {
  constexpr int NT = 8 * RC, SLOT = (PJ_T + NT) * PJ_LD;
  extern __shared__ __align__(16) float sm_pj[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, jg = lane & 3, cg = lane >> 2;
  const long long j0 = (long long)blockIdx.x * PJ_T;
  const int c0 = blockIdx.y * NT;
  const long long kb = blockIdx.z * kchunk, ke = min(kb + kchunk, m);
  out += (long long)blockIdx.z * n * ldo;  // K splits write partial blocks
  const int nch = ke > kb ? (int)((ke - kb + PJ_KC - 1) / PJ_KC) : 0;
  const bool va = (m & 3) == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
  const bool vq = (ldq & 3) == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0;
  // chunk of 32 k: rows of A and Q into rows of PJ_LD floats, zero past the ends.  The aligned copy of a
  // thread is k 4 (tid & 7) .. + 3 of rows tid / 8 + 16 u, the other one (m no multiple of 4, the last chunk) k
  // tid & 31 of rows tid / 32 + 4 u: addresses are set up once (97 x 700k, 24 outputs: 243 us with an index
  // calculation per copy, 170 so).
  const int cr = tid >> 3, ck = 4 * (tid & 7);
  const float* const asrc = a + (j0 + cr) * m + kb + ck;
  const float* const qsrc = q + (c0 + cr) * ldq + kb + ck;
  const long long astep = 16 * m, qstep = 16 * ldq;
  const int arows = (int)min((long long)PJ_T, n - j0) - cr, qrows = N - c0 - cr;  // rows left for this thread
  const float* const asrc1 = a + (j0 + warp) * m + kb + lane;
  const float* const qsrc1 = q + (c0 + warp) * ldq + kb + lane;
  const int arows1 = (int)min((long long)PJ_T, n - j0) - warp, qrows1 = N - c0 - warp;
  auto copy1 = [&](auto count, float* dst, const float* src, long long step, int rows, const float* safe) {
#pragma unroll 16
    for (int u = 0; u < decltype(count)::value / 4; ++u) {
      const bool ok = 4 * u < rows;
      cp_async4(dst + 4 * u * PJ_LD, ok ? src : safe, ok);
      src += step;
    }
  };
  auto load = [&](int ch) {
    if (ch < nch) {
      float* const as = sm_pj + (ch % PJ_ST) * SLOT;
      const long long k0 = kb + (long long)ch * PJ_KC;
      const bool whole = k0 + PJ_KC <= ke;
      if (va && whole) {
        const float* src = asrc + ch * PJ_KC;
        float* dst = as + cr * PJ_LD + ck;
#pragma unroll
        for (int u = 0; u < PJ_T / 16; ++u) {
          cp_async16z(dst + 16 * u * PJ_LD, 16 * u < arows ? src : a, 16 * u < arows);
          src += astep;
        }
      } else {
        copy1(std::integral_constant<int, PJ_T>{}, as + warp * PJ_LD + lane, asrc1 + ch * PJ_KC, 4 * m,
              k0 + lane < ke ? arows1 : 0, a);
      }
      if (vq && whole) {
        const float* src = qsrc + ch * PJ_KC;
        float* dst = as + (PJ_T + cr) * PJ_LD + ck;
#pragma unroll
        for (int u = 0; u < (NT + 15) / 16; ++u) {
          if (cr + 16 * u < NT) cp_async16z(dst + 16 * u * PJ_LD, 16 * u < qrows ? src : q, 16 * u < qrows);
          src += qstep;
        }
      } else {
        copy1(std::integral_constant<int, NT>{}, as + (PJ_T + warp) * PJ_LD + lane, qsrc1 + ch * PJ_KC, 4 * ldq,
              k0 + lane < ke ? qrows1 : 0, q);
      }
    }
    cp_async_commit();
  };
  uint64_t acc[8][RC];  // column j0 + 32 warp + jg + 4 e of A, output c0 + cg + 8 c
#pragma unroll
  for (int e = 0; e < 8; ++e)
#pragma unroll
    for (int c = 0; c < RC; ++c) acc[e][c] = 0ull;
#pragma unroll
  for (int s = 0; s < PJ_ST - 1; ++s) load(s);
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<PJ_ST - 2>();
    __syncthreads();  // chunk ch landed for every thread; the chunk before it is consumed
    load(ch + PJ_ST - 1);
    const float* as = sm_pj + (ch % PJ_ST) * SLOT + (32 * warp + jg) * PJ_LD;
    const float* qs = sm_pj + (ch % PJ_ST) * SLOT + (PJ_T + cg) * PJ_LD;
#pragma unroll 4
    for (int k = 0; k < PJ_KC; k += 4) {
      ulonglong2 qv[RC];
#pragma unroll
      for (int c = 0; c < RC; ++c) qv[c] = *reinterpret_cast<const ulonglong2*>(qs + 8 * c * PJ_LD + k);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(as + 4 * e * PJ_LD + k);
#pragma unroll
        for (int c = 0; c < RC; ++c) ffma2(acc[e][c], x.x, qv[c].x);
#pragma unroll
        for (int c = 0; c < RC; ++c) ffma2(acc[e][c], x.y, qv[c].y);
      }
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const long long j = j0 + 32 * warp + jg + 4 * e;
    if (j >= n) continue;
#pragma unroll
    for (int c = 0; c < RC; ++c) {
      const int col = c0 + cg + 8 * c;
      if (col >= N) continue;
      float lo, hi;
      f2_unpack(acc[e][c], lo, hi);
      const float v = lo + hi;
      if (mode == OUT_ROWMAJOR) {
        out[j * ldo + col] = v;
      } else if (mode == OUT_COLMAJOR) {
        out[j + ldo * col] = v;
      } else {
        const int ai = col % r0, bi = col / r0;
        out[(long long)bi + (long long)r1 * (j + n * (long long)ai)] = v;
      }
    }
  }
}

// Sum of the K-split partial projections (row-major n x N blocks) into the requested layout.
__global__ void k_project_reduce(const float* __restrict__ part, long long n, int N, int nsplit,
                                 float* __restrict__ out, long long ldo, int mode, int r0, int r1) {
  const long long total = n * N;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    double vd = 0.0;
#pragma unroll 8
    for (int z = 0; z < nsplit; ++z) vd += (double)part[(long long)z * total + idx];
    const float v = (float)vd;
    const long long j = idx / N;
    const int c = (int)(idx - j * N);
    if (mode == OUT_ROWMAJOR) {
      out[j * ldo + c] = v;
    } else if (mode == OUT_COLMAJOR) {
      out[j + ldo * c] = v;
    } else {
      const int ai = c % r0, bi = c / r0;
      out[(long long)bi + (long long)r1 * (j + n * (long long)ai)] = v;
    }
  }
}

// Small-K projection out = Q^T A for K = m <= 64 (the rotation E_r^T B of a small factor, or an m <= 64
// unfolding): a tile of columns is one contiguous block, staged whole in shared memory with an odd row
// stride (m odd: as it lies; m = 2 mod 4: as it lies, two-way conflicts), Q as float4 rows.  A thread
// computes NPT outputs of CT columns, so a row of Q is loaded once for CT columns; G groups of threads
// share a column.  Products in one chain over k per output.  Row-major outputs and the TR bond permute
// leave through shared memory as contiguous runs.  HBM / FP32 FMA bound: 30 -> 20 rows of 19M columns
// 960 us (1885 with one column per thread).
template <int NP, int G, int CT>
__global__ void __launch_bounds__(256) k_proj_smallk(const float* __restrict__ a, int m, long long n,
                                                     const float* __restrict__ q, int N, long long ldq,
                                                     float* __restrict__ out, long long ldo, int mode,
                                                     int r0, int r1) {
  constexpr int TH = 256 / G, TJ = CT * TH;  // threads across the columns, columns per tile
  constexpr int NPT = NP / G;                // outputs per thread
  static_assert(NPT % 4 == 0, "outputs per thread");
  extern __shared__ __align__(16) float sm_pk[];
  float* Es = sm_pk;           // m x NP: Es[k * NP + c] = Q[k + ldq c]
  float* Xs = Es + 64 * NP;    // TJ x S input tile, then TJ x (NP + 1) output tile
  const bool lin = (m & 3) != 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
  const int S = lin || (m & 1) ? m : m + 1;
  constexpr int OS = NP + 1;
  const int tid = threadIdx.x;
  const int col_t = tid % TH, grp = tid / TH;
  for (int idx = tid; idx < m * NP; idx += 256) {
    const int k = idx / NP, c = idx - (idx / NP) * NP;
    Es[idx] = (c < N) ? q[k + ldq * (long long)c] : 0.f;
  }
  const bool vec = (m & 3) == 0 && ((reinterpret_cast<uintptr_t>(a) & 15) == 0);
  // Row-major outputs with ldo == N form one contiguous block per tile; bond-permuted outputs
  // (r0, r1, n) -> (r1, n, r0) form r0 contiguous runs of r1 * nj values per tile.
  const bool staged_out = (mode == OUT_ROWMAJOR && ldo == N) || (mode == OUT_PERM231 && r0 * r1 == N);
  // Quotients of tile-local indices (< 2^15) by m, N or r1 (<= 128) through a float reciprocal:
  // the rounding error is far below the 0.5 / divisor margin, so the floor is exact.
  const float inv_m = 1.0f / (float)m, inv_n = 1.0f / (float)N, inv_r1 = 1.0f / (float)(r1 > 0 ? r1 : 1);
  auto qdiv = [](int e, float inv) { return (int)(((float)e + 0.5f) * inv); };
  for (long long tile = blockIdx.x; tile * TJ < n; tile += gridDim.x) {
    const long long j0 = tile * TJ;
    const int nj = (int)((n - j0 < TJ) ? n - j0 : TJ);
    const float* src = a + j0 * m;
    const int cnt = nj * m;
    __syncthreads();
    if (lin) {
      for (int f4 = tid; f4 < (cnt >> 2); f4 += 256) cp_async16(Xs + 4 * f4, src + 4 * f4);
      if (tid < (cnt & 3)) cp_async4(Xs + (cnt & ~3) + tid, src + (cnt & ~3) + tid, true);
      cp_async_commit();
      cp_async_wait<0>();
    } else if (vec) {
      for (int f4 = tid; f4 < (cnt >> 2); f4 += 256) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(src) + f4);
        const int e = 4 * f4, col = qdiv(e, inv_m), k = e - col * m;
        float* d = Xs + col * S + k;
        d[0] = v.x;
        d[1] = v.y;
        d[2] = v.z;
        d[3] = v.w;
      }
    } else {
      for (int f = tid; f < cnt; f += 256) {
        const int col = qdiv(f, inv_m), k = f - col * m;
        Xs[col * S + k] = __ldg(src + f);
      }
    }
    __syncthreads();
    uint64_t acc[CT][NPT / 2];  // output pairs of columns col_t + TH u (columns past nj: stale values, not stored)
#pragma unroll
    for (int u = 0; u < CT; ++u)
#pragma unroll
      for (int c = 0; c < NPT / 2; ++c) acc[u][c] = 0ull;
    {
      const float* xr = Xs + col_t * S;
      const float* er = Es + grp * NPT;
#pragma unroll 2
      for (int k = 0; k < m; ++k) {
        uint64_t xd[CT];
#pragma unroll
        for (int u = 0; u < CT; ++u) xd[u] = f2_dup(xr[u * TH * S + k]);
#pragma unroll
        for (int c4 = 0; c4 < NPT / 4; ++c4) {
          const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(er + k * NP + 4 * c4);
#pragma unroll
          for (int u = 0; u < CT; ++u) {
            ffma2(acc[u][2 * c4], xd[u], e.x);
            ffma2(acc[u][2 * c4 + 1], xd[u], e.y);
          }
        }
      }
    }
    if (staged_out) __syncthreads();
#pragma unroll
    for (int u = 0; u < CT; ++u) {
      const int cl = col_t + TH * u;
      if (cl >= nj) continue;
      const long long j = j0 + cl;
#pragma unroll
      for (int cc = 0; cc < NPT; ++cc) {
        const int c = grp * NPT + cc;
        if (c >= N) continue;
        float lo, hi;
        f2_unpack(acc[u][cc / 2], lo, hi);
        const float v = (cc & 1) ? hi : lo;
        if (staged_out) {
          Xs[cl * OS + c] = v;
        } else if (mode == OUT_ROWMAJOR) {
          out[j * ldo + c] = v;
        } else if (mode == OUT_COLMAJOR) {
          out[j + ldo * c] = v;
        } else {
          const int ai = c % r0, bi = c / r0;
          out[(long long)bi + (long long)r1 * (j + n * (long long)ai)] = v;
        }
      }
    }
    if (staged_out) {
      __syncthreads();
      if (mode == OUT_ROWMAJOR) {
        float* dst = out + j0 * N;
        for (int f = tid; f < nj * N; f += 256) {
          const int col = qdiv(f, inv_n), c = f - col * N;
          dst[f] = Xs[col * OS + c];
        }
      } else {
        const int run = r1 * nj;
        for (int ai = 0; ai < r0; ++ai) {
          float* dst = out + (long long)r1 * (j0 + n * (long long)ai);
          for (int f = tid; f < run; f += 256) {
            const int col = qdiv(f, inv_r1), bi = f - col * r1;
            dst[f] = Xs[col * OS + ai + r0 * bi];
          }
        }
      }
    }
  }
}

template <int NP, int G, int CT>
int run_smallk(const float* a, int m, long long n, const float* q, int N, long long ldq, float* out, long long ldo,
               int mode, int r0, int r1, cudaStream_t s) {
  constexpr int TJ = CT * 256 / G;
  const size_t shm = (64 * (size_t)NP + (size_t)TJ * std::max(m + 1, NP + 1)) * sizeof(float);
  TT_TRY(smem_optin_k(k_proj_smallk<NP, G, CT>, (64 * (size_t)NP + (size_t)TJ * 65) * sizeof(float)));
  const int grid = (int)std::min<long long>(ceil_div_ll(n, TJ), 16LL * dev_sms());
  k_proj_smallk<NP, G, CT><<<grid, 256, shm, s>>>(a, m, n, q, N, ldq, out, ldo, mode, r0, r1);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

// Columns per thread: 4 (2 for up to 16 outputs, whose tiles are twice as wide) where two blocks of
// tiles still share an SM and the tiles still fill the SMs; 1 otherwise.
int project_smallk(const float* a, int m, long long n, const float* q, int N, long long ldq, float* out,
                   long long ldo, int mode, int r0, int r1, cudaStream_t s) {
#define SMALLK(NP, G, CT) run_smallk<NP, G, CT>(a, m, n, q, N, ldq, out, ldo, mode, r0, r1, s)
  const bool wide = n >= 512LL * dev_sms();
  if (N <= 8) return wide && m <= 48 ? SMALLK(8, 1, 2) : SMALLK(8, 1, 1);
  if (N <= 16) return wide && m <= 48 ? SMALLK(16, 1, 2) : SMALLK(16, 1, 1);
  if (N <= 24) return wide ? (m <= 48 ? SMALLK(24, 2, 4) : SMALLK(24, 2, 2)) : SMALLK(24, 2, 1);
  if (N <= 32) return wide ? (m <= 48 ? SMALLK(32, 2, 4) : SMALLK(32, 2, 2)) : SMALLK(32, 2, 1);
  if (N <= 48) return wide ? SMALLK(48, 4, 4) : SMALLK(48, 4, 1);
  return wide ? SMALLK(64, 4, 4) : SMALLK(64, 4, 1);
#undef SMALLK
}

constexpr size_t kProjectSplitCap = 16u << 20;  // bytes of K-split partials

// Output tile width: the multiple of 8 in 16..64 that covers N in as few, evenly filled column blocks.
int pj_width(int N, int* blocks) {
  *blocks = ceil_div(N, 64);
  return std::max(16, (ceil_div(N, *blocks) + 7) / 8 * 8);
}

// K splits for projections whose column tiles alone cannot fill the GPU (3 blocks of 4 warps per SM).
int project_ksplit(long long m, long long n, int N, long long* kchunk) {
  int cb;
  pj_width(N, &cb);
  const long long blocks = ceil_div_ll(n, PJ_T) * cb;
  int ks = 1;
  if (m >= 128 && blocks < 3LL * dev_sms()) {
    ks = (int)std::min<long long>(ceil_div_ll(3LL * dev_sms(), blocks), m / 64);
    const long long cap = (long long)(kProjectSplitCap / (sizeof(float) * (size_t)n * N));
    ks = (int)std::max<long long>(1, std::min<long long>(ks, cap));
  }
  long long kc = ceil_div_ll(m, ks);
  kc = ceil_div_ll(kc, PJ_KC) * PJ_KC;
  *kchunk = kc;
  return (int)ceil_div_ll(m, kc);
}

// Lowers the split count to `fit` where it is above.
int project_split_fit(long long m, long long fit, int ks, long long* kchunk) {
  if (ks <= fit) return ks;
  *kchunk = ceil_div_ll(ceil_div_ll(m, std::max(1LL, fit)), PJ_KC) * PJ_KC;
  return (int)ceil_div_ll(m, *kchunk);
}

template <int RC>
int run_project32(const float* a, long long m, long long n, const float* q, int N, long long ldq, float* out,
                  long long ldo, int mode, int r0, int r1, int cb, int ks, long long kc, cudaStream_t s) {
  TT_TRY(smem_optin_k(k_project32<RC>, pj_smem(8 * RC)));
  const dim3 grid(ceil_div(n, PJ_T), cb, ks);
  k_project32<RC><<<grid, PJ_T, pj_smem(8 * RC), s>>>(a, m, n, q, N, ldq, out, ldo, mode, r0, r1, kc);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

}  // namespace

size_t sketch_ws_bytes(long long m, long long n, int N) {
  long long jchunk;
  int nsplit;
  sketch_split_plan(m, n, N, &jchunk, &nsplit);
  const size_t simt = (size_t)nsplit * (size_t)N * (size_t)m * sizeof(double) + 4096;
  return std::max(simt, sketch_tc_ws_bytes(m, n, N));
}

size_t sketch_ws_least(long long m, long long n, int N) {
  const long long jc = ceil_div_ll(sketch_chain(m, n), 32) * 32;
  const size_t simt = (size_t)ceil_div_ll(n, jc) * (size_t)N * (size_t)m * sizeof(double) + 4096;
  return std::min(sketch_ws_bytes(m, n, N), std::max(simt, sketch_tc_ws_bytes(m, n, N)));
}

int launch_reduce_splits(const double* part, long long count, int nsplit, double* y, cudaStream_t s) {
  if (count <= 0) return TT_OK;
  k_reduce_splits<<<(int)std::min<long long>(ceil_div_ll(count, 32), 16LL * dev_sms()), 256, 0, s>>>(
      part, count, nsplit, y);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

int launch_sketch(const float* a, long long m, long long n, const float* w, int N, long long wj,
                  long long wc, double* y, int engine, Arena& ws, DevStatus* st, cudaStream_t s) {
  if (m <= 0 || n <= 0 || N <= 0) return TT_OK;
  if (engine == TT_GEMM_TC) {
    int rc = launch_sketch_tc(a, m, n, w, N, wj, wc, y, ws, st, s);
    if (rc != TT_ERR_UNSUPPORTED) return rc;
  }
  long long jchunk;
  int nsplit;
  sketch_split_plan(m, n, N, &jchunk, &nsplit);
  const size_t mk = ws.mark();
  const size_t left = (ws.cap - std::min(ws.cap, (mk + 255) & ~size_t(255))) & ~size_t(255);
  TT_TRY(sketch_split_fit(m, n, N, left / sizeof(double), &jchunk, &nsplit));
  double* part = ws.take<double>((size_t)nsplit * N * m);
  if (!part) {
    set_error(TT_ERR_NOMEM, "sketch workspace");
    return TT_ERR_NOMEM;
  }
  TT_TRY(sketch32(a, m, n, w, N, wj, wc, jchunk, nsplit, part, s));
  TT_TRY(launch_reduce_splits(part, (long long)N * m, nsplit, y, s));
  ws.reset(mk);
  return TT_OK;
}

// FP32 sketch with the split partials in caller-provided scratch (`part`, `part_cap` doubles);
// the split count is lowered until the partials fit.  Allocates nothing.
int launch_sketch_simt_static(const float* a, long long m, long long n, const float* w, int N,
                              long long wj, long long wc, double* y, double* part, size_t part_cap,
                              cudaStream_t s) {
  if (m <= 0 || n <= 0 || N <= 0) return TT_OK;
  long long jchunk;
  int nsplit;
  sketch_split_plan(m, n, N, &jchunk, &nsplit);
  if (sketch_split_fit(m, n, N, part_cap, &jchunk, &nsplit) != TT_OK) {
    set_error(TT_ERR_SHAPE, "sketch partials of %lld x %d doubles exceed the scratch of %zu doubles", m, N,
              part_cap);
    return TT_ERR_SHAPE;
  }
  TT_TRY(sketch32(a, m, n, w, N, wj, wc, jchunk, nsplit, part, s));
  return launch_reduce_splits(part, (long long)N * m, nsplit, y, s);
}

size_t project_ws_bytes(long long m, long long n, int N) {
  long long kc;
  const int ks = project_ksplit(m, n, N, &kc);
  const size_t split = ks > 1 ? (size_t)ks * n * N * sizeof(float) : 0;
  return split + 2 * (size_t)m * N * sizeof(float) + 4096;
}

size_t project_ws_least(long long m, long long n, int N) {
  const int nt = N <= 16 ? 16 : N <= 32 ? 32 : N <= 48 ? 48 : 64;
  const long long blocks = ceil_div_ll(n, 256) * ceil_div(N, nt);
  long long kc, least = 1;
  int ks = project_ksplit(m, n, N, &kc);
  if (m >= 256 && blocks < 2LL * dev_sms()) least = std::min(ceil_div_ll(2LL * dev_sms(), blocks), m / 64);
  ks = project_split_fit(m, least, ks, &kc);
  const size_t split = ks > 1 ? (size_t)ks * n * N * sizeof(float) : 0;
  return split + 2 * (size_t)m * N * sizeof(float) + 4096;
}

int launch_project(const float* a, long long m, long long n, const float* q, int N, long long ldq,
                   float* out, long long ldo, int mode, int r0, int r1, int engine, Arena& ws,
                   DevStatus* st, cudaStream_t s) {
  if (n <= 0 || N <= 0) return TT_OK;
  if (engine == TT_GEMM_TC) {
    int rc = launch_project_tc(a, m, n, q, N, ldq, out, ldo, mode, r0, r1, ws, st, s);
    if (rc != TT_ERR_UNSUPPORTED) return rc;
  }
  if (m <= 64 && N <= 64) return project_smallk(a, (int)m, n, q, N, ldq, out, ldo, mode, r0, r1, s);
  long long kc;
  int ks = project_ksplit(m, n, N, &kc);
  float* part = nullptr;
  const size_t mk = ws.mark();
  const size_t left = (ws.cap - std::min(ws.cap, (mk + 255) & ~size_t(255))) & ~size_t(255);
  ks = project_split_fit(m, (long long)(left / (sizeof(float) * (size_t)n * N)), ks, &kc);
  if (ks > 1) part = ws.take<float>((size_t)ks * n * N);
  if (!part) {
    ks = 1;
    kc = m;
  }
  float* dst = ks > 1 ? part : out;
  const long long ldd = ks > 1 ? N : ldo;
  const int md = ks > 1 ? OUT_ROWMAJOR : mode;
  int cb, rc;
#define PJ_CASE(V) \
  case 8 * V: rc = run_project32<V>(a, m, n, q, N, ldq, dst, ldd, md, r0, r1, cb, ks, kc, s); break;
  switch (pj_width(N, &cb)) {
    PJ_CASE(2)
    PJ_CASE(3)
    PJ_CASE(4)
    PJ_CASE(5)
    PJ_CASE(6)
    PJ_CASE(7)
    default:
    PJ_CASE(8)
  }
#undef PJ_CASE
  TT_TRY(rc);
  if (ks > 1) {
    const long long total = n * N;
    k_project_reduce<<<(int)std::min<long long>(ceil_div_ll(total, 256), 8LL * dev_sms()), 256, 0, s>>>(
        part, n, N, ks, out, ldo, mode, r0, r1);
    count_launch();
    TT_LAUNCH_CHECK();
  }
  ws.reset(mk);
  return TT_OK;
}

}  // namespace ttr
