// Gram W = sum_j x_j x_j^T (M x M, M <= 128) of many short FP32 vectors with FP64 products and sums: the
// Gram of a small factor B, of a power basis Z, of an unfolding with 33..128 rows or few vectors.
//
// Bound by the FP64 FMAs (64 per clock and SM).  They run as mma.m8n8k4.f64: it has the rate of the FP64
// FMAs, but 256 FMAs take one operand register a lane, where a register-tiled FMA loop is held up by its
// shared-memory loads (two wavefronts per 64-bit load).  In X^T X both operands of a step are the same
// registers: lane l holds component 8 b + l / 4 of vector l % 4 for block b, as A and as B.  So a value is
// loaded and converted once per warp (conversions run at ~15 per clock and SM).  Each warp streams its
// own vectors through its own cp.async ring (no block barrier until the end) and keeps all 8 x 8 tiles of
// its part of W's upper triangle in registers: blocks of up to 6 x 6 tiles, larger M being split into
// jobs (pairs of component groups) with blocks in proportion to their tiles.  One kernel for either layout,
// any M and any alignment.  24 x 8.4M: 249 us; 85 x 950k: 329; 45 x 850k: 77; 80 x 262k (column-major): 75.
#include <algorithm>

#include "kernels.cuh"

namespace ttr {
namespace {

constexpr int GR_W = 8;   // warps per block
constexpr int gr_st(int ng) { return ng == 1 ? 4 : 3; }  // chunks in a warp's ring

// Component groups of gs blocks of 8; job n multiplies groups a[n] <= b[n] on blocks start[n]..start[n+1]-1.
struct GramJobs {
  int gs, n, start[7], a[6], b[6];
};
constexpr int gr_vc(int gs) { return gs <= 3 ? 32 : 16; }  // vectors per chunk
// row stride of a chunk of row-major vectors: 8 or 24 mod 32 floats, so that 4 vectors x 8 components hit
// distinct banks
constexpr int gr_rs(int w) { return (w & 15) == 8 ? w : w + 8; }
// floats of a ring slot holding ng groups
constexpr int gr_slot(int gs, int ng, bool col) {
  // (row-major, two groups: or the whole vectors of up to 128 components)
  return col ? ng * 8 * gs * (gr_vc(gs) + 4) : gr_vc(gs) * (ng == 1 ? gr_rs(8 * gs) : 144);
}
constexpr size_t gr_smem(int gs, int ng, bool col) {
  const size_t ring = (size_t)GR_W * gr_st(ng) * gr_slot(gs, ng, col) * sizeof(float);
  const size_t red = (size_t)GR_W * 64 * (ng == 1 ? gs * (gs + 1) / 2 : gs * gs) * sizeof(double);
  return ring > red ? ring : red;
}

GramJobs gr_jobs(long long nvec, int M) {
  GramJobs J = {};
  const int tt = (M + 7) / 8, ng = (tt + 5) / 6;
  J.gs = (tt + ng - 1) / ng;
  // enough vectors per warp to fill its ring, as many blocks as the SMs take
  const long long most = std::max<long long>(1, ceil_div_ll(nvec, 2LL * GR_W * gr_vc(J.gs)));
  const long long sms = (long long)dev_sms() * (J.gs <= 3 ? 2 : 1);
  int tiles = 0;
  for (int a = 0; a < ng; ++a)
    for (int b = a; b < ng; ++b) tiles += a == b ? J.gs * (J.gs + 1) / 2 : J.gs * J.gs;
  for (int a = 0; a < ng; ++a)
    for (int b = a; b < ng; ++b) {
      const int t = a == b ? J.gs * (J.gs + 1) / 2 : J.gs * J.gs;
      const long long share = std::max<long long>(1, sms * t / tiles);
      J.a[J.n] = a;
      J.b[J.n] = b;
      J.start[J.n + 1] = J.start[J.n] + (int)std::min(most, share);
      ++J.n;
    }
  return J;
}

// One warp's share of a job: NG = 1, one group against itself (upper tiles); NG = 2, two groups against
// each other; MULTI: M has more than one group.  Ends with the block's sum of the tiles, rows of 8 GS, in
// dst.
template <int GS, int NG, bool MULTI, bool COL>
__device__ __forceinline__ void gram_job(const float* __restrict__ x, long long nvec, int M, long long vs,
                                         long long es, int ga, int gb, int blk, int nblk, float* sm,
                                         double* __restrict__ dst) {
  constexpr int VC = gr_vc(GS), W8 = 8 * GS, RS = gr_rs(W8);
  constexpr int SLOT = gr_slot(GS, MULTI ? 2 : 1, COL), GR_ST = gr_st(MULTI ? 2 : 1);
  constexpr int NT = NG == 1 ? GS * (GS + 1) / 2 : GS * GS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* const ring = sm + (size_t)warp * GR_ST * SLOT;
  const long long nch = (nvec + VC - 1) / VC, gw = (long long)blk * GR_W + warp, GW = (long long)nblk * GR_W;
  const long long my = gw < nch ? (nch - 1 - gw) / GW + 1 : 0;
  const bool al = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const bool v16 = al && (COL ? vs == 1 && (es & 3) == 0 : es == 1 && (vs & 3) == 0);
  // contiguous vectors whose starts are not 16-byte aligned: a chunk is copied whole, as it lies
  const bool lin = !COL && al && es == 1 && vs == M && (M & 3) != 0;
  auto load = [&](long long k) {
    if (k < my) {
      const long long v0 = (gw + k * GW) * VC;
      const int nv = (int)min((long long)VC, nvec - v0);
      float* const d0 = ring + (k % GR_ST) * SLOT;
      if (lin) {
        const float* src = x + v0 * M;
        if (nv == VC) {
          for (int f = lane; f < VC / 4 * M; f += 32) cp_async16(d0 + 4 * f, src + 4 * f);
        } else {
          for (int f = lane; f < VC * M; f += 32) cp_async4(d0 + f, f < nv * M ? src + f : x, f < nv * M);
        }
        cp_async_commit();
        return;
      }
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        const int c0 = (g == 0 ? ga : gb) * W8, nc = min(W8, M - c0);
        if (COL) {
          float* const d = d0 + g * W8 * (VC + 4);
          if (v16 && nv == VC) {
            for (int f = lane; f < nc * (VC / 4); f += 32) {
              const int c = f / (VC / 4), v = 4 * (f % (VC / 4));
              cp_async16(d + c * (VC + 4) + v, x + (v0 + v) + es * (c0 + c));
            }
          } else {
            for (int f = lane; f < nc * VC; f += 32) {
              const int c = f / VC, v = f % VC;
              cp_async4(d + c * (VC + 4) + v, v < nv ? x + vs * (v0 + v) + es * (c0 + c) : x, v < nv);
            }
          }
        } else {
          float* const d = d0 + g * VC * RS;
          if (v16 && (nc & 3) == 0) {
            for (int f = lane; f < VC * (W8 / 4); f += 32) {
              const int v = f / (W8 / 4), c = 4 * (f % (W8 / 4));
              if (c < nc) cp_async16z(d + v * RS + c, v < nv ? x + vs * (v0 + v) + (c0 + c) : x, v < nv);
            }
          } else {
            for (int f = lane; f < VC * W8; f += 32) {
              const int v = f / W8, c = f % W8;
              if (c < nc) cp_async4(d + v * RS + c, v < nv ? x + vs * (v0 + v) + es * (c0 + c) : x, v < nv);
            }
          }
        }
      }
    }
    cp_async_commit();
  };
  double acc[NT][2];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = 0.0;
  // components past M are whatever the ring held: they reach only rows and columns past M
#pragma unroll
  for (int s = 0; s < GR_ST - 1; ++s) load(s);
  const int lv = lane & 3, lc = lane >> 2;
  const int rs = lin ? M : RS;  // row-major: stride of a vector, and where the groups start
  const int goff[2] = {lin ? ga * W8 : 0, lin ? gb * W8 : VC * RS};
  for (long long k = 0; k < my; ++k) {
    cp_async_wait<GR_ST - 2>();
    __syncwarp();  // chunk k landed for every lane; the chunk before it is consumed
    load(k + GR_ST - 1);
    const float* const s0 = ring + (k % GR_ST) * SLOT;
#pragma unroll 2
    for (int v = 0; v < VC; v += 4) {
      double f[NG][GS];
#pragma unroll
      for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int b = 0; b < GS; ++b)
          f[g][b] = COL ? (double)s0[(g * W8 + 8 * b + lc) * (VC + 4) + v + lv]
                        : (double)s0[goff[g] + (v + lv) * rs + 8 * b + lc];
      int t = 0;
#pragma unroll
      for (int a = 0; a < GS; ++a)
#pragma unroll
        for (int b = NG == 1 ? a : 0; b < GS; ++b, ++t) mma_f64(acc[t], f[0][a], f[NG - 1][b]);
    }
  }
  cp_async_wait<0>();
  __syncthreads();  // the rings are free: sum the warps' tiles
  double* const red = reinterpret_cast<double*>(sm);
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    red[(warp * NT + t) * 64 + 2 * lane] = acc[t][0];
    red[(warp * NT + t) * 64 + 2 * lane + 1] = acc[t][1];
  }
  __syncthreads();
  int t = 0;
#pragma unroll
  for (int a = 0; a < GS; ++a)
#pragma unroll
    for (int b = NG == 1 ? a : 0; b < GS; ++b, ++t)
      if (threadIdx.x < 64) {
        const int e = threadIdx.x;  // row e / 8, column e % 8 of the tile
        double sum = 0.0;
#pragma unroll
        for (int w = 0; w < GR_W; ++w) sum += red[(w * NT + t) * 64 + e];
        dst[(8 * a + e / 8) * W8 + 8 * b + e % 8] = sum;
      }
}

// Component c of vector j at x[j vs + c es]; COL: the vectors of a component are the closer ones.
template <int GS, bool MULTI, bool COL>
__global__ void __launch_bounds__(32 * GR_W) k_gram64(const float* __restrict__ x, long long nvec, int M, long long vs,
                                                     long long es, const GramJobs J, double* __restrict__ part) {
  extern __shared__ __align__(16) double sm_gr[];
  float* const sm = reinterpret_cast<float*>(sm_gr);
  int n = 0;
  while ((int)blockIdx.x >= J.start[n + 1]) ++n;
  const int blk = blockIdx.x - J.start[n], nblk = J.start[n + 1] - J.start[n];
  double* const dst = part + (long long)blockIdx.x * (8 * GS) * (8 * GS);
  if (!MULTI || J.a[n] == J.b[n])
    gram_job<GS, 1, MULTI, COL>(x, nvec, M, vs, es, J.a[n], J.b[n], blk, nblk, sm, dst);
  else if constexpr (MULTI)
    gram_job<GS, 2, MULTI, COL>(x, nvec, M, vs, es, J.a[n], J.b[n], blk, nblk, sm, dst);
}

// W (M x M, column-major) = sum of the blocks' partials of each job (rows of stride w8, bs doubles apart):
// a warp per entry of the upper triangle, lanes stride over the blocks, fixed-order shuffle tree
// (deterministic).
__global__ void __launch_bounds__(256) k_gram_reduce(const double* __restrict__ part, const GramJobs J, int w8,
                                                     long long bs, int M, double* __restrict__ w) {
  const int idx = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const int i = idx / M, j = idx - i * M;
  if (i >= M || i > j) return;
  const int ga = i / w8, gb = j / w8;
  int n = 0;
  while (J.a[n] != ga || J.b[n] != gb) ++n;
  const double* src = part + (i - ga * w8) * w8 + (j - gb * w8);
  double sum = 0.0;
#pragma unroll 4
  for (int k = J.start[n] + lane; k < J.start[n + 1]; k += 32) sum += src[k * bs];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) {
    w[i + (long long)M * j] = sum;
    w[j + (long long)M * i] = sum;
  }
}

template <int GS, bool MULTI, bool COL>
int run_gram64(const float* x, long long nvec, int M, long long vs, long long es, const GramJobs& J, double* part,
               cudaStream_t st) {
  constexpr size_t shm = gr_smem(GS, MULTI ? 2 : 1, COL);
  TT_TRY(smem_optin_k(k_gram64<GS, MULTI, COL>, shm));
  k_gram64<GS, MULTI, COL><<<J.start[J.n], 32 * GR_W, shm, st>>>(x, nvec, M, vs, es, J, part);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}
template <int GS, bool MULTI>
int run_gram64(const float* x, long long nvec, int M, long long vs, long long es, const GramJobs& J, double* part,
               cudaStream_t st) {
  // row-major when a vector's components are the closer ones
  return es <= vs ? run_gram64<GS, MULTI, false>(x, nvec, M, vs, es, J, part, st)
                  : run_gram64<GS, MULTI, true>(x, nvec, M, vs, es, J, part, st);
}

// The exact Gram of k_gram32x (k_tc.cu: FP32 products, FP32 sums over 64 vectors, then FP64; lane 10 u +
// t takes 8 x 8 tile t of vector 3 it + u) for vectors whose length is not a multiple of 4, which the
// TMA cannot address as rows: a box of 48 vectors is one contiguous run, copied as it lies by 16-byte
// cp.async (48 M floats are always a multiple of 16 bytes), and read by 8-byte (EVEN: M even) or 4-byte
// loads.  FP32 FMA and shared-memory issue bound; 30 x 19M: 667 us.  Used where the FP64 form has 4 x 4 blocks and
// many vectors (25 to 31 components; the rule and both times are at gram_rows in driver.cu).
constexpr int G32U_VPS = 48, G32U_ST = 4, G32U_WARPS = 8;
constexpr int g32u_stage(int M) { return G32U_VPS * M + 32; }  // floats; the last vector is read 32 wide
constexpr size_t g32u_smem(int M) {
  return std::max((size_t)G32U_WARPS * G32U_ST * ((g32u_stage(M) + 3) & ~3) * sizeof(float),
                  (size_t)32 * G32U_WARPS * 65 * sizeof(double));
}
template <bool EVEN>
__global__ void __launch_bounds__(32 * G32U_WARPS, 1) k_gram32u(const float* __restrict__ x, long long nvec, int M,
                                                                double* __restrict__ part) {
  extern __shared__ __align__(16) double sm_gu[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int SF = (g32u_stage(M) + 3) & ~3;
  float* const ring = reinterpret_cast<float*>(sm_gu) + (size_t)warp * G32U_ST * SF;
  const long long nbox = (nvec + G32U_VPS - 1) / G32U_VPS;
  const long long gw = (long long)blockIdx.x * G32U_WARPS + warp, GW = (long long)gridDim.x * G32U_WARPS;
  const long long my = gw < nbox ? (nbox - 1 - gw) / GW + 1 : 0;
  auto load = [&](long long k) {
    if (k < my) {
      const long long v0 = (gw + k * GW) * G32U_VPS;
      const long long left = (nvec - v0) * M;  // floats from here to the end
      const int n4 = G32U_VPS * M / 4;
      const float* src = x + v0 * M;
      float* dst = ring + (k % G32U_ST) * SF;
      if (left >= G32U_VPS * M) {
        for (int f = lane; f < n4; f += 32) cp_async16(dst + 4 * f, src + 4 * f);
      } else {  // the last box: zeros past the end
        for (int f = lane; f < G32U_VPS * M; f += 32) cp_async4(dst + f, f < left ? src + f : x, f < left);
      }
    }
    cp_async_commit();
  };
  const int t = lane % 10, u = lane / 10;
  const int p = t < 4 ? 0 : t < 7 ? 1 : t < 9 ? 2 : 3;
  const int q = t < 4 ? t : t < 7 ? t - 3 : t < 9 ? t - 5 : 3;
  uint64_t acc[8][4];  // (W[8p+i][8q+2j], W[8p+i][8q+2j+1])
  double accd[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int j = 0; j < 8; ++j) accd[i][j] = 0.0;
  }
  auto flush = [&]() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float lo, hi;
        f2_unpack(acc[i][j], lo, hi);
        accd[i][2 * j] += (double)lo;
        accd[i][2 * j + 1] += (double)hi;
        acc[i][j] = 0ull;
      }
  };
#pragma unroll
  for (int s = 0; s < G32U_ST - 1; ++s) load(s);
  for (long long k = 0; k < my; ++k) {
    cp_async_wait<G32U_ST - 2>();
    __syncwarp();  // box k landed for every lane; the box before it is consumed
    load(k + G32U_ST - 1);
    const float* buf = ring + (k % G32U_ST) * SF;
    if (u < 3) {
#pragma unroll 2
      for (int it = 0; it < G32U_VPS / 3; ++it) {
        const float* vec = buf + (3 * it + u) * M;
        float a[8];
        uint64_t b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (EVEN) {
            f2_unpack(*reinterpret_cast<const uint64_t*>(vec + 8 * p + 2 * i), a[2 * i], a[2 * i + 1]);
            b[i] = *reinterpret_cast<const uint64_t*>(vec + 8 * q + 2 * i);
          } else {
            a[2 * i] = vec[8 * p + 2 * i];
            a[2 * i + 1] = vec[8 * p + 2 * i + 1];
            b[i] = f2_pack(vec[8 * q + 2 * i], vec[8 * q + 2 * i + 1]);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint64_t ad = f2_dup(a[i]);
#pragma unroll
          for (int j = 0; j < 4; ++j) ffma2(acc[i][j], ad, b[j]);
        }
      }
    }
    if ((k & 3) == 3) flush();  // 64 vectors of a lane
  }
  flush();
  cp_async_wait<0>();
  __syncthreads();  // every warp is done with its ring: reuse it for the block reduction
  double* const red = sm_gu;
  const int tid = threadIdx.x;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) red[tid * 65 + i * 8 + j] = accd[i][j];
  __syncthreads();
  double* dst = part + (long long)blockIdx.x * 1024;
  for (int e = tid; e < 10 * 64; e += blockDim.x) {
    const int tt = e >> 6, ij = e & 63;
    double sum = 0.0;
    for (int w = 0; w < G32U_WARPS; ++w)
      for (int uu = 0; uu < 3; ++uu) sum += red[(w * 32 + uu * 10 + tt) * 65 + ij];
    const int pp = tt < 4 ? 0 : tt < 7 ? 1 : tt < 9 ? 2 : 3;
    const int qq = tt < 4 ? tt : tt < 7 ? tt - 3 : tt < 9 ? tt - 5 : 3;
    dst[(8 * pp + (ij >> 3)) * 32 + 8 * qq + (ij & 7)] = sum;
  }
}

}  // namespace

// Sum of nblk partials of one 32-wide job (the exact Grams of up to 32 rows).
int launch_gram32_reduce(const double* part, int nblk, int M, double* w, cudaStream_t s) {
  GramJobs J = {};
  J.gs = 4;
  J.n = 1;
  J.start[1] = nblk;
  k_gram_reduce<<<ceil_div(32LL * M * M, 256), 256, 0, s>>>(part, J, 32, 1024, M, w);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

size_t gram_ws_bytes(long long nvec, int M) {
  if (M <= 0) return 4096;
  const GramJobs J = gr_jobs(nvec, M);
  return (size_t)J.start[J.n] * 64 * J.gs * J.gs * sizeof(double) + 4096;
}

int launch_gram(const float* x, long long nvec, int M, long long vs, long long es, double* w, Arena& ws,
                cudaStream_t s) {
  if (M <= 0) return TT_OK;
  if (M > TT_MAX_SMALL) {
    set_error(TT_ERR_UNSUPPORTED, "gram size %d > %d", M, TT_MAX_SMALL);
    return TT_ERR_UNSUPPORTED;
  }
  const GramJobs J = gr_jobs(std::max<long long>(nvec, 1), M);
  const size_t mk = ws.mark();
  double* part = ws.take<double>((size_t)J.start[J.n] * 64 * J.gs * J.gs);
  if (!part) {
    set_error(TT_ERR_NOMEM, "gram workspace");
    return TT_ERR_NOMEM;
  }
  int rc;
  if (J.n > 1) {
    switch (J.gs) {
      case 4: rc = run_gram64<4, true>(x, nvec, M, vs, es, J, part, s); break;
      case 5: rc = run_gram64<5, true>(x, nvec, M, vs, es, J, part, s); break;
      default: rc = run_gram64<6, true>(x, nvec, M, vs, es, J, part, s); break;
    }
  } else {
    switch (J.gs) {
      case 1: rc = run_gram64<1, false>(x, nvec, M, vs, es, J, part, s); break;
      case 2: rc = run_gram64<2, false>(x, nvec, M, vs, es, J, part, s); break;
      case 3: rc = run_gram64<3, false>(x, nvec, M, vs, es, J, part, s); break;
      case 4: rc = run_gram64<4, false>(x, nvec, M, vs, es, J, part, s); break;
      case 5: rc = run_gram64<5, false>(x, nvec, M, vs, es, J, part, s); break;
      default: rc = run_gram64<6, false>(x, nvec, M, vs, es, J, part, s); break;
    }
  }
  TT_TRY(rc);
  k_gram_reduce<<<ceil_div(32LL * M * M, 256), 256, 0, s>>>(part, J, 8 * J.gs, 64LL * J.gs * J.gs, M, w);
  count_launch();
  TT_LAUNCH_CHECK();
  ws.reset(mk);
  return TT_OK;
}

int launch_gram32u(const float* x, long long nvec, int M, double* w, Arena& ws, cudaStream_t s) {
  if (M < 1 || M > 32 || nvec < 1 || (reinterpret_cast<uintptr_t>(x) & 15)) return TT_ERR_UNSUPPORTED;
  const int grid =
      (int)std::max<long long>(1, std::min<long long>(dev_sms(), ceil_div_ll(nvec, (long long)G32U_VPS * G32U_WARPS)));
  const size_t mk = ws.mark();
  double* part = ws.take<double>((size_t)grid * 1024);
  if (!part) {
    set_error(TT_ERR_NOMEM, "gram32u workspace");
    return TT_ERR_NOMEM;
  }
  const size_t shm = g32u_smem(M);
  TT_TRY(smem_optin_k(k_gram32u<true>, g32u_smem(32)));
  TT_TRY(smem_optin_k(k_gram32u<false>, g32u_smem(32)));
  if (M & 1)
    k_gram32u<false><<<grid, 32 * G32U_WARPS, shm, s>>>(x, nvec, M, part);
  else
    k_gram32u<true><<<grid, 32 * G32U_WARPS, shm, s>>>(x, nvec, M, part);
  count_launch();
  TT_LAUNCH_CHECK();
  TT_TRY(launch_gram32_reduce(part, grid, M, w, s));
  ws.reset(mk);
  return TT_OK;
}

}  // namespace ttr
