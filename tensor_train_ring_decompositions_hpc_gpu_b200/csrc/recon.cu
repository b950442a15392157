// Reconstruction error of a train or ring: merged halves of the cores, then one contraction compared with X.
//
// X^[i, J] = sum_{a,b} L[a, i, b] R[b, J, a] over q = r0 rk products, L (r0, P, rk) the merged left cores and
// R (rk, N, r0) the merged right ones.  Everything between the FP32 cores and the two sums is FP64: at a
// relative error of 1e-4 an FP32 X^ moves the result by 3e-6 (its tile loop takes 2.4 ms for a 32^6 tensor at
// ranks 32, this one 3.5).  Bound by the FP64 matrix instructions (mma.m8n8k4.f64, 64 FMAs per clock and SM
// without a register-tiled loop's loads): q FMAs per element of X, 1.85 ms at q = 32, next to one read of X
// (0.66 ms).  X is copied behind the products; read by the lanes that need it the check takes 3.7 ms.
#include <algorithm>

#include "kernels.cuh"

namespace ttr {
namespace {

constexpr int RE_I = 128, RE_J = 64, RE_K = 16;      // block tile, K chunk
constexpr int RE_LI = RE_I + 4, RE_LJ = RE_J + 4;    // row strides: 4 k x 4 columns of a half warp in distinct banks
constexpr int RE_LX = 32 + 8;                        // X: a warp's 32 x 32 entries, 4 rows x 4 pairs in distinct banks
constexpr size_t RE_SMEM = (size_t)2 * RE_K * (RE_LI + RE_LJ) * sizeof(double) + 8 * 32 * RE_LX * sizeof(float);

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(valid ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_t(float* dst, const float* src, bool valid) { cp_async4(dst, src, valid); }
__device__ __forceinline__ void cp_async_t(double* dst, const double* src, bool valid) { cp_async8(dst, src, valid); }

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r += sh[i];
  __syncthreads();
  return r;
}

// acc[0] += sum (X - X^)^2, acc[1] += sum X^2.  8 warps of 32 x 32 entries (4 along i, 2 along J), K chunks of
// 16 double-buffered by cp.async.  The rows of a matrix instruction are J, its columns i, so that a lane's two
// entries are neighbours in X.  TL, TR: FP64 for a merged side, FP32 for a side that is one core.
// Entries past the ends of X are zero, since one side is; not so where the other one is infinite.  ENDS leaves them
// out, which takes registers that the loop wants (32^6: 3.51 -> 3.67 ms): it runs where the sum came out NaN.
template <typename TL, typename TR, bool RING, bool ENDS>
__global__ void __launch_bounds__(256, 2) k_recon_err(const float* __restrict__ x, long long P, long long N,
                                                      const TL* __restrict__ lf, const TR* __restrict__ rf,
                                                      int r0, int rk, double* acc) {
  extern __shared__ __align__(16) double sm_re[];
  TL* const ls = reinterpret_cast<TL*>(sm_re);                              // [2][K][LI]
  TR* const rs = reinterpret_cast<TR*>(sm_re + 2 * RE_K * RE_LI);           // [2][K][LJ]
  float* const xw = reinterpret_cast<float*>(sm_re + 2 * RE_K * (RE_LI + RE_LJ)) + (threadIdx.x >> 5) * 32 * RE_LX;
  __shared__ double sh[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wi = 32 * (warp & 3), wj = 32 * (warp >> 2), lk = lane & 3, lr = lane >> 2;
  const int q = r0 * rk, nk = (q + RE_K - 1) / RE_K;
  const long long pt = (P + RE_I - 1) / RE_I, nt = (N + RE_J - 1) / RE_J, ntiles = pt * nt;
  const long long my = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;  // tiles of this block
  const long long stages = my * nk;
  // stage st: K chunk st % nk of this block's tile st / nk, into buffer st & 1
  auto load = [&](long long st) {
    const long long t = blockIdx.x + (st / nk) * gridDim.x;
    const int k0 = (int)(st % nk) * RE_K;
    const long long i0 = (t % pt) * RE_I, j0 = (t / pt) * RE_J;
    TL* const l = ls + (st & 1) * RE_K * RE_LI;
    TR* const r = rs + (st & 1) * RE_K * RE_LJ;
    {  // L: a row of the chunk (fixed contraction index) per half block, its entries along i
      const int i = tid & 127, kh = tid >> 7;
      const bool in = i0 + i < P;
#pragma unroll
      for (int u = 0; u < RE_K / 2; ++u) {
        const int kk = kh + 2 * u, c = k0 + kk, b = RING ? c / r0 : c, a = RING ? c - b * r0 : 0;
        const bool ok = in && c < q;
        cp_async_t(l + kk * RE_LI + i, ok ? lf + a + r0 * ((i0 + i) + P * b) : lf, ok);
      }
    }
    {  // R: consecutive lanes take consecutive contraction indices (contiguous in a train)
      const int kk = tid & 15, c = k0 + kk, b = RING ? c / r0 : c, a = RING ? c - b * r0 : 0;
      const TR* src = rf + b + rk * ((j0 + (tid >> 4)) + N * a);
      const int nj = c < q ? (int)min((long long)RE_J, N - j0) : 0;
#pragma unroll
      for (int u = 0; u < RE_J / 16; ++u) {
        const int j = (tid >> 4) + 16 * u;
        cp_async_t(r + kk * RE_LJ + j, j < nj ? src + (long long)(16 * rk) * u : rf, j < nj);
      }
    }
  };
  double s[4][4][2];  // tile (J block, i block)
  double d2 = 0.0, x2 = 0.0, e2 = 0.0, y2 = 0.0;
  const bool xv = (P & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  // this warp's part of X, zero outside; copied while its products are formed
  auto load_x = [&](long long i0, long long j0) {
    if (xv) {
      const int i = 4 * (lane & 7);
      const bool in = i0 + i < P;  // P % 4 == 0: four entries or none
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int j = (lane >> 3) + 4 * u;
        const bool ok = in && j0 + j < N;
        cp_async16z(xw + j * RE_LX + i, ok ? x + (i0 + i) + P * (j0 + j) : x, ok);
      }
    } else {
#pragma unroll 4
      for (int j = 0; j < 32; ++j) {
        const bool ok = i0 + lane < P && j0 + j < N;
        cp_async4(xw + j * RE_LX + lane, ok ? x + (i0 + lane) + P * (j0 + j) : x, ok);
      }
    }
  };
  long long i0 = 0, j0 = 0;
  if (stages > 0) load(0);
  cp_async_commit();
  for (long long st = 0; st < stages; ++st) {
    cp_async_wait<0>();
    __syncthreads();  // stage st landed for every thread; buffer (st + 1) & 1 is no longer read
    const int kc = (int)(st % nk);
    if (kc == 0) {
      const long long t = blockIdx.x + (st / nk) * gridDim.x;
      i0 = (t % pt) * RE_I + wi;
      j0 = (t / pt) * RE_J + wj;
      load_x(i0, j0);
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int c = 0; c < 4; ++c) s[p][c][0] = s[p][c][1] = 0.0;
    }
    cp_async_commit();
    if (st + 1 < stages) load(st + 1);
    cp_async_commit();
    const TL* l = ls + (st & 1) * RE_K * RE_LI + lk * RE_LI + wi + lr;
    const TR* r = rs + (st & 1) * RE_K * RE_LJ + lk * RE_LJ + wj + lr;
    const int ksteps = (min(RE_K, q - kc * RE_K) + 3) / 4;  // indices past q are zero
    for (int k = 0; k < ksteps; ++k) {
      double a[4], b[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        a[p] = (double)r[4 * k * RE_LJ + 8 * p];
        b[p] = (double)l[4 * k * RE_LI + 8 * p];
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int c = 0; c < 4; ++c) mma_f64(s[p][c], a[p], b[c]);
    }
    if (kc + 1 < nk) continue;
    cp_async_wait<1>();  // X is here (each thread's own copies), the next chunk may not be
    __syncwarp();
    if constexpr (ENDS) {
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const long long i = i0 + 8 * c + 2 * lk;
          const bool in = j0 + 8 * p + lr < N;
          if (!in || i >= P) s[p][c][0] = 0.0;
          if (!in || i + 1 >= P) s[p][c][1] = 0.0;
        }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int c = 0; c < 4; ++c) {  // entries outside X are zero on both sides
        const float2 v = *reinterpret_cast<const float2*>(xw + (8 * p + lr) * RE_LX + 8 * c + 2 * lk);
        const double a = v.x, b = v.y, da = a - s[p][c][0], db = b - s[p][c][1];
        d2 = fma(da, da, d2);
        x2 = fma(a, a, x2);
        e2 = fma(db, db, e2);
        y2 = fma(b, b, y2);
      }
    __syncwarp();  // before the next tile's X
  }
  d2 = block_sum(d2 + e2, sh);
  x2 = block_sum(x2 + y2, sh);
  if (threadIdx.x == 0) {
    atomicAdd(&acc[0], d2);
    atomicAdd(&acc[1], x2);
  }
}

// C (M x N, FP64) = A (M x K) * B (K x N), column-major, K small: the merge of two cores.  Column n of B lies at
// b + K (n + n / bn * bgap): a part of the last mode of a ring's core.
template <typename TA, typename TB>
__global__ void __launch_bounds__(128) k_merge(const TA* __restrict__ a, long long M, int K, const TB* __restrict__ b,
                                               long long N, long long bn, long long bgap,
                                               double* __restrict__ c) {
  constexpr int NC = 8;
  __shared__ double bs[64][NC];
  const long long nblk = (M + 127) / 128, tiles = nblk * ((N + NC - 1) / NC);
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const long long i = (t % nblk) * 128 + threadIdx.x, n0 = (t / nblk) * NC;
    double acc[NC];
#pragma unroll
    for (int u = 0; u < NC; ++u) acc[u] = 0.0;
    for (int k0 = 0; k0 < K; k0 += 64) {
      __syncthreads();
      for (int f = threadIdx.x; f < 64 * NC; f += 128) {
        const int kk = f & 63, u = f >> 6;
        const long long n = n0 + u;
        bs[kk][u] = (n < N && k0 + kk < K) ? (double)b[(k0 + kk) + (long long)K * (n + (bgap ? n / bn * bgap : 0))] : 0.0;
      }
      __syncthreads();
      if (i < M) {
        const int kmax = min(64, K - k0);
#pragma unroll 8  // loads of A in flight: a merge of small cores is all latency
        for (int kk = 0; kk < kmax; ++kk) {
          const double av = (double)a[i + M * (long long)(k0 + kk)];
#pragma unroll
          for (int u = 0; u < NC; ++u) acc[u] = fma(av, bs[kk][u], acc[u]);
        }
      }
    }
    if (i < M) {
#pragma unroll
      for (int u = 0; u < NC; ++u)
        if (n0 + u < N) c[i + M * (n0 + u)] = acc[u];
    }
  }
}

template <typename TL, typename TR, bool RING, bool ENDS>
int run_recon(const float* x, long long P, long long N, const void* lf, const void* rf, int r0, int rk, double* acc,
              cudaStream_t s) {
  const long long tiles = ceil_div_ll(P, RE_I) * ceil_div_ll(N, RE_J);
  const int grid = (int)std::min<long long>(tiles, 2LL * dev_sms());
  TT_TRY(smem_optin_k(k_recon_err<TL, TR, RING, ENDS>, RE_SMEM));
  k_recon_err<TL, TR, RING, ENDS><<<grid, 256, RE_SMEM, s>>>(x, P, N, static_cast<const TL*>(lf),
                                                             static_cast<const TR*>(rf), r0, rk, acc);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}
template <typename TL, typename TR>
int run_recon(const float* x, long long P, long long N, const void* lf, const void* rf, int r0, int rk, bool ends,
              double* acc, cudaStream_t s) {
  if (r0 == 1) return ends ? run_recon<TL, TR, false, true>(x, P, N, lf, rf, r0, rk, acc, s)
                           : run_recon<TL, TR, false, false>(x, P, N, lf, rf, r0, rk, acc, s);
  return ends ? run_recon<TL, TR, true, true>(x, P, N, lf, rf, r0, rk, acc, s)
              : run_recon<TL, TR, true, false>(x, P, N, lf, rf, r0, rk, acc, s);
}

}  // namespace

long long recon_tiles(long long P, long long N) { return ceil_div_ll(P, RE_I) * ceil_div_ll(N, RE_J); }

int launch_recon_err(const float* x, long long P, long long N, const void* lf, bool l64, const void* rf, bool r64,
                     int r0, int rk, bool ends, double* acc, cudaStream_t s) {
  if (l64) return r64 ? run_recon<double, double>(x, P, N, lf, rf, r0, rk, ends, acc, s)
                      : run_recon<double, float>(x, P, N, lf, rf, r0, rk, ends, acc, s);
  return r64 ? run_recon<float, double>(x, P, N, lf, rf, r0, rk, ends, acc, s)
             : run_recon<float, float>(x, P, N, lf, rf, r0, rk, ends, acc, s);
}

int launch_merge(const void* a, bool a64, long long M, int K, const void* b, bool b64, long long N, long long bn,
                 long long bgap, double* c, cudaStream_t s) {
  if (M <= 0 || N <= 0) return TT_OK;
  const int grid = (int)std::min<long long>(ceil_div_ll(M, 128) * ceil_div_ll(N, 8), 64LL * dev_sms());
  const double* a8 = static_cast<const double*>(a);
  const float* a4 = static_cast<const float*>(a);
  const double* b8 = static_cast<const double*>(b);
  const float* b4 = static_cast<const float*>(b);
  if (a64 && b64) k_merge<<<grid, 128, 0, s>>>(a8, M, K, b8, N, bn, bgap, c);
  else if (a64) k_merge<<<grid, 128, 0, s>>>(a8, M, K, b4, N, bn, bgap, c);
  else if (b64) k_merge<<<grid, 128, 0, s>>>(a4, M, K, b8, N, bn, bgap, c);
  else k_merge<<<grid, 128, 0, s>>>(a4, M, K, b4, N, bn, bgap, c);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

}  // namespace ttr
