// CUDA-core kernels of the TT/TR-SVD chain: Gaussian test matrix, Jacobi eigen-solvers, bond permute,
// core folding and the small helpers between them.
#include <float.h>
#include <stdlib.h>
#include <math.h>

#include <algorithm>

#include "kernels.cuh"
#include "philox.cuh"
#include "jacobi_rot.cuh"
#include "bl_solver.cuh"

namespace ttr {

thread_local int g_kernel_launches = 0;

static int num_sms() { return dev_sms(); }

// ---------------------------------------------------------------------------------------
// Philox4x32-10 Gaussian generator (replaces curandGenerateNormal, TT3O:585-587)
// ---------------------------------------------------------------------------------------

__global__ void k_gaussian(float* __restrict__ out, long long rows, long long total, long long ld,
                           unsigned long long seed, unsigned stream_id) {
  const long long ncall = (total + 3) / 4;
  if (ld == rows) {
    // contiguous matrix: element e sits at out[e]; whole float4 stores when aligned
    const bool v4 = (total & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncall;
         c += (long long)gridDim.x * blockDim.x) {
      const float4 gv = philox_normal4((unsigned long long)c, stream_id, seed);
      if (v4) {
        reinterpret_cast<float4*>(out)[c] = gv;
      } else {
        const float g[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
        for (int l = 0; l < 4; ++l)
          if (4 * c + l < total) out[4 * c + l] = g[l];
      }
    }
    return;
  }
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncall;
       c += (long long)gridDim.x * blockDim.x) {
    const float4 gv = philox_normal4((unsigned long long)c, stream_id, seed);
    const float g[4] = {gv.x, gv.y, gv.z, gv.w};
    // element e = row + rows * col; one 64-bit division per call, then step through rows
    long long col = (4 * c) / rows;
    long long row = 4 * c - col * rows;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      if (4 * c + l < total) out[row + ld * col] = g[l];
      if (++row == rows) {
        row = 0;
        ++col;
      }
    }
  }
}

// Rows [row0, row0 + nrows) of the (total_rows x cols) matrix k_gaussian generates (its element
// (i, c) is component e % 4 of Philox call e / 4, e = i + total_rows * c): the block of a
// column-sharded Omega that one rank multiplies with its columns.
__global__ void k_gaussian_rows(float* __restrict__ out, long long row0, long long nrows, long long total_rows,
                                int cols, long long ld, unsigned long long seed, unsigned stream_id) {
  const long long total = nrows * cols;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long c = idx / nrows, i = idx - c * nrows;
    const long long e = row0 + i + total_rows * c;
    const float4 g = philox_normal4((unsigned long long)(e >> 2), stream_id, seed);
    const int l = (int)(e & 3);
    out[i + ld * c] = l == 0 ? g.x : l == 1 ? g.y : l == 2 ? g.z : g.w;
  }
}

int launch_gaussian_rows(float* out, long long row0, long long nrows, long long total_rows, int cols, long long ld,
                         unsigned long long seed, unsigned stream_id, cudaStream_t s) {
  const long long total = nrows * (long long)cols;
  if (total <= 0) return TT_OK;
  k_gaussian_rows<<<(int)std::min<long long>(ceil_div_ll(total, 256), 8LL * num_sms()), 256, 0, s>>>(
      out, row0, nrows, total_rows, cols, ld, seed, stream_id);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

int launch_gaussian(float* out, long long rows, int cols, long long ld, unsigned long long seed,
                    unsigned stream_id, cudaStream_t s) {
  const long long total = rows * (long long)cols;
  if (total <= 0) return TT_OK;
  const long long ncall = (total + 3) / 4;
  const int grid = (int)std::min<long long>(ceil_div_ll(ncall, 256), 8LL * num_sms());
  k_gaussian<<<grid, 256, 0, s>>>(out, rows, total, ld, seed, stream_id);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

// ---------------------------------------------------------------------------------------
// Symmetric eigen-decomposition: parallel cyclic Jacobi (round-robin pairs), FP64
// ---------------------------------------------------------------------------------------
// Single-matrix solver for N <= 64 (bl_solver.cuh): one CTA of bl_shape's warp count, compiled
// for the smallest thread bound that holds it, so that the compiler may give each thread the
// registers it needs (at 1024 threads it has 64 and spills).
template <int MAXT, int VN>
__global__ void __launch_bounds__(MAXT, 1) k_syev_bl(const double* __restrict__ w_in, int N,
                                                   double* __restrict__ evals,
                                                   double* __restrict__ evecs, int max_sweeps,
                                                   DevStatus* st) {
  extern __shared__ __align__(16) double sm_bl[];
  const int sw = bl_solve<VN>(w_in, N, evals, evecs, max_sweeps, sm_bl);
  if (threadIdx.x == 0 && st) {
    atomicMax(&st->sweeps, min(sw, max_sweeps));
    if (sw > max_sweeps) dev_fail(st, TT_ERR_NOCONV, max_sweeps);
  }
}

// Large-N variant (64 < N <= 128) of the Brent-Luk solver.  W alone stays in shared memory: its
// upper triangle packed by rows (row P stored from column P & ~1, so every 2 x 2 block row is a
// 16-byte load), double-buffered (2 x 66.5 KB for N = 128).  The eigenvectors are not updated
// round by round: the rotation warps log each round's renormalised FP64 (c, s) pairs to global
// memory (so the replay's per-round chain has no conversion or renormalisation), and
// k_bl_replay applies them afterwards to the rows of V, one CTA per row (rows are independent),
// with the same moves.  Two warps compute the next round's rotations during the update; every
// W thread's block addresses and the rotation lanes' entry offsets are computed once.
__device__ __forceinline__ int blp_off(int P, int Np) {
  // sum over rows p < P of (Np - (p & ~1)): pairs of rows (2a, 2a + 1) hold 2 (Np - 2a) entries
  const int a = P >> 1;
  return 2 * (a * Np - a * (a - 1)) + (P & 1) * (Np - 2 * a);
}

__global__ void __launch_bounds__(1024) k_syev_blw(const double* __restrict__ w_in, int N,
                                                    double* __restrict__ evals, double2* __restrict__ tlog,
                                                    int* __restrict__ meta, int max_sweeps, DevStatus* st) {
  constexpr int RW0 = 30;  // warps 30, 31 compute the next round's rotations
  constexpr int NE = RW0 * 32;
  extern __shared__ __align__(16) double sm_blw[];
  const int Np = N + (N & 1);
  const int NR = Np - 1;
  const int H = Np / 2;
  const int PS = blp_off(Np, Np);
  double* Wb0 = sm_blw;
  double* Wb1 = Wb0 + PS;
  __shared__ double2 pcs[2][64];
  __shared__ int mv[128], imv[128];
  __shared__ double dg[128];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // offset of entry (P, Q), P <= Q: arithmetic (a few integer ops) rather than a table lookup,
  // which would add a shared-memory load to every access
  auto at = [&](int P, int Q) { return blp_off(P, Np) + (Q - (P & ~1)); };
  for (int P = tid; P < Np; P += blockDim.x) {
    const int x = P % 2 == 0 ? P / 2 : Np - 1 - P / 2;
    const int xn = x == 0 ? 0 : (x == 1 ? NR : x - 1);
    const int Pn = bl_pos(xn, Np);
    mv[P] = Pn;
    imv[Pn] = P;
  }
  __syncthreads();
  for (int e = tid; e < 2 * PS; e += blockDim.x) Wb0[e] = 0.0;
  __syncthreads();
  for (int idx = tid; idx < Np * Np; idx += blockDim.x) {
    const int i = idx / Np, j = idx - (idx / Np) * Np;
    const int Pi = bl_pos(i, Np), Pj = bl_pos(j, Np);
    if (Pi > Pj) continue;
    double v = 0.0;
    if (i < N && j < N) v = 0.5 * (w_in[i + (long long)N * j] + w_in[j + (long long)N * i]);
    Wb0[at(Pi, Pj)] = v;
  }
  double dm = 0.0;
  for (int i = 0; i < N; ++i) dm = fmax(dm, fabs(w_in[i + (long long)N * i]));
  const double inv_s = dm > 0.0 ? 1.0 / dm : 1.0;
  __syncthreads();
  const int rl = tid - NE;  // rotation lane (0..63) on the rotation warps
  if (warp >= RW0 && rl < H) {
    const int k = rl;
    const int i0 = k, i1 = Np - 1 - k;
    float2 r = make_float2(1.0f, 0.0f);
    if (i0 < N && i1 < N)
      r = jacobi_cs32(Wb0[at(2 * k, 2 * k)], Wb0[at(2 * k + 1, 2 * k + 1)], Wb0[at(2 * k, 2 * k + 1)], inv_s);
    double c, sn;
    rot_from_cs32(r, c, sn);
    pcs[0][k] = make_double2(c, sn);
    tlog[k] = make_double2(c, sn);
  }
  __syncthreads();
  const int NWB = H * (H + 1) / 2;
  constexpr int MAXIT = (64 * 65 / 2 + NE - 1) / NE;
  // With at most a block per thread (N <= 86) the rotation warps are the longer part, and their 12 loads
  // would queue behind the other warps' for a third of the round: those wait until they are issued (a
  // round at N = 72: 0.77 us, 0.94 without; at N = 128 the blocks are the longer part, and waiting costs 8 %).
  const bool first = NWB <= NE;
  // per block of this thread: the pair indices (a | b << 8, -1 for none), the offsets of its two
  // rows in W and of its four entries' next-round upper positions (fixed over the rounds)
  int dsc[MAXIT], ldo[MAXIT], sto[MAXIT][4];
#pragma unroll
  for (int u = 0; u < MAXIT; ++u) {
    const int it = tid + u * NE;
    dsc[u] = -1;
    ldo[u] = 0;
    sto[u][0] = sto[u][1] = sto[u][2] = sto[u][3] = 0;
    if (warp < RW0 && it < NWB) {
      int a = 0, rem = it;
      while (rem >= H - a) {
        rem -= H - a;
        ++a;
      }
      const int b = a + rem;
      dsc[u] = a | (b << 8);
      ldo[u] = at(2 * a, 2 * b);
      const int r0 = mv[2 * a], r1 = mv[2 * a + 1], q0 = mv[2 * b], q1 = mv[2 * b + 1];
      sto[u][0] = at(min(r0, q0), max(r0, q0));
      sto[u][1] = at(min(r0, q1), max(r0, q1));
      sto[u][2] = at(min(r1, q0), max(r1, q0));
      sto[u][3] = at(min(r1, q1), max(r1, q1));
    }
  }
  int aP = 0, xP = 0, aQ = 0, xQ = 0;
  int wo[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};  // offsets of the entries the rotation lane reads
  if (warp >= RW0 && rl < H) {
    const int P = imv[2 * rl], Q = imv[2 * rl + 1];
    aP = P >> 1;
    xP = P & 1;
    aQ = Q >> 1;
    xQ = Q & 1;
    const int P0 = 2 * aP, Q0 = 2 * aQ;
    auto ou = [&](int r, int c2) { return at(min(r, c2), max(r, c2)); };
    wo[0] = ou(P0, P0);
    wo[1] = ou(P0, P0 + 1);
    wo[2] = ou(P0 + 1, P0 + 1);
    wo[3] = ou(Q0, Q0);
    wo[4] = ou(Q0, Q0 + 1);
    wo[5] = ou(Q0 + 1, Q0 + 1);
    wo[6] = ou(P0, Q0);
    wo[7] = ou(P0 + 1, Q0);
    wo[8] = ou(P0, Q0 + 1);
    wo[9] = ou(P0 + 1, Q0 + 1);
  }
  int R = 0;
  int sweep = 0;
  bool converged = false;
  for (; sweep < max_sweeps; ++sweep) {
    bool stop = false;
    for (int rnd = 0; rnd < NR; ++rnd, ++R) {
      const int cb = R & 1;
      const double* W = cb ? Wb1 : Wb0;
      double* Wn = cb ? Wb0 : Wb1;
      const double2* cs_ = pcs[cb];
      if (warp < RW0) {
        if (first) asm volatile("bar.sync 1, 1024;" ::: "memory");
#pragma unroll
        for (int u = 0; u < MAXIT; ++u) {
          const int dd = dsc[u];
          if (dd < 0) continue;
          const int a = dd & 255, b = (dd >> 8) & 255;
          const double2 csa = cs_[a], csb = cs_[b];
          const double ca = csa.x, sa = csa.y, cbv = csb.x, sb = csb.y;
          // row 2a + 1 starts (Np - 2a) entries after row 2a (both stored from column 2a)
          const double2 r0v = *reinterpret_cast<const double2*>(&W[ldo[u]]);
          const double2 r1v = *reinterpret_cast<const double2*>(&W[ldo[u] + (Np - 2 * a)]);
          const double w00 = r0v.x, w01 = r0v.y, w11 = r1v.y;
          const double w10 = (a == b) ? w01 : r1v.x;
          const double x00 = ca * w00 - sa * w10, x01 = ca * w01 - sa * w11;
          const double x10 = sa * w00 + ca * w10, x11 = sa * w01 + ca * w11;
          const double y00 = x00 * cbv - x01 * sb, y01 = x00 * sb + x01 * cbv;
          const double y10 = x10 * cbv - x11 * sb, y11 = x10 * sb + x11 * cbv;
          Wn[sto[u][0]] = y00;
          Wn[sto[u][1]] = y01;
          if (a != b) Wn[sto[u][2]] = y10;
          Wn[sto[u][3]] = y11;
        }
      } else {
        const double2 csP = cs_[aP], csQ = cs_[aQ];
        double we[10];
#pragma unroll
        for (int e = 0; e < 10; ++e) we[e] = W[wo[e]];
        if (first) asm volatile("bar.arrive 1, 1024;" ::: "memory");
        const int rn = (rnd + 1 == NR) ? 0 : rnd + 1;
        bool live = rl < H;
        if (Np != N) {
          const int xs = bl_slot(Np - 1, rn, NR);
          live = live && (xs != rl) && (xs != Np - 1 - rl);
        }
        float2 r = make_float2(1.0f, 0.0f);
        if (live) {
          const double cP = csP.x, sP = csP.y, cQ = csQ.x, sQ = csQ.y;
          const double tP0 = xP ? sP : cP, tP1 = xP ? cP : -sP;
          const double tQ0 = xQ ? sQ : cQ, tQ1 = xQ ? cQ : -sQ;
          const double p0 = tP0 * we[0] + tP1 * we[1];
          const double p1 = tP0 * we[1] + tP1 * we[2];
          const double q0 = tQ0 * we[3] + tQ1 * we[4];
          const double q1 = tQ0 * we[4] + tQ1 * we[5];
          const double m0 = tP0 * we[6] + tP1 * we[7];
          const double m1 = tP0 * we[8] + tP1 * we[9];
          r = jacobi_cs32(p0 * tP0 + p1 * tP1, q0 * tQ0 + q1 * tQ1, m0 * tQ0 + m1 * tQ1, inv_s);
        }
        if (rl < H) {
          double c, sn;
          rot_from_cs32(r, c, sn);
          pcs[cb ^ 1][rl] = make_double2(c, sn);
          tlog[(size_t)(R + 1) * H + rl] = make_double2(c, sn);  // rotations of round R + 1
        }
      }
      __syncthreads();
      if (rnd + 1 == NR) {
        int need = 0;
        for (int idx = tid; idx < Np * Np; idx += blockDim.x) {
          const int P = idx / Np, Q = idx - (idx / Np) * Np;
          if (P < Q && jacobi_needed(Wn[at(P, P)], Wn[at(Q, Q)], Wn[at(P, Q)], inv_s)) need = 1;
        }
        if (!__syncthreads_or(need)) stop = true;
      }
    }
    if (stop) {
      converged = true;
      ++sweep;
      break;
    }
  }
  // eigenvalues by rank; meta = [rounds, rank of index 0..N-1, final position of index 0..N-1]
  const double* Wf = (R & 1) ? Wb1 : Wb0;
  if (tid < N) {
    const int P = bl_pos(bl_slot(tid, R, NR), Np);
    dg[tid] = Wf[at(P, P)];
  }
  __syncthreads();
  if (tid < N) {
    double la = dg[tid];
    if (la != la) la = -INFINITY;
    int rank = 0;
    for (int b = 0; b < N; ++b) {
      double lb = dg[b];
      if (lb != lb) lb = -INFINITY;
      rank += (lb > la || (lb == la && b < tid)) ? 1 : 0;
    }
    evals[rank] = dg[tid];
    meta[1 + tid] = rank;
    meta[1 + 128 + tid] = bl_pos(bl_slot(tid, R, NR), Np);
  }
  if (tid == 0) {
    meta[0] = R;
    if (st) {
      atomicMax(&st->sweeps, sweep);
      if (!converged) dev_fail(st, TT_ERR_NOCONV, sweep);
    }
  }
}

// Replays the logged rotations on row i of V (one CTA per row, one thread per pair; V starts as
// the identity with index i at its round-0 position) and writes the eigenvectors by rank.
__global__ void __launch_bounds__(64) k_bl_replay(const double2* __restrict__ tlog, const int* __restrict__ meta,
                                                  int N, double* __restrict__ evecs) {
  __shared__ double vb[2][128];
  __shared__ int mvs[128];
  const int Np = N + (N & 1), H = Np / 2, NR = Np - 1;
  const int i = blockIdx.x, k = threadIdx.x;
  for (int P = k; P < Np; P += blockDim.x) {
    const int x = P % 2 == 0 ? P / 2 : Np - 1 - P / 2;
    const int xn = x == 0 ? 0 : (x == 1 ? NR : x - 1);
    mvs[P] = bl_pos(xn, Np);
    vb[0][P] = (P == bl_pos(i, Np)) ? 1.0 : 0.0;
  }
  __syncthreads();
  const int rounds = meta[0];
  const int m0 = k < H ? mvs[2 * k] : 0, m1 = k < H ? mvs[2 * k + 1] : 0;
  constexpr int U = 8;
  for (int R0 = 0; R0 < rounds; R0 += U) {
    double2 tf[U];
#pragma unroll
    for (int j = 0; j < U; ++j)
      tf[j] = (k < H && R0 + j < rounds) ? tlog[(size_t)(R0 + j) * H + k] : make_double2(1.0, 0.0);
#pragma unroll
    for (int j = 0; j < U; ++j) {
      if (R0 + j >= rounds) break;
      const int cb = (R0 + j) & 1;
      if (k < H) {
        const double c = tf[j].x, sn = tf[j].y;
        const double v0 = vb[cb][2 * k], v1 = vb[cb][2 * k + 1];
        vb[cb ^ 1][m0] = v0 * c - v1 * sn;
        vb[cb ^ 1][m1] = v0 * sn + v1 * c;
      }
      __syncthreads();
    }
  }
  const double* vf = vb[rounds & 1];
  for (int a = k; a < N; a += blockDim.x) evecs[i + (long long)N * meta[1 + a]] = vf[meta[1 + 128 + a]];
}

size_t syev_ws_bytes(int N, int max_sweeps) {
  if (N <= 64) return 0;
  const int Np = N + (N & 1);
  const int sw = max_sweeps > 0 ? max_sweeps : 40;
  return ((size_t)sw * (Np - 1) + 2) * (Np / 2) * sizeof(double2) + (1 + 2 * 128) * sizeof(int) + 1024;
}

int launch_syev(const double* w, int N, double* evals, double* evecs, int max_sweeps, Arena& ws,
                DevStatus* st, cudaStream_t s) {
  if (N <= 0) return TT_OK;
  if (N > TT_MAX_SMALL) {
    set_error(TT_ERR_UNSUPPORTED, "eigen-solver size %d > %d", N, TT_MAX_SMALL);
    return TT_ERR_UNSUPPORTED;
  }
  if (N <= 64) {
    const int Nps = N + (N & 1);
    const size_t shm_bl = 2 * (size_t)Nps * Nps * sizeof(double);
    int iso, warps;
    bl_shape(N, &iso, &warps);
    if (N <= 32) {
      smem_optin_k(k_syev_bl<384, 32>, shm_bl);
      k_syev_bl<384, 32><<<1, 32 * warps, shm_bl, s>>>(w, N, evals, evecs, max_sweeps, st);
    } else if (N <= 46) {
      smem_optin_k(k_syev_bl<768, 48>, shm_bl);
      k_syev_bl<768, 48><<<1, 32 * warps, shm_bl, s>>>(w, N, evals, evecs, max_sweeps, st);
    } else {
      smem_optin_k(k_syev_bl<832, 64>, shm_bl);
      k_syev_bl<832, 64><<<1, 32 * warps, shm_bl, s>>>(w, N, evals, evecs, max_sweeps, st);
    }
    count_launch();
    TT_LAUNCH_CHECK();
    return TT_OK;
  }
  // 64 < N <= 128: packed Brent-Luk on W, eigenvectors by replaying the logged rotations
  const int Np = N + (N & 1), H = Np / 2;
  const int sw = max_sweeps > 0 ? max_sweeps : 40;
  const size_t mk = ws.mark();
  double2* tlog = ws.take<double2>(((size_t)sw * (Np - 1) + 2) * H);
  int* meta = ws.take<int>(1 + 2 * 128);
  if (!tlog || !meta) {
    set_error(TT_ERR_NOMEM, "eigen-solver rotation log");
    return TT_ERR_NOMEM;
  }
  const size_t shm = 2 * (size_t)(2 * (H * Np - H * (H - 1))) * sizeof(double);
  TT_TRY(smem_optin_k(k_syev_blw, shm));
  k_syev_blw<<<1, 1024, shm, s>>>(w, N, evals, tlog, meta, sw, st);
  count_launch();
  TT_LAUNCH_CHECK();
  k_bl_replay<<<N, 64, 0, s>>>(tlog, meta, N, evecs);
  count_launch();
  TT_LAUNCH_CHECK();
  ws.reset(mk);
  return TT_OK;
}

// ---------------------------------------------------------------------------------------
// TR bond permute (r0, r1, n) -> (r1, n, r0), staged through shared memory
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_permute231(const float* __restrict__ in,
                                                    float* __restrict__ out, int r0, int r1,
                                                    long long n, int jt) {
  extern __shared__ float tile[];  // jt * r0 * r1 floats
  const long long j0 = (long long)blockIdx.x * jt;
  const int q = r0 * r1;
  const long long jn = (j0 + jt <= n) ? jt : (n - j0);
  const long long cnt = jn * q;
  const float* src = in + j0 * q;
  for (long long f = threadIdx.x; f < cnt; f += blockDim.x) tile[f] = src[f];
  __syncthreads();
  // out[b + r1*(j + n*a)]: for each a, a contiguous run of r1*jn floats
  for (long long f = threadIdx.x; f < cnt; f += blockDim.x) {
    const int a = (int)(f / (r1 * jn));
    const long long rem = f % (r1 * jn);
    const int b = (int)(rem % r1);
    const long long jj = rem / r1;
    out[(long long)r1 * (j0 + n * a) + rem] = tile[jj * q + a + (long long)r0 * b];
  }
}

int launch_permute231(const float* in, float* out, int r0, int r1, long long n, cudaStream_t s) {
  const int q = r0 * r1;
  if (q <= 0 || n <= 0) return TT_OK;
  int jt = std::max(1, 8192 / q);
  const size_t shm = (size_t)jt * q * sizeof(float);
  k_permute231<<<(int)ceil_div_ll(n, jt), 256, shm, s>>>(in, out, r0, r1, n, jt);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

// ---------------------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------------------
__global__ void k_small_nn(const float* __restrict__ a, long long M, int K, long long lda,
                           const double* __restrict__ b, int N, long long ldb,
                           const double* __restrict__ colscale, int nvalid,
                           float* __restrict__ c, long long ldc) {
  const long long total = M * (long long)N;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx % M;
    const int col = (int)(idx / M);
    double acc = 0.0;
    if (col < nvalid) {
      for (int k = 0; k < K; ++k) acc += (double)a[i + lda * k] * b[k + ldb * col];
      if (colscale) acc *= colscale[col];
    }
    c[i + ldc * col] = (float)acc;
  }
}

int launch_small_nn(const float* a, long long M, int K, long long lda, const double* b, int N,
                    long long ldb, const double* colscale, int nvalid, float* c, long long ldc,
                    cudaStream_t s) {
  const long long total = M * (long long)N;
  if (total <= 0) return TT_OK;
  k_small_nn<<<(int)std::min<long long>(ceil_div_ll(total, 256), 8LL * num_sms()), 256, 0, s>>>(
      a, M, K, lda, b, N, ldb, colscale, nvalid, c, ldc);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

__global__ void k_fold_rows(const float* __restrict__ in, float* __restrict__ out,
                            const double* __restrict__ p, int R, long long ni, int ncols) {
  const long long M = (long long)R * ni;
  const long long total = M * ncols;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long row = idx % M;
    const long long bcol = idx / M;
    const int a = (int)(row % R);
    const long long i = row / R;
    double acc = 0.0;
    for (int ap = 0; ap < R; ++ap)
      acc += p[ap + (long long)R * a] * (double)in[(ap + (long long)R * i) + M * bcol];
    out[idx] = (float)acc;
  }
}

int launch_fold_rows(const float* in, float* out, const double* p, int R, long long ni, int ncols,
                     cudaStream_t s) {
  const long long total = (long long)R * ni * ncols;
  if (total <= 0) return TT_OK;
  k_fold_rows<<<(int)std::min<long long>(ceil_div_ll(total, 256), 8LL * num_sms()), 256, 0, s>>>(
      in, out, p, R, ni, ncols);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

// out (Rout, cols) <- in (Rin, cols), rows Rin..Rout-1 zero (Rin <= Rout), column-major.
__global__ void k_expand_rows(const float* __restrict__ in, int Rin, float* __restrict__ out, int Rout,
                              long long cols) {
  const long long total = (long long)Rout * cols;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long c = idx / Rout;
    const int a = (int)(idx - c * Rout);
    out[idx] = (a < Rin) ? in[a + (long long)Rin * c] : 0.f;
  }
}

int launch_expand_rows(const float* in, int Rin, float* out, int Rout, long long cols, cudaStream_t s) {
  const long long total = (long long)Rout * cols;
  if (total <= 0) return TT_OK;
  k_expand_rows<<<(int)std::min<long long>(ceil_div_ll(total, 256), 8LL * num_sms()), 256, 0, s>>>(
      in, Rin, out, Rout, cols);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

__global__ void k_f64_to_f32_cols(const double* __restrict__ in, long long rows, long long ldin,
                                  int k, float* __restrict__ out, long long ldout, int ncols) {
  const long long total = rows * ncols;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx % rows;
    const int c = (int)(idx / rows);
    out[i + ldout * c] = (c < k) ? (float)in[i + ldin * c] : 0.f;
  }
}

int launch_f64_to_f32_cols(const double* in, long long rows, long long ldin, int k, float* out,
                           long long ldout, int ncols, cudaStream_t s) {
  const long long total = rows * ncols;
  if (total <= 0) return TT_OK;
  k_f64_to_f32_cols<<<(int)std::min<long long>(ceil_div_ll(total, 256), 8LL * num_sms()), 256, 0,
                      s>>>(in, rows, ldin, k, out, ldout, ncols);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

__global__ void k_sigma_vt(const double* __restrict__ evals, const double* __restrict__ v, int n,
                           int k, int kvalid, float* __restrict__ out) {
  const int total = n * k;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const int a = idx % k, j = idx / k;
    out[idx] = (a < kvalid) ? (float)(sqrt(fmax(evals[a], 0.0)) * v[j + (long long)n * a]) : 0.f;
  }
}

int launch_sigma_vt(const double* evals, const double* v, int n, int k, int kvalid, float* out,
                    cudaStream_t s) {
  if (n * k <= 0) return TT_OK;
  k_sigma_vt<<<ceil_div(n * k, 256), 256, 0, s>>>(evals, v, n, k, kvalid, out);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

__global__ void k_inv_sigma(const double* __restrict__ evals, int k, double* __restrict__ cs,
                            double rel_floor) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= k) return;
  const double s0 = sqrt(fmax(evals[0], 0.0));
  const double sa = sqrt(fmax(evals[a], 0.0));
  cs[a] = (sa > rel_floor * s0 && sa > 0.0) ? 1.0 / sa : 0.0;
}

int launch_inv_sigma(const double* evals, int k, double* colscale, double rel_floor, cudaStream_t s) {
  if (k <= 0) return TT_OK;
  k_inv_sigma<<<ceil_div(k, 128), 128, 0, s>>>(evals, k, colscale, rel_floor);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

__global__ void k_ring_core1(const float* __restrict__ u, int n1, int r0, int r1,
                             float* __restrict__ core) {
  const int total = n1 * r0 * r1;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const int a = idx % r0;
    const int i = (idx / r0) % n1;
    const int b = idx / (r0 * n1);
    core[idx] = u[i + (long long)n1 * (a + r0 * b)];
  }
}

int launch_ring_core1(const float* u, int n1, int r0, int r1, float* core, cudaStream_t s) {
  const int total = n1 * r0 * r1;
  if (total <= 0) return TT_OK;
  k_ring_core1<<<ceil_div(total, 256), 256, 0, s>>>(u, n1, r0, r1, core);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

// Sign convention of every basis column: the entry of largest magnitude (lowest row on ties)
// is made positive, and column a of the FP64 companion (the small factor that produced the
// basis) is negated together with it.  TR-SVD's later unfoldings depend on these signs.
__global__ void __launch_bounds__(256) k_canon_cols(float* __restrict__ u, long long m, int r,
                                                    long long ldu, double* __restrict__ comp, int K,
                                                    long long ldc) {
  __shared__ float bv[256];
  __shared__ long long bi[256];
  __shared__ int flip;
  const int a = blockIdx.x;
  if (a >= r) return;
  float best = -1.f;
  long long besti = 0;
  for (long long i = threadIdx.x; i < m; i += blockDim.x) {
    const float v = fabsf(u[i + ldu * a]);
    if (v > best) {
      best = v;
      besti = i;
    }
  }
  bv[threadIdx.x] = best;
  bi[threadIdx.x] = besti;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      const float v2 = bv[threadIdx.x + o];
      const long long i2 = bi[threadIdx.x + o];
      if (v2 > bv[threadIdx.x] || (v2 == bv[threadIdx.x] && i2 < bi[threadIdx.x])) {
        bv[threadIdx.x] = v2;
        bi[threadIdx.x] = i2;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) flip = (bv[0] > 0.f && u[bi[0] + ldu * a] < 0.f) ? 1 : 0;
  __syncthreads();
  if (!flip) return;
  for (long long i = threadIdx.x; i < m; i += blockDim.x) u[i + ldu * a] = -u[i + ldu * a];
  if (comp)
    for (int k = threadIdx.x; k < K; k += blockDim.x) comp[k + ldc * a] = -comp[k + ldc * a];
}

int launch_canon_cols(float* u, long long m, int r, long long ldu, double* comp, int K,
                      long long ldc, cudaStream_t s) {
  if (r <= 0 || m <= 0) return TT_OK;
  k_canon_cols<<<r, 256, 0, s>>>(u, m, r, ldu, comp, K, ldc);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

// Residual energies of the probe columns outside range(Q): out[j] = ||y_j - Q (Q^T y_j)||^2,
// Q (m x ks, FP32, ldq, orthonormal columns), Y0 (m x q, FP64, ldy).  One block per probe
// column; FP64 throughout, so the difference of two nearly equal energies is not formed.
__global__ void __launch_bounds__(256) k_probe_resid(const float* __restrict__ q, long long m, int ks, long long ldq,
                                                     const double* __restrict__ y0, long long ldy,
                                                     double* __restrict__ out) {
  extern __shared__ double sh_pr[];  // c[ks] + 8 warp partials
  double* c = sh_pr;
  double* red = sh_pr + ks;
  const int j = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* y = y0 + (long long)j * ldy;
  // c = Q^T y: warp w takes columns w, w + 8, ...
  for (int a = warp; a < ks; a += 8) {
    const float* qa = q + (long long)a * ldq;
    double t = 0.0;
    for (long long i = lane; i < m; i += 32) t = fma((double)qa[i], y[i], t);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) c[a] = t;
  }
  __syncthreads();
  double acc = 0.0;
  for (long long i = tid; i < m; i += blockDim.x) {
    double r = y[i];
    for (int a = 0; a < ks; ++a) r = fma(-(double)q[i + (long long)a * ldq], c[a], r);
    acc = fma(r, r, acc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w];
    out[j] = t;
  }
}

int launch_probe_resid(const float* q, long long m, int ks, long long ldq, const double* y0, long long ldy, int nq,
                       double* out, cudaStream_t s) {
  if (nq <= 0) return TT_OK;
  const size_t shm = (size_t)(ks + 8) * sizeof(double);
  k_probe_resid<<<nq, 256, shm, s>>>(q, m, ks, ldq, y0, ldy, out);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

__global__ void k_check_finite(const float* __restrict__ x, long long count, int* flag) {
  int bad = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
       i += (long long)gridDim.x * blockDim.x)
    bad |= !isfinite(x[i]);
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}

int launch_check_finite(const float* x, long long count, int* flag, cudaStream_t s) {
  if (count <= 0) return TT_OK;
  k_check_finite<<<(int)std::min<long long>(ceil_div_ll(count, 256), 8LL * num_sms()), 256, 0, s>>>(
      x, count, flag);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

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

__global__ void k_diff_norm(const float* __restrict__ x, const float* __restrict__ y,
                            long long count, double* acc) {
  __shared__ double sh[32];
  double d2 = 0.0, x2 = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
       i += (long long)gridDim.x * blockDim.x) {
    const double xv = x[i];
    const double dv = xv - (y ? (double)y[i] : 0.0);
    d2 += dv * dv;
    x2 += xv * xv;
  }
  d2 = block_sum(d2, sh);
  x2 = block_sum(x2, sh);
  if (threadIdx.x == 0) {
    atomicAdd(&acc[0], d2);
    atomicAdd(&acc[1], x2);
  }
}

int launch_diff_norm(const float* x, const float* y, long long count, double* acc, cudaStream_t s) {
  if (count <= 0) return TT_OK;
  k_diff_norm<<<(int)std::min<long long>(ceil_div_ll(count, 256), 4LL * num_sms()), 256, 0, s>>>(
      x, y, count, acc);
  count_launch();
  TT_LAUNCH_CHECK();
  return TT_OK;
}

}  // namespace ttr
