// rbrp_adjoint.cu - loss and adjoint of the fixed-skeleton interpolative
// decomposition, FP32 kernels (no counterpart in the reference).
//
// With the skeleton S held fixed, C = A(:, S) (m x k), B = A(:, rd) (m x nc)
// and T = C^+ B (the k x nc interpolation matrix of the last fixed-skeleton
// run, T = R11^{-1} R12), the loss is
//     L = ||E||_F^2 + ||T w||^2,   E = B - C T,   w = dW(rd).
// Its gradient (T optimal for the first term, so only the second term sees
// dT = -C^+ dC T + (C^T C)^{-1} dC^T E + C^+ dB), with u = T w and
// z = (C^T C)^{-1} u = R11^{-1} R11^{-T} u:
//     dL/dB = 2 E + 2 (C z) w^T
//     dL/dC = -2 E T^T - 2 (C z) u^T + 2 (E w) z^T.
// Nothing of the forward factorisation is stored: R11 and T come from the
// handle's last run (the caller recomputes it for the backward), C and B are
// read from A through perm.  The two products E = B - C T and E T^T run on the
// tensor cores (tcgen05, 3xTF32, rbrp_gemm_tc.cuh) with the loss terms, E w and
// the rank-one terms fused into their epilogues (the handle's variant 1 keeps
// them as 128 x 128-tiled FP32 FFMA GEMMs); z is a double-float triangular
// solve by one cluster of CTAs.
//
// Tensor-core operand layouts (K-major, leading dimensions rounded up to 4
// floats for TMA):
//   E = B - C T:  M = rd columns c, N = rows r, K = skeleton index t
//                 X = T (k x nc, ld kp), Y = C^T (k x m, ld kp, TF32 hi / lo)
//                 written as E^T (nc x m, ld ncp): the drain lanes run along c
//   E T^T:        M = rows r, N = skeleton index t, K = rd columns c
//                 X = E^T, Y = T^T (nc x k, ld ncp, TF32 hi / lo)
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "rbrp_internal.h"
#include "rbrp_df.cuh"
#include "rbrp_gemm.cuh"
#include "rbrp_gemm_tc.cuh"

namespace cg = cooperative_groups;

namespace rbrp {
namespace {

constexpr int PARTS = 16;      // split of the GEMV contractions

// Tr[t * nc + c] = T[t + c * k] (row major copy) and Tc = FP32 T (column major);
// wr[c] = W[perm[k + c]].
__global__ void k_adj_prep(const double* __restrict__ T, int k, int nc, const float* __restrict__ W,
                           const int* __restrict__ perm, float* __restrict__ Tr, float* __restrict__ Tc,
                           float* __restrict__ wr) {
  __shared__ float tile[32][33];
  const int t0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
  for (int q = ty; q < 32; q += 8) {
    const int t = t0 + tx, c = c0 + q;
    float v = 0.f;
    if (t < k && c < nc) {
      v = (float)T[t + (int64_t)c * k];
      Tc[t + (int64_t)c * k] = v;
    }
    tile[q][tx] = v;
  }
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int t = t0 + q, c = c0 + tx;
    if (t < k && c < nc) Tr[(int64_t)t * nc + c] = tile[tx][q];
  }
  if (blockIdx.x == 0)
    for (int c = c0 + threadIdx.x; c < min(nc, c0 + 32); c += blockDim.x) wr[c] = W[perm[k + c]];
}

// upart[p][t] = sum over columns c of part p of T[t, c] wr[c] (double-float, as float2);
// T is FP32, k x nc, column major with leading dimension ldt >= k
__global__ void k_adj_u(const float* __restrict__ Tc, int64_t ldt, int k, int nc, const float* __restrict__ wr,
                        float2* __restrict__ upart) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = blockIdx.y, chunk = (nc + PARTS - 1) / PARTS;
  const int cb = p * chunk, ce = min(nc, cb + chunk);
  if (t >= k) return;
  float hi = 0.f, lo = 0.f;
  for (int c = cb; c < ce; ++c) {
    const float prod = Tc[t + (int64_t)c * ldt] * wr[c];
    const float e = fmaf(Tc[t + (int64_t)c * ldt], wr[c], -prod);
    const float s = hi + prod, z = s - hi;
    lo += ((hi - (s - z)) + (prod - z)) + e;
    hi = s;
  }
  upart[(int64_t)p * k + t] = make_float2(hi, lo);
}

// out[i] = sum of the PARTS partials (fixed order), as float and (if out_df)
// double-float.
__global__ void k_adj_sum_parts(const float2* __restrict__ part, int len, float* __restrict__ out,
                                float2* __restrict__ out_df) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= len) return;
  dfl s = {part[i].x, part[i].y};
  for (int p = 1; p < PARTS; ++p) {
    const float2 v = part[(int64_t)p * len + i];
    s = df_add(s, {v.x, v.y});
  }
  s = df_two_sum(s.hi, s.lo);
  out[i] = s.hi;
  if (out_df) out_df[i] = make_float2(s.hi, s.lo);
}

// out[i] = sum over p < nparts of part[p][i] (fixed order, double-float).
__global__ void k_adj_sum_rows(const float2* __restrict__ part, int nparts, int len, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= len) return;
  dfl s = {0.f, 0.f};
  for (int p = 0; p < nparts; ++p) {
    const float2 v = part[(int64_t)p * len + i];
    s = df_add(s, {v.x, v.y});
  }
  out[i] = df_two_sum(s.hi, s.lo).hi;
}

// R11 (FP64, row major, ld ldr, upper) as double-float pairs, row major ld k, with R11^T
// in the lower triangle: both directions of the solve then read rows.
__global__ void k_adj_split_r(const double* __restrict__ R, int64_t ldr, int k, float2* __restrict__ Rdf) {
  __shared__ float2 tile[32][33];
  const int c0 = blockIdx.x * 32, a0 = blockIdx.y * 32;
  if (a0 > c0) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int q = ty; q < 32; q += 8) {
    const int a = a0 + q, c = c0 + tx;
    if (a < k && c < k && c >= a) {
      const double x = R[(int64_t)a * ldr + c];
      const float hi = (float)x;
      const float2 v = make_float2(hi, (float)(x - (double)hi));
      Rdf[(int64_t)a * k + c] = v;
      tile[q][tx] = v;
    }
  }
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int c = c0 + q, a = a0 + tx;
    if (c < k && a < c) Rdf[(int64_t)c * k + a] = tile[tx][q];
  }
}

// z = R11^{-1} R11^{-T} u in double-float, one kernel per direction.  Rows are taken in the
// order of the substitution (q = row, backward k - 1 - row) in blocks of 32; thread g of a
// cluster of 8 CTAs has the rows q = g, g + 4096, ... in shared memory.  A step: the warp
// whose lanes have the block's rows solves the 32 x 32 triangle (the lane of row q finishes
// x_q, every later lane subtracts its term) and sends the solution to all 8 CTAs; one
// cluster barrier; every thread subtracts the block's terms from its later rows.  The
// triangle of the next block, its reciprocals and the entries that a thread's first later
// row needs are loaded before the barrier.
// Bound by the chain of k substitutions (about 3,500 clocks per 32).  A launch per block
// and direction, every CTA solving the triangle for itself, took 17.6 and 14.3 us a block
// (4.1 ms at k = 4096); each row's operations and their order are the same.
constexpr int ZC = 8;              // CTAs of the cluster
constexpr int ZT = 512;            // threads per CTA
constexpr int ZG = ZC * ZT;

template <bool BACK>
__global__ void __cluster_dims__(ZC, 1, 1) __launch_bounds__(ZT)
k_adj_zsolve(const float2* __restrict__ R, int k, const float2* __restrict__ rhs, float2* __restrict__ sol,
             float* __restrict__ z) {
  extern __shared__ float2 zr[];                // [row of the thread][thread]: right-hand side
  __shared__ dfl xb[2][32];                     // the block's solution, by step parity
  __shared__ dfl tri[2][32][33];                // coefficient of solved a in row c
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = (int)cl.block_rank() * ZT + tid;
  const int nt = (k + 31) / 32;
  auto row = [&](int q) { return BACK ? k - 1 - q : q; };
  // what row q (later) takes of the solved p
  auto coef = [&](int p, int q) { return __ldg(R + (int64_t)row(p) * k + row(q)); };
  for (int r = 0; g + r * ZG < k; ++r) zr[r * ZT + tid] = rhs[row(g + r * ZG)];
  dfl rinv = {0.f, 0.f};
  auto mine = [&](int t) { return (32 * t) % ZG / 32 == g / 32; };   // the warp has block t
  auto load_tri = [&](int t) {
    const int q0 = 32 * t, q = q0 + lane;
    for (int a = 0; a < 32; ++a) {
      const float2 v = q < k && a <= lane ? coef(q0 + a, q) : make_float2(a == lane ? 1.f : 0.f, 0.f);
      tri[t & 1][a][lane] = {v.x, v.y};
    }
    rinv = df_recip(tri[t & 1][lane][lane]);
    __syncwarp();
  };
  if (mine(0)) load_tri(0);
  cl.sync();                                    // every CTA runs before anything is sent to it
  for (int t = 0; t < nt; ++t) {
    const int q0 = 32 * t, jl = min(32, k - q0);
    if (mine(t)) {
      dfl b = {0.f, 0.f};
      if (lane < jl) {
        const float2 v = zr[q0 / ZG * ZT + tid];
        b = {v.x, v.y};
      }
      dfl x = {0.f, 0.f};
      for (int a = 0; a < jl; ++a) {
        if (lane == a) x = df_mul(b, rinv);
        const dfl xa = {__shfl_sync(0xffffffffu, x.hi, a), __shfl_sync(0xffffffffu, x.lo, a)};
        if (lane > a && lane < jl) b = df_fms(b, tri[t & 1][a][lane], xa);
      }
#pragma unroll
      for (int c = 0; c < ZC; ++c) cl.map_shared_rank(&xb[0][0], c)[32 * (t & 1) + lane] = x;
      if (lane < jl) {
        const int o = row(q0 + lane);
        if (BACK) z[o] = x.hi;
        else sol[o] = make_float2(x.hi, x.lo);
      }
    }
    if (t + 1 < nt && mine(t + 1)) load_tri(t + 1);
    // the first of the thread's rows behind the block
    int r = q0 / ZG;
    if (g + r * ZG < q0 + 32) ++r;
    const int q1 = g + r * ZG;
    float2 cf[32];
    if (q1 < k) {
#pragma unroll
      for (int a = 0; a < 32; ++a) cf[a] = coef(q0 + a, q1);   // a block before a later row is whole
    }
    cl.sync();
    auto apply = [&](int at) {                  // in order of rising rows, both directions
      const float2 w = zr[at];
      dfl v = {w.x, w.y};
#pragma unroll
      for (int a = 0; a < 32; ++a) {
        const int aa = BACK ? 31 - a : a;
        v = df_fms(v, {cf[aa].x, cf[aa].y}, xb[t & 1][aa]);
      }
      zr[at] = make_float2(v.hi, v.lo);
    };
    if (q1 < k) apply(r * ZT + tid);
    for (++r; g + r * ZG < k; ++r) {
#pragma unroll
      for (int a = 0; a < 32; ++a) cf[a] = coef(q0 + a, g + r * ZG);
      apply(r * ZT + tid);
    }
  }
  cl.sync();                                    // no CTA leaves while another may still send to it
}

// z (FP32) = R11^{-1} R11^{-T} u; ys holds k double-float scratch values.
rbrp_status solve_z(rbrp_handle h, const float2* Rdf, int k, const float2* udf, float2* ys, float* z) {
  const size_t smem = (size_t)((k + ZG - 1) / ZG) * ZT * sizeof(float2);
  // one limit for every k (the attribute is the process's): k <= 196608, whose R11 alone is 309 GB
  constexpr int lim = 192 * 1024;
  rbrp_status s = cuda_check(h, cudaFuncSetAttribute(k_adj_zsolve<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     lim), "cudaFuncSetAttribute(k_adj_zsolve)");
  if (s == RBRP_OK)
    s = cuda_check(h, cudaFuncSetAttribute(k_adj_zsolve<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim),
                   "cudaFuncSetAttribute(k_adj_zsolve)");
  if (s != RBRP_OK) return s;
  k_adj_zsolve<false><<<ZC, ZT, smem, h->stream>>>(Rdf, k, udf, ys, nullptr);
  k_adj_zsolve<true><<<ZC, ZT, smem, h->stream>>>(Rdf, k, ys, nullptr, z);
  return cuda_check(h, cudaGetLastError(), "k_adj_zsolve");
}

// czpart[p][r] = sum over the part-p skeleton columns t of A[r, perm[t]] z[t]
__global__ void k_adj_cz(const float* __restrict__ A, int64_t lda, int m, int k, const int* __restrict__ perm,
                         const float* __restrict__ z, float2* __restrict__ czpart) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = blockIdx.y, chunk = (k + PARTS - 1) / PARTS;
  const int tb = p * chunk, te = min(k, tb + chunk);
  if (r >= m) return;
  float hi = 0.f, lo = 0.f;
  for (int t = tb; t < te; ++t) {
    const float a = A[r + (int64_t)perm[t] * lda];
    const float prod = a * z[t];
    const float e = fmaf(a, z[t], -prod);
    const float s = hi + prod, zz = s - hi;
    lo += ((hi - (s - zz)) + (prod - zz)) + e;
    hi = s;
  }
  czpart[(int64_t)p * m + r] = make_float2(hi, lo);
}

// E = B - C T for a 128 x 128 tile: E stored (if Eout), ||E||^2 and E w row
// sums as per-tile partials, and G(:, rd) = scale * 2 (E + (C z) w^T).
__global__ void __launch_bounds__(GT) k_adj_gemm1(const float* __restrict__ A, int64_t lda, int m, int k, int nc,
                                                  const int* __restrict__ perm, const float* __restrict__ Tr,
                                                  const float* __restrict__ wr, const float* __restrict__ cz,
                                                  float* __restrict__ Eout, float* __restrict__ G, int64_t ldg,
                                                  float scale, float2* __restrict__ loss_part,
                                                  float2* __restrict__ ew_part) {
  __shared__ GemmSmem sm;
  __shared__ float2 red[GT];
  const int r0 = blockIdx.x * GTILE, c0 = blockIdx.y * GTILE;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  float acc[8][8];
  gemm_tile(sm, LoadC{A, lda, perm, m, k}, LoadRowMajor{Tr, k, nc}, k, r0, c0, acc);
  dfl sq = {0.f, 0.f};
  float ew[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) ew[i] = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = c0 + tile_col(tx, j);
    if (c >= nc) continue;
    const int col = perm[k + c];
    const float w = wr[c];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = r0 + tile_row(ty, i);
      if (r >= m) continue;
      const float e = A[r + (int64_t)col * lda] - acc[i][j];
      df_acc_prod(sq, e, e);
      ew[i] = fmaf(e, w, ew[i]);
      if (Eout) Eout[r + (int64_t)c * m] = e;
      if (G) G[r + (int64_t)col * ldg] = scale * 2.f * fmaf(cz[r], w, e);
    }
  }
  // row sums of E w over the tile's 16 column groups: through shared memory, fixed order
  float* ews = reinterpret_cast<float*>(&sm);  // the staging buffers are idle now
#pragma unroll
  for (int i = 0; i < 8; ++i) ews[tile_row(ty, i) * 16 + tx] = ew[i];
  red[tid] = make_float2(sq.hi, sq.lo);
  __syncthreads();
  if (tid < GTILE) {
    float s = 0.f;
    for (int q = 0; q < 16; ++q) s += ews[tid * 16 + q];
    if (r0 + tid < m) ew_part[(int64_t)blockIdx.y * m + r0 + tid] = make_float2(s, 0.f);
  }
  if (tid == 0) {
    dfl t = {red[0].x, red[0].y};
    for (int q = 1; q < GT; ++q) t = df_add(t, {red[q].x, red[q].y});
    loss_part[blockIdx.y * gridDim.x + blockIdx.x] = make_float2(t.hi, t.lo);
  }
}

// G(:, S) = scale * (-2 E T^T - 2 (C z) u^T + 2 (E w) z^T) for a 128 x 128 tile.
__global__ void __launch_bounds__(GT) k_adj_gemm2(const float* __restrict__ E, int m, int k, int nc,
                                                  const int* __restrict__ perm, const float* __restrict__ Tc,
                                                  const float* __restrict__ cz, const float* __restrict__ ew,
                                                  const float* __restrict__ u, const float* __restrict__ z,
                                                  float* __restrict__ G, int64_t ldg, float scale) {
  __shared__ GemmSmem sm;
  const int r0 = blockIdx.x * GTILE, c0 = blockIdx.y * GTILE;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  float acc[8][8];
  // E T^T: contraction over the nc rd columns; T^T (nc x k) row major is T column major
  gemm_tile(sm, LoadE{E, m, nc}, LoadRowMajor{Tc, nc, k}, nc, r0, c0, acc);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int t = c0 + tile_col(tx, j);
    if (t >= k) continue;
    const int col = perm[t];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = r0 + tile_row(ty, i);
      if (r >= m) continue;
      const float g = -2.f * acc[i][j] - 2.f * cz[r] * u[t] + 2.f * ew[r] * z[t];
      G[r + (int64_t)col * ldg] = scale * g;
    }
  }
}

__global__ void k_adj_loss(const float2* __restrict__ loss_part, int nparts, const float2* __restrict__ udf, int k,
                           double* __restrict__ out) {
  __shared__ float2 red[256];
  dfl s = {0.f, 0.f};
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) s = df_add(s, {loss_part[i].x, loss_part[i].y});
  dfl su = {0.f, 0.f};
  for (int i = threadIdx.x; i < k; i += blockDim.x) {
    const dfl v = {udf[i].x, udf[i].y};
    su = df_add(su, df_mul(v, v));
  }
  red[threadIdx.x] = make_float2(s.hi, s.lo);
  __syncthreads();
  if (threadIdx.x == 0) {
    dfl t = {red[0].x, red[0].y};
    for (int q = 1; q < (int)blockDim.x; ++q) t = df_add(t, {red[q].x, red[q].y});
    out[0] = (double)t.hi + (double)t.lo;
  }
  __syncthreads();
  red[threadIdx.x] = make_float2(su.hi, su.lo);
  __syncthreads();
  if (threadIdx.x == 0) {
    dfl t = {red[0].x, red[0].y};
    for (int q = 1; q < (int)blockDim.x; ++q) t = df_add(t, {red[q].x, red[q].y});
    out[1] = (double)t.hi + (double)t.lo;
  }
}

// ---------------------------------------------------------------------------
// tensor-core path
// ---------------------------------------------------------------------------
// Tx (k x nc, ld kp) = FP32 T; T^T hi / lo (nc x k, ld ncp) = tf32_rn(t), tf32_rn(t - hi)
// from the FP64 T; wr[c] = W[perm[k + c]].  32 x 32 tiles through shared memory.
__global__ void k_adj_prep_tc(const double* __restrict__ T, int k, int nc, int kp, int ncp,
                              const float* __restrict__ W, const int* __restrict__ perm, float* __restrict__ Tx,
                              float* __restrict__ Trh, float* __restrict__ Trl, float* __restrict__ wr) {
  __shared__ double tile[32][33];
  const int t0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
  for (int q = ty; q < 32; q += 8) {
    const int t = t0 + tx, c = c0 + q;
    double v = 0.0;
    if (t < k && c < nc) {
      v = T[t + (int64_t)c * k];
      Tx[t + (int64_t)c * kp] = (float)v;
    }
    tile[q][tx] = v;
  }
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int t = t0 + q, c = c0 + tx;
    if (t < k && c < nc) {
      const double v = tile[tx][q];
      const float h = tf32_rn((float)v);
      Trh[c + (int64_t)t * ncp] = h;
      Trl[c + (int64_t)t * ncp] = tf32_rn((float)(v - (double)h));
    }
  }
  if (blockIdx.x == 0)
    for (int c = c0 + threadIdx.x; c < min(nc, c0 + 32); c += blockDim.x) wr[c] = W[perm[k + c]];
}

// C^T hi / lo (k x m, ld kp): element (t, r) = A[r, perm[t]] split by tf32_split.
__global__ void k_adj_gather_ct(const float* __restrict__ A, int64_t lda, const int* __restrict__ perm, int k,
                                int m, int kp, float* __restrict__ Cth, float* __restrict__ Ctl) {
  __shared__ float tile[32][33];
  const int r0 = blockIdx.x * 32, t0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int q = ty; q < 32; q += 8) {
    const int r = r0 + tx, t = t0 + q;
    tile[q][tx] = (r < m && t < k) ? A[r + (int64_t)perm[t] * lda] : 0.f;
  }
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int t = t0 + tx, r = r0 + q;
    if (t < k && r < m) {
      float h, l;
      tf32_split(tile[tx][q], h, l);
      Cth[t + (int64_t)r * kp] = h;
      Ctl[t + (int64_t)r * kp] = l;
    }
  }
}

// Per-CTA reduction buffers of the E epilogue (one instance per CTA).
__device__ __forceinline__ float* epi_ew_buf() {
  __shared__ float buf[64 * 4];  // [row slot][lane quarter]
  return buf;
}
__device__ __forceinline__ float2* epi_sq_buf() {
  __shared__ float2 buf[8];      // [drain warp]
  return buf;
}

// E = B - C T on a (128 rd columns) x (64 rows) tile: E^T stored (when Et), ||E||^2
// and the row sums of E w as per-CTA partials, G(:, rd) = scale * 2 (E + (C z) w^T).
// A thread has 32 rows of one column, which it reads and writes by 16 bytes where the
// columns start on 16, else by element (32 lines per instruction).  By element, with a
// shuffle tree per row and E w summed for the loss alone too, the 8192 x 4096 x 4096
// product took 2.54 ms, now 2.08 (E T^T, with a plain epilogue: 1.90).
struct EpiE {
  const float* A;
  int64_t lda;
  const int* perm;
  int k, m, nc;
  const float* wr;
  const float* cz;
  float* Et;
  int64_t ldet;
  float* G;
  int64_t ldg;
  float scale;
  float2* loss_part;
  float2* ew_part;
  bool vecA, vecG;   // columns start on 16 bytes

  __device__ void operator()(int c, int r0, const float (&hi)[32], const float (&lo)[32], int dw) const {
    float* s_ew = epi_ew_buf();
    float2* s_sq = epi_sq_buf();
    const int lane = threadIdx.x & 31, quarter = (c & 127) >> 5, ch = dw >> 2;
    const bool vc = c < nc;
    const float w = vc ? wr[c] : 0.f;
    const int64_t col = vc ? (int64_t)perm[k + c] : 0;
    const bool whole = vc && r0 + 32 <= m;
    const float* a = A + r0 + col * lda;
    float e[32];
    if (whole && vecA) {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(a + j);
        e[j] = x.x, e[j + 1] = x.y, e[j + 2] = x.z, e[j + 3] = x.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) e[j] = vc && r0 + j < m ? a[j] : 0.f;
    }
    dfl sq = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      e[j] = vc && r0 + j < m ? (e[j] - hi[j]) - lo[j] : 0.f;
      df_acc_prod(sq, e[j], e[j]);
    }
    if (Et) {   // E w and the outputs: only for the gradient
      if (vc) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (r0 + j < m) Et[c + (int64_t)(r0 + j) * ldet] = e[j];
      }
      float* g = G + r0 + col * ldg;
      if (whole && vecG) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 x = *reinterpret_cast<const float4*>(cz + r0 + j);
          *reinterpret_cast<float4*>(g + j) =
              make_float4(scale * 2.f * fmaf(x.x, w, e[j]), scale * 2.f * fmaf(x.y, w, e[j + 1]),
                          scale * 2.f * fmaf(x.z, w, e[j + 2]), scale * 2.f * fmaf(x.w, w, e[j + 3]));
        }
      } else if (vc) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (r0 + j < m) g[j] = scale * 2.f * fmaf(cz[r0 + j], w, e[j]);
      }
      // row sums over the warp's 32 columns: a shuffle reduce-scatter, lane j gets row j
#pragma unroll
      for (int j = 0; j < 32; ++j) e[j] *= w;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (j < o) {
            const float keep = upper ? e[j + o] : e[j], send = upper ? e[j] : e[j + o];
            e[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        }
      }
      s_ew[(ch * 32 + lane) * 4 + quarter] = e[0];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const dfl t = {__shfl_xor_sync(0xffffffffu, sq.hi, o), __shfl_xor_sync(0xffffffffu, sq.lo, o)};
      sq = df_add(sq, t);
    }
    if (lane == 0) s_sq[dw] = make_float2(sq.hi, sq.lo);
  }

  // after the CTA barrier: fixed-order sums of the shared partials
  __device__ void finish(bool ok) const {
    if (!ok) return;
    const float* s_ew = epi_ew_buf();
    const float2* s_sq = epi_sq_buf();
    const int t = threadIdx.x;
    if (t < 64) {
      const int r = blockIdx.y * 64 + t;
      if (Et && r < m) {
        const float s = ((s_ew[t * 4] + s_ew[t * 4 + 1]) + s_ew[t * 4 + 2]) + s_ew[t * 4 + 3];
        ew_part[(int64_t)blockIdx.x * m + r] = make_float2(s, 0.f);
      }
    } else if (t == 64) {
      dfl a = {s_sq[0].x, s_sq[0].y};
      for (int q = 1; q < 8; ++q) a = df_add(a, {s_sq[q].x, s_sq[q].y});
      loss_part[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = make_float2(a.hi, a.lo);
    }
  }
};

// G(:, S) = scale * (-2 E T^T - 2 (C z) u^T + 2 (E w) z^T) on a (128 rows) x (64 skeleton) tile.
struct EpiG {
  const int* perm;
  int m, k;
  const float* cz;
  const float* ew;
  const float* u;
  const float* z;
  float* G;
  int64_t ldg;
  float scale;

  __device__ void operator()(int r, int a0, const float (&hi)[32], const float (&lo)[32], int) const {
    if (r >= m) return;
    const float czr = cz[r], ewr = ew[r];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int a = a0 + j;
      if (a < k) {
        const float g = -2.f * (hi[j] + lo[j]) - 2.f * czr * u[a] + 2.f * ewr * z[a];
        G[r + (int64_t)perm[a] * ldg] = scale * g;
      }
    }
  }
  __device__ void finish(bool) const {}
};

size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace
}  // namespace rbrp

namespace rbrp {
namespace {

// The tensor-core form of the loss and gradient (same outputs as the FFMA kernels).
rbrp_status adjoint_tc(rbrp_handle h, int m, int k, int nc, int kp, int ncp, const float* dA, int64_t lda,
                       const float* dW, float scale, float* dG, int64_t ldg, double* loss, float* Trh, float* Trl,
                       float* Tx, float* wr, float2* up, float* u, float2* udf, float* z, float2* Rdf,
                       float2* ys, float2* czp, float* cz, float* Et, float2* ewp, float* ew, float2* lp, double* lout,
                       float* Cth, float* Ctl, int* dstatus) {
  cudaStream_t st = h->stream;
  const int n = h->n;
  if (!h->smem_attr_gemm_tc) {
    rbrp_status s = cuda_check(h, cudaFuncSetAttribute(tc::k_gemm_tc<EpiE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)tc::GEMM_SMEM), "cudaFuncSetAttribute(k_gemm_tc<E>)");
    if (s == RBRP_OK)
      s = cuda_check(h, cudaFuncSetAttribute(tc::k_gemm_tc<EpiG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)tc::GEMM_SMEM), "cudaFuncSetAttribute(k_gemm_tc<G>)");
    if (s != RBRP_OK) return s;
    h->smem_attr_gemm_tc = true;
  }
  const long long budget = h->wait_budget > 0 ? h->wait_budget : kWaitBudgetDefault;
  CUtensorMap tmX1, tmY1h, tmY1l;
  rbrp_status s = make_tmap_f32(h, &tmX1, Tx, k, nc, kp, tc::BK, tc::BM);
  if (s == RBRP_OK) s = make_tmap_f32(h, &tmY1h, Cth, k, m, kp, tc::BK, tc::BN);
  if (s == RBRP_OK) s = make_tmap_f32(h, &tmY1l, Ctl, k, m, kp, tc::BK, tc::BN);
  if (s != RBRP_OK) return s;
  s = cuda_check(h, cudaMemsetAsync(dstatus, 0, sizeof(int), st), "clear status");
  if (s != RBRP_OK) return s;

  k_adj_prep_tc<<<dim3((k + 31) / 32, (nc + 31) / 32), 256, 0, st>>>(h->T, k, nc, kp, ncp, dW, h->perm, Tx, Trh,
                                                                     Trl, wr);
  k_adj_gather_ct<<<dim3((m + 31) / 32, (k + 31) / 32), 256, 0, st>>>(dA, lda, h->perm, k, m, kp, Cth, Ctl);
  k_adj_u<<<dim3((k + 255) / 256, PARTS), 256, 0, st>>>(Tx, kp, k, nc, wr, up);
  k_adj_sum_parts<<<(k + 255) / 256, 256, 0, st>>>(up, k, u, udf);
  if (dG) {
    k_adj_split_r<<<dim3((k + 31) / 32, (k + 31) / 32), 256, 0, st>>>(h->R, n, k, Rdf);
    s = solve_z(h, Rdf, k, udf, ys, z);
    if (s != RBRP_OK) return s;
    k_adj_cz<<<dim3((m + 255) / 256, PARTS), 256, 0, st>>>(dA, lda, m, k, h->perm, z, czp);
    k_adj_sum_parts<<<(m + 255) / 256, 256, 0, st>>>(czp, m, cz, nullptr);
  }
  const int tx1 = (nc + tc::BM - 1) / tc::BM, ty1 = (m + tc::BN - 1) / tc::BN;
  auto vec = [](const float* p, int64_t ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0; };
  EpiE e1{dA, lda, h->perm, k, m, nc, wr, cz, dG ? Et : nullptr, ncp, dG, ldg, scale, lp, ewp, vec(dA, lda),
          vec(dG, ldg)};
  tc::k_gemm_tc<EpiE><<<dim3(tx1, ty1), tc::NTHREADS, tc::GEMM_SMEM, st>>>(tmX1, tmY1h, tmY1l, nc, m, k, budget,
                                                                       dstatus, e1);
  if (dG) k_adj_sum_rows<<<(m + 255) / 256, 256, 0, st>>>(ewp, tx1, m, ew);
  k_adj_loss<<<1, 256, 0, st>>>(lp, tx1 * ty1, udf, k, lout);
  if (dG) {
    CUtensorMap tmX2, tmY2h, tmY2l;
    s = make_tmap_f32(h, &tmX2, Et, nc, m, ncp, tc::BK, tc::BM);
    if (s == RBRP_OK) s = make_tmap_f32(h, &tmY2h, Trh, nc, k, ncp, tc::BK, tc::BN);
    if (s == RBRP_OK) s = make_tmap_f32(h, &tmY2l, Trl, nc, k, ncp, tc::BK, tc::BN);
    if (s != RBRP_OK) return s;
    EpiG e2{h->perm, m, k, cz, ew, u, z, dG, ldg, scale};
    tc::k_gemm_tc<EpiG><<<dim3((m + tc::BM - 1) / tc::BM, (k + tc::BN - 1) / tc::BN), tc::NTHREADS, tc::GEMM_SMEM, st>>>(
        tmX2, tmY2h, tmY2l, m, k, nc, budget, dstatus, e2);
  }
  s = cuda_check(h, cudaGetLastError(), "adjoint kernels");
  if (s != RBRP_OK) return s;
  double hl[2] = {0.0, 0.0};
  int hs = 0;
  s = cuda_check(h, cudaMemcpyAsync(hl, lout, sizeof(hl), cudaMemcpyDeviceToHost, st), "copy loss");
  if (s == RBRP_OK) s = cuda_check(h, cudaMemcpyAsync(&hs, dstatus, sizeof(int), cudaMemcpyDeviceToHost, st), "status");
  if (s == RBRP_OK) s = cuda_check(h, cudaStreamSynchronize(st), "adjoint kernels");
  if (s != RBRP_OK) return s;
  if (hs == tc::ST_ERR_TIMEOUT)
    return set_error(h, RBRP_ERR_DEVICE_TIMEOUT, "a device-side wait of the adjoint GEMMs timed out; they aborted cleanly");
  if (loss) *loss = hl[0] + hl[1];
  return RBRP_OK;
}

}  // namespace
}  // namespace rbrp

using namespace rbrp;

extern "C" rbrp_status rbrp_fixed_id_adjoint_f32(rbrp_handle h, int m, int n, const float* dA, int64_t lda,
                                                 const float* dW, float scale, float* dG, int64_t ldg,
                                                 double* loss) {
  if (!h) return RBRP_ERR_INVALID_ARG;
  if (!h->have_result || h->prec != RBRP_PREC_F32_MIXED)
    return set_error(h, RBRP_ERR_NOT_COMPUTED, "needs a preceding FP32 run (rbrp_fixed_id_f32) on this matrix");
  if (m != h->m || n != h->n || !dA || lda < m || !dW)
    return set_error(h, RBRP_ERR_INVALID_ARG, "A / W do not match the last run");
  if (dG && ldg < m) return set_error(h, RBRP_ERR_INVALID_ARG, "ldg < m");
  const int k = h->k, nc = n - k;
  if (k < 1 || nc < 1 || !h->T) return set_error(h, RBRP_ERR_NOT_COMPUTED, "the last run has no T (k = 0 or n)");
  DeviceGuard g(h->device);
  cudaStream_t st = h->stream;
  // workspace: Tr, Tc (k x nc), wr (nc), u parts / u / udf, z, Rdf (k x k), work (k), cz parts / cz,
  // E (m x nc), E w parts / E w, loss parts, loss out
  const bool use_tc = h->variant == 0;
  const int gx = (m + GTILE - 1) / GTILE, gy1 = (nc + GTILE - 1) / GTILE, gy2 = (k + GTILE - 1) / GTILE;
  const int kp = (k + 3) & ~3, ncp = (nc + 3) & ~3;           // TMA leading dimensions (16-byte rows)
  const int tx1 = (nc + tc::BM - 1) / tc::BM, ty1 = (m + tc::BN - 1) / tc::BN;   // E tiles
  const size_t kn = (size_t)k * nc;
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t o = off; off += al(bytes); return o; };
  const size_t o_Tr = take(4 * (use_tc ? (size_t)ncp * k : kn)), o_Tc = take(4 * (use_tc ? (size_t)kp * nc : kn));
  const size_t o_wr = take(4 * (size_t)nc);
  const size_t o_up = take(8 * (size_t)PARTS * k), o_u = take(4 * (size_t)k), o_udf = take(8 * (size_t)k);
  const size_t o_z = take(4 * (size_t)k), o_R = take(8 * (size_t)k * k);
  const size_t o_ys = take(8 * (size_t)k);
  const size_t o_czp = take(8 * (size_t)PARTS * m), o_cz = take(4 * (size_t)m);
  const size_t o_E = take(4 * (use_tc ? (size_t)ncp * m : (size_t)m * nc)), o_ewp = take(8 * (size_t)gy1 * m);
  const size_t o_ew = take(4 * (size_t)m);
  const size_t o_lp = take(8 * std::max((size_t)gx * gy1, (size_t)tx1 * ty1)), o_loss = take(16);
  // tensor-core operands: T^T lo, C^T hi / lo, the timeout status
  const size_t o_Trl = use_tc ? take(4 * (size_t)ncp * k) : 0;
  const size_t o_Cth = use_tc ? take(4 * (size_t)kp * m) : 0, o_Ctl = use_tc ? take(4 * (size_t)kp * m) : 0;
  const size_t o_st = take(16);
  if (h->adj_bytes < off) {
    if (h->adj_ws) cudaFree(h->adj_ws);
    h->adj_ws = nullptr;
    h->adj_bytes = 0;
    rbrp_status s = device_alloc(h, (void**)&h->adj_ws, off, "cudaMalloc(adjoint workspace)");
    if (s != RBRP_OK) return s;
    h->adj_bytes = off;
  }
  unsigned char* w = static_cast<unsigned char*>(h->adj_ws);
  float* Tr = reinterpret_cast<float*>(w + o_Tr);
  float* Tc = reinterpret_cast<float*>(w + o_Tc);
  float* wr = reinterpret_cast<float*>(w + o_wr);
  float2* up = reinterpret_cast<float2*>(w + o_up);
  float* u = reinterpret_cast<float*>(w + o_u);
  float2* udf = reinterpret_cast<float2*>(w + o_udf);
  float* z = reinterpret_cast<float*>(w + o_z);
  float2* Rdf = reinterpret_cast<float2*>(w + o_R);
  float2* ys = reinterpret_cast<float2*>(w + o_ys);
  float2* czp = reinterpret_cast<float2*>(w + o_czp);
  float* cz = reinterpret_cast<float*>(w + o_cz);
  float* E = reinterpret_cast<float*>(w + o_E);
  float2* ewp = reinterpret_cast<float2*>(w + o_ewp);
  float* ew = reinterpret_cast<float*>(w + o_ew);
  float2* lp = reinterpret_cast<float2*>(w + o_lp);
  double* lout = reinterpret_cast<double*>(w + o_loss);
  int* dstatus = reinterpret_cast<int*>(w + o_st);

  if (use_tc) return adjoint_tc(h, m, k, nc, kp, ncp, dA, lda, dW, scale, dG, ldg, loss, Tr /* T^T hi */,
                                reinterpret_cast<float*>(w + o_Trl), Tc /* Tx */, wr, up, u, udf, z, Rdf, ys, czp,
                                cz, E /* E^T */, ewp, ew, lp, lout, reinterpret_cast<float*>(w + o_Cth),
                                reinterpret_cast<float*>(w + o_Ctl), dstatus);
  k_adj_prep<<<dim3((k + 31) / 32, (nc + 31) / 32), 256, 0, st>>>(h->T, k, nc, dW, h->perm, Tr, Tc, wr);
  k_adj_u<<<dim3((k + 255) / 256, PARTS), 256, 0, st>>>(Tc, k, k, nc, wr, up);
  k_adj_sum_parts<<<(k + 255) / 256, 256, 0, st>>>(up, k, u, udf);
  if (dG) {
    k_adj_split_r<<<dim3((k + 31) / 32, (k + 31) / 32), 256, 0, st>>>(h->R, n, k, Rdf);
    rbrp_status s = solve_z(h, Rdf, k, udf, ys, z);
    if (s != RBRP_OK) return s;
    k_adj_cz<<<dim3((m + 255) / 256, PARTS), 256, 0, st>>>(dA, lda, m, k, h->perm, z, czp);
    k_adj_sum_parts<<<(m + 255) / 256, 256, 0, st>>>(czp, m, cz, nullptr);
  }
  k_adj_gemm1<<<dim3(gx, gy1), GT, 0, st>>>(dA, lda, m, k, nc, h->perm, Tr, wr, cz, dG ? E : nullptr, dG, ldg, scale,
                                            lp, ewp);
  if (dG) k_adj_sum_rows<<<(m + 255) / 256, 256, 0, st>>>(ewp, gy1, m, ew);
  k_adj_loss<<<1, 256, 0, st>>>(lp, gx * gy1, udf, k, lout);
  if (dG) {
    k_adj_gemm2<<<dim3(gx, gy2), GT, 0, st>>>(E, m, k, nc, h->perm, Tc, cz, ew, u, z, dG, ldg, scale);
  }
  double hl[2] = {0.0, 0.0};
  rbrp_status s = cuda_check(h, cudaMemcpyAsync(hl, lout, sizeof(hl), cudaMemcpyDeviceToHost, st), "copy loss");
  if (s == RBRP_OK) s = cuda_check(h, cudaStreamSynchronize(st), "adjoint kernels");
  if (s != RBRP_OK) return s;
  if (loss) *loss = hl[0] + hl[1];
  return RBRP_OK;
}
