// rbrp_kernels.cuh - sm_103a kernels of one adaptive RBRP block step.
//
// Per block (positions [i, i+bs) are filled), in launch order:
//   k_sample      weighted block sampling (np-compat / exponential keys / greedy)
//   (rbrp_panel64.cuh, FP64 form)
//   k_gather_coef C = Q(:, :i)^T A(:, J), from R
//                 (k_cgs_coef where R holds no slice products)
//   k_cgs_panel   V = A(:, J) - Q(:, :i) C
//   k_gram64      V^T V, and Q1^T Q1 after the first pass
//   k_pchol       CPQR pivots + robust filter from V^T V, R11, block swap
//   k_panel_solve Q1 = V_p R11^{-1}, then Q_blk = Q1 R2^{-1}
//   k_chol2       R2 = chol(Q1^T Q1);  k_panel_r  R(I2, I2) = R2 R11
//   (here)
//   k_swap_R      R(:i, K2) = R(:i, K1), R(:i, I2) = R(:i, J)
//   k_project     W = Q_blk^T A(:, perm[p]) for the remaining positions p,
//                 R(I2, p) = W, diags(p) -= ||W(:, p)||^2 (clipped at 0);
//                 k_project_skinny for blocks of b <= 8 (column streams)
//   k_finish      residual, stop rule, per-block trace
#pragma once
#include <type_traits>
#include "rbrp_common.cuh"
#include "rbrp_df.cuh"
#include "rbrp_sampler.cuh"

namespace rbrp {
// Internal linkage: this header is compiled into one translation unit per
// element type, and each keeps its own copy of the type-independent kernels.
namespace {

// ===========================================================================
// a1: squared column norms (initial weights) - one HBM pass over A.
// gpu/rbrp.cu:82-99,352-356; python/RBRP.ipynb cell 11 lines 93-94.
// One warp per column, 16-byte vector loads when the column starts are
// 16-byte aligned, four loads in flight per lane.  The FP64 form also keeps
// the exponent of each column's largest entry (exps, or NULL).
// ===========================================================================
__device__ __forceinline__ void max_hi(unsigned& mx, double v) {
  mx = max(mx, (unsigned)__double2hiint(v) & 0x7FFFFFFFu);
}
__device__ __forceinline__ double col_sumsq(const double* __restrict__ col, int m, int lane, bool vec, unsigned& mx) {
  double s0 = 0.0, s1 = 0.0;
  if (vec) {
    const double2* c2 = reinterpret_cast<const double2*>(col);
    const int m2 = m >> 1;
    int r = lane;
    for (; r + 96 < m2; r += 128) {
      const double2 a = __ldg(c2 + r), b = __ldg(c2 + r + 32), c = __ldg(c2 + r + 64), d = __ldg(c2 + r + 96);
      s0 = fma(a.x, a.x, s0); s1 = fma(a.y, a.y, s1);
      s0 = fma(b.x, b.x, s0); s1 = fma(b.y, b.y, s1);
      s0 = fma(c.x, c.x, s0); s1 = fma(c.y, c.y, s1);
      s0 = fma(d.x, d.x, s0); s1 = fma(d.y, d.y, s1);
      max_hi(mx, a.x); max_hi(mx, a.y); max_hi(mx, b.x); max_hi(mx, b.y);
      max_hi(mx, c.x); max_hi(mx, c.y); max_hi(mx, d.x); max_hi(mx, d.y);
    }
    for (; r < m2; r += 32) {
      const double2 a = __ldg(c2 + r);
      s0 = fma(a.x, a.x, s0); s1 = fma(a.y, a.y, s1);
      max_hi(mx, a.x); max_hi(mx, a.y);
    }
    if ((m & 1) && lane == 0) { const double v = col[m - 1]; s0 = fma(v, v, s0); max_hi(mx, v); }
  } else {
    for (int r = lane; r < m; r += 32) { const double v = col[r]; s0 = fma(v, v, s0); max_hi(mx, v); }
  }
  return warp_sum(s0 + s1);
}

__device__ __forceinline__ double col_sumsq(const float* __restrict__ col, int m, int lane, bool vec, unsigned&) {
  DF acc{0.f, 0.f};
  if (vec) {
    const float4* c4 = reinterpret_cast<const float4*>(col);
    const int m4 = m >> 2;
    int r = lane;
    for (; r + 96 < m4; r += 128) {
      const float4 a = __ldg(c4 + r), b = __ldg(c4 + r + 32), c = __ldg(c4 + r + 64), d = __ldg(c4 + r + 96);
      df_add_sq(acc, a.x); df_add_sq(acc, a.y); df_add_sq(acc, a.z); df_add_sq(acc, a.w);
      df_add_sq(acc, b.x); df_add_sq(acc, b.y); df_add_sq(acc, b.z); df_add_sq(acc, b.w);
      df_add_sq(acc, c.x); df_add_sq(acc, c.y); df_add_sq(acc, c.z); df_add_sq(acc, c.w);
      df_add_sq(acc, d.x); df_add_sq(acc, d.y); df_add_sq(acc, d.z); df_add_sq(acc, d.w);
    }
    for (; r < m4; r += 32) {
      const float4 a = __ldg(c4 + r);
      df_add_sq(acc, a.x); df_add_sq(acc, a.y); df_add_sq(acc, a.z); df_add_sq(acc, a.w);
    }
    for (int t = (m4 << 2) + lane; t < m; t += 32) df_add_sq(acc, col[t]);
  } else {
    for (int r = lane; r < m; r += 32) df_add_sq(acc, col[r]);
  }
  return warp_sum((double)acc.hi + (double)acc.lo);
}

template <typename T>
__global__ void __launch_bounds__(256) k_colnorm(const T* __restrict__ A, int64_t lda, int m, int n,
                                                 double* __restrict__ diags, int* __restrict__ perm,
                                                 State* st, int* __restrict__ exps) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (c >= n) return;
  const bool vec = ((reinterpret_cast<uintptr_t>(A) & 15) == 0) && ((lda * (int64_t)sizeof(T)) % 16 == 0);
  unsigned mx = 0u;
  const double s = col_sumsq(A + (int64_t)c * lda, m, lane, vec, mx);
  if (exps) {
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) exps[c] = (int)max(mx >> 20, 1u) - 1022;   // |a| < 2^exps
  }
  if (lane == 0) {
    diags[c] = s;
    perm[c] = c;
    if (!isfinite(s)) st->status = ST_ERR_NUMERIC;
  }
}

// Initial totals and loop state.  One CTA.
__global__ void __launch_bounds__(1024) k_init(State* st, const double* __restrict__ diags, int n, int kmax) {
  __shared__ double shd[32];
  __shared__ int shi[32];
  double s = 0.0;
  int c = 0;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const double d = diags[j];
    s += d;
    c += d > 0.0;
  }
  s = block_sum(s, shd);
  c = block_sum(c, shi);
  if (threadIdx.x == 0) {
    st->i = 0;
    st->bs_sampled = 0;
    st->bs = 0;
    st->nblocks = 0;
    st->zero_panel = 0;
    st->nK = 0;
    st->recomputes = 0;
    st->attempts = 0;
    st->draws = 0ull;
    st->res0 = s;
    st->residual = s;
    st->nnz_rem = c;
    st->done = (c == 0 || kmax <= 0 || st->status != 0) ? 1 : 0;
  }
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
k_sample(State* st, const double* __restrict__ diags, const int* __restrict__ perm, int n, int kmax,
         int b, uint64_t seed, int sampler, double* __restrict__ pbuf,
         unsigned long long* __restrict__ kbuf, int* __restrict__ js, int* __restrict__ cols,
         const int* __restrict__ order_of, const double* __restrict__ pre_tot, const int* __restrict__ pre_pos) {
  sample_block(st, diags, perm, n, kmax, b, seed, sampler, pbuf, kbuf, js, cols, order_of, pre_tot, pre_pos);
}

// Deterministic sum of split partials: out[x] = sum_z part[z*stride + x].
template <typename V>
__global__ void k_reduce_parts(const V* __restrict__ part, int nparts, int64_t stride, int64_t count,
                               V* __restrict__ out) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < count;
       x += (int64_t)gridDim.x * blockDim.x) {
    V s = V(0);
#pragma unroll 8
    for (int z = 0; z < nparts; ++z) s += part[(int64_t)z * stride + x];
    out[x] = s;
  }
}

// Column swap of the rows above the block: R(:i, K2) = R(:i, K1); R(:i, I2) = R(:i, J).
// One warp per row, two block positions per lane, every load before the first store (a
// thread per row walked 64 scattered columns in turn: 33 us at 640 rows of 8192 columns,
// now 4.2).
__global__ void __launch_bounds__(256)
k_swap_R(double* __restrict__ R, int64_t ldr, const State* __restrict__ st, const int* __restrict__ Jg,
         const int* __restrict__ K1g, const int* __restrict__ K2g) {
  const int i = st->i, kept = st->bs, nK = st->nK, lane = threadIdx.x & 31;
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= i || kept == 0) return;
  double* Rr = R + (int64_t)row * ldr;
  double tj[2], tk[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int s = lane + 32 * u;
    tj[u] = s < kept ? Rr[Jg[s]] : 0.0;
    tk[u] = s < nK ? Rr[K1g[s]] : 0.0;
  }
  __syncwarp();
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int s = lane + 32 * u;
    if (s < nK) Rr[K2g[s]] = tk[u];
    if (s < kept) Rr[i + s] = tj[u];
  }
}

// ===========================================================================
// a7 + a8: projection of the remaining columns on the new block and the
// residual-norm downdate (python/RBRP.ipynb cell 11 lines 132, 154-158;
// matlab/RBRP.m:103-104,112; the reference applies Householder reflectors to
// the whole trailing matrix instead, gpu/rbrp.cu:297-330, 453-466).
// CTA tile: KB basis vectors (KB >= kept, chosen on the host from b) x PC
// positions, K loop over m in chunks of KC rows; every thread holds an MU x VP
// accumulator block: 4 x 4 (PC = 4096 / KB), or 2 x 1 and PC = 8 or 16 where the
// large tiles would not fill the SMs.  Each accumulator sums over the rows in
// ascending order, so W is the same for every tile: the tile only spreads the
// work and drops basis rows that do not exist (the FP64 pipe is the bound of
// this kernel; 1000 x 1000, b = 40: 610 us a block in 16 large tiles, 120 in
// small ones).
// ===========================================================================
template <int KB_, int VP_>
struct ProjTile {
  static constexpr int KB = KB_, VP = VP_;
  static constexpr int MU = VP == 4 ? 4 : KB >= 32 ? 2 : 1;    // basis rows per thread
  static constexpr int TY = KB / MU;             // thread rows
  static constexpr int TX = 256 / TY;            // thread columns
  static constexpr int PC = TX * VP;             // positions per CTA
  static constexpr int KC = 4096 / PC < 32 ? 4096 / PC : 32;   // rows per K chunk
};

template <typename T, typename P>
__global__ void __launch_bounds__(256)
k_project(const T* __restrict__ Q, int64_t ldq, const T* __restrict__ A, int64_t lda,
          const int* __restrict__ perm, const State* __restrict__ st, int m, int n,
          double* __restrict__ R, int64_t ldr, double* __restrict__ diags,
          double* __restrict__ part_res, int* __restrict__ part_nnz) {
  constexpr int KB = P::KB, VP = P::VP, PC = P::PC, KC = P::KC, TX = P::TX, TY = P::TY, MU = P::MU;
  constexpr int NRED = PC < 64 ? 1 : PC / 64, RLEN = PC < 64 ? PC : 64;
  constexpr size_t kOps = sizeof(T) * (KC * KB + KC * (PC + 1));
  constexpr size_t kW = sizeof(double) * KB * (PC + 1);
  __shared__ __align__(16) unsigned char raw[kOps > kW ? kOps : kW];
  T(*Qs)[KB] = reinterpret_cast<T(*)[KB]>(raw);
  T(*As)[PC + 1] = reinterpret_cast<T(*)[PC + 1]>(raw + sizeof(T) * KC * KB);
  double(*Ws)[PC + 1] = reinterpret_cast<double(*)[PC + 1]>(raw);
  __shared__ int cs[PC];
  __shared__ double snew[PC];
  __shared__ double red_s[NRED];
  __shared__ int red_c[NRED];
  const int tid = threadIdx.x;
  // kept <= b <= KB by construction (the host picks KB from b); the clamp only keeps smem in bounds
  const int i = st->i, kept = min(st->bs, KB);
  const int pbase = i + st->bs + blockIdx.x * PC;
  if (kept == 0 || pbase >= n) {
    if (tid == 0) { part_res[blockIdx.x] = 0.0; part_nnz[blockIdx.x] = 0; }
    return;
  }
  for (int t = tid; t < PC; t += 256) cs[t] = (pbase + t < n) ? perm[pbase + t] : -1;
  const int ty = tid / TX, tx = tid % TX;
  const int ty0 = (tid & ~31) / TX;      // the warp's first basis row
  const int me = kept > ty0 ? (kept - ty0 + TY - 1) / TY : 0;   // <= MU
  T acc[MU][VP];
#pragma unroll
  for (int u = 0; u < MU; ++u)
#pragma unroll
    for (int v = 0; v < VP; ++v) acc[u][v] = T(0);
  const T* Qb = Q + (int64_t)i * ldq;
  for (int r0 = 0; r0 < m; r0 += KC) {
    __syncthreads();
    for (int idx = tid; idx < KC * KB; idx += 256) {
      const int kk = idx % KC, aa = idx / KC;
      const int r = r0 + kk;
      Qs[kk][aa] = (r < m && aa < kept) ? Qb[r + (int64_t)aa * ldq] : T(0);
    }
#pragma unroll
    for (int q = 0; q < (KC * PC) / 256; ++q) {
      const int idx = tid + 256 * q, kk = idx % KC, cc = idx / KC;
      const int r = r0 + kk, c = cs[cc];
      As[kk][cc] = (r < m && c >= 0) ? A[r + (int64_t)c * lda] : T(0);
    }
    __syncthreads();
    // basis rows per thread that exist (kept <= TY * me) as a compile-time count:
    // predicated-off FP64 FMAs would still take issue slots on the FP64 pipe
    auto fmas = [&](auto mec) {
      constexpr int ME = decltype(mec)::value;
#pragma unroll 4
      for (int kk = 0; kk < KC; ++kk) {
        T qv[ME], av[VP];
#pragma unroll
        for (int u = 0; u < ME; ++u) qv[u] = Qs[kk][ty + TY * u];
#pragma unroll
        for (int v = 0; v < VP; ++v) av[v] = As[kk][tx + TX * v];
#pragma unroll
        for (int u = 0; u < ME; ++u)
#pragma unroll
          for (int v = 0; v < VP; ++v) acc[u][v] = fma(qv[u], av[v], acc[u][v]);
      }
    };
    if (me == 0) continue;
    if (MU == 1 || me <= 1) fmas(std::integral_constant<int, 1>{});
    else if (me <= 2) fmas(std::integral_constant<int, (MU < 2 ? MU : 2)>{});
    else if (me <= 3) fmas(std::integral_constant<int, (MU < 3 ? MU : 3)>{});
    else fmas(std::integral_constant<int, MU>{});
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < MU; ++u)
#pragma unroll
    for (int v = 0; v < VP; ++v) Ws[ty + TY * u][tx + TX * v] = (double)acc[u][v];
  __syncthreads();
  for (int idx = tid; idx < kept * PC; idx += 256) {
    const int a = idx / PC, c = idx % PC;
    if (pbase + c < n) R[(int64_t)(i + a) * ldr + pbase + c] = Ws[a][c];
  }
  for (int t = tid; t < PC; t += 256) {
    const int p = pbase + t;
    double d = 0.0;
    if (p < n) {
      double s = 0.0;
      for (int a = 0; a < kept; ++a) s = fma(Ws[a][t], Ws[a][t], s);
      d = diags[p] - s;
      d = d > 0.0 ? d : (d == d ? 0.0 : d);
      diags[p] = d;
    }
    snew[t] = d;
  }
  __syncthreads();
  // CTA partial of the residual and of the nonzero count, positions in ascending order
  // in chunks of 64 (of the tile where it is smaller, which moves the trace by 5e-17)
  if (tid < NRED) {
    double sacc = 0.0;
    int c = 0;
    for (int t = tid * RLEN; t < (tid + 1) * RLEN; ++t) { sacc += snew[t]; c += snew[t] > 0.0; }
    red_s[tid] = sacc;
    red_c[tid] = c;
  }
  __syncthreads();
  if (tid == 0) {
    double sacc = 0.0;
    int c = 0;
    for (int t = 0; t < NRED; ++t) { sacc += red_s[t]; c += red_c[t]; }
    part_res[blockIdx.x] = sacc;
    part_nnz[blockIdx.x] = c;
  }
}

// Skinny form of the same projection for b <= 8 (a GEMV shape: greedy b = 1 is
// column-pivoted QR).  Each warp streams CW = 4 whole columns (coalesced over
// rows) against the basis staged in shared memory, MC rows at a time; lanes keep
// strided partial sums that a butterfly combines.  32 positions per CTA.
constexpr int SKINNY_COLS = 32;

template <typename T, int KB>
__global__ void __launch_bounds__(256)
k_project_skinny(const T* __restrict__ Q, int64_t ldq, const T* __restrict__ A, int64_t lda,
                 const int* __restrict__ perm, const State* __restrict__ st, int m, int n,
                 double* __restrict__ R, int64_t ldr, double* __restrict__ diags,
                 double* __restrict__ part_res, int* __restrict__ part_nnz) {
  constexpr int CW = 4, MC = 256, NW = 8;
  static_assert(NW * CW == SKINNY_COLS, "positions per CTA");
  __shared__ T Qs[KB][MC];   // basis chunk, row index fastest: lanes read consecutive rows
  __shared__ double red_s[NW];
  __shared__ int red_c[NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // kept <= b <= KB by construction (the host picks KB from b); the clamp only keeps smem in bounds
  const int i = st->i, kept = min(st->bs, KB);
  const int pbase = i + st->bs + blockIdx.x * SKINNY_COLS;
  if (kept == 0 || pbase >= n) {
    if (tid == 0) { part_res[blockIdx.x] = 0.0; part_nnz[blockIdx.x] = 0; }
    return;
  }
  int col[CW];
#pragma unroll
  for (int c = 0; c < CW; ++c) {
    const int p = pbase + warp * CW + c;
    col[c] = p < n ? perm[p] : -1;
  }
  T acc[CW][KB];
#pragma unroll
  for (int c = 0; c < CW; ++c)
#pragma unroll
    for (int a = 0; a < KB; ++a) acc[c][a] = T(0);
  const T* Qb = Q + (int64_t)i * ldq;
  for (int r0 = 0; r0 < m; r0 += MC) {
    __syncthreads();
    for (int idx = tid; idx < KB * MC; idx += 256) {
      const int a = idx / MC, rr = idx % MC, r = r0 + rr;
      Qs[a][rr] = (r < m && a < kept) ? Qb[r + (int64_t)a * ldq] : T(0);
    }
    __syncthreads();
    const int rend = min(MC, m - r0);
#pragma unroll 2
    for (int rr = lane; rr < rend; rr += 32) {
      T av[CW], qv[KB];
#pragma unroll
      for (int c = 0; c < CW; ++c) av[c] = col[c] >= 0 ? A[(r0 + rr) + (int64_t)col[c] * lda] : T(0);
#pragma unroll
      for (int a = 0; a < KB; ++a) qv[a] = Qs[a][rr];
#pragma unroll
      for (int c = 0; c < CW; ++c)
#pragma unroll
        for (int a = 0; a < KB; ++a) acc[c][a] = fma(av[c], qv[a], acc[c][a]);
    }
  }
#pragma unroll
  for (int c = 0; c < CW; ++c)
#pragma unroll
    for (int a = 0; a < KB; ++a)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[c][a] += __shfl_xor_sync(0xffffffffu, acc[c][a], o);
  double dsum = 0.0;
  int dcnt = 0;
#pragma unroll
  for (int c = 0; c < CW; ++c) {
    const int p = pbase + warp * CW + c;
    if (lane == c && p < n) {
      double s = 0.0;
#pragma unroll
      for (int a = 0; a < KB; ++a) {
        if (a < kept) {
          const double w = (double)acc[c][a];
          R[(int64_t)(i + a) * ldr + p] = w;
          s = fma(w, w, s);
        }
      }
      double d = diags[p] - s;
      d = d > 0.0 ? d : (d == d ? 0.0 : d);
      diags[p] = d;
      dsum = d;
      dcnt = d > 0.0;
    }
  }
#pragma unroll
  for (int o = 1; o < CW; o <<= 1) {
    dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
    dcnt += __shfl_xor_sync(0xffffffffu, dcnt, o);
  }
  if (lane == 0) {
    red_s[warp] = dsum;
    red_c[warp] = dcnt;
  }
  __syncthreads();
  if (tid == 0) {
    double sacc = 0.0;
    int c = 0;
    for (int w = 0; w < NW; ++w) { sacc += red_s[w]; c += red_c[w]; }
    part_res[blockIdx.x] = sacc;
    part_nnz[blockIdx.x] = c;
  }
}

// ===========================================================================
// Residual form (FP32 storage).  The residual A_res = (I - Q Q^T) A is kept
// explicitly, position ordered, and updated after every block - the
// trailing-matrix update of gpu/rbrp.cu:297-330,448 (Householder there,
// Q_blk W here) - so every residual norm is recomputed exactly from the
// residual instead of downdated: a downdate ||a||^2 - ||Q^T a||^2 in FP32
// arithmetic cannot resolve residuals below ~1e-7 of ||a||^2.
// ===========================================================================

// Block swap of the residual's columns: A_res(:, K2) = A_res(:, K1).  Kept
// columns need no copy (their residual was gathered into the panel already).
__global__ void k_swap_cols(float* __restrict__ Ares, int64_t ld, const State* __restrict__ st, int m,
                            const int* __restrict__ K1g, const int* __restrict__ K2g) {
  const int t = blockIdx.y;
  if (t >= st->nK) return;
  const float* src = Ares + (int64_t)K1g[t] * ld;
  float* dst = Ares + (int64_t)K2g[t] * ld;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x) dst[r] = src[r];
}

__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float x) {
  const float t = hi + x;
  const float bb = t - hi;
  lo += (hi - (t - bb)) + (x - bb);
  hi = t;
}

// P1: W = Q_blk^T A_res(:, p) for the remaining positions p, into R(I2, p).
// CTA tile 64 basis vectors x 64 positions, 32-row K stages; each stage's FP32
// partial sums are folded into double-float accumulators (TwoSum), so W is
// accurate to ~1e-8 relative over m = 16384 rows.
__global__ void __launch_bounds__(128)
k_proj_w(const float* __restrict__ Qb, int64_t ldq, const float* __restrict__ Ares, int64_t ld,
         const State* __restrict__ st, int m, int n, double* __restrict__ R, int64_t ldr) {
  __shared__ __align__(16) float Qs[32][MAXB];
  __shared__ __align__(16) float As[32][MAXB + 4];
  const int tid = threadIdx.x;
  const int i = st->i, kept = st->bs;
  const int p0 = i + kept + blockIdx.x * 64;
  if (kept == 0 || p0 >= n) return;
  const int ncol = min(64, n - p0);
  const int ta = tid >> 4, tc = tid & 15;  // rows a = ta*8 + u, columns c = tc*4 + v
  float hi[8][4], lo[8][4];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) hi[u][v] = lo[u][v] = 0.f;
  for (int r0 = 0; r0 < m; r0 += 32) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int idx = tid + 128 * q, kk = idx & 31, aa = idx >> 5, r = r0 + kk;
      Qs[kk][aa] = (r < m && aa < kept) ? Qb[r + (int64_t)aa * ldq] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int idx = tid + 128 * q, kk = idx & 31, cc = idx >> 5, r = r0 + kk;
      As[kk][cc] = (r < m && cc < ncol) ? Ares[r + (int64_t)(p0 + cc) * ld] : 0.f;
    }
    __syncthreads();
    float c[8][4];
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) c[u][v] = 0.f;
#pragma unroll 8
    for (int kk = 0; kk < 32; ++kk) {
      const float4 q0 = *reinterpret_cast<const float4*>(&Qs[kk][ta * 8]);
      const float4 q1 = *reinterpret_cast<const float4*>(&Qs[kk][ta * 8 + 4]);
      const float4 a4 = *reinterpret_cast<const float4*>(&As[kk][tc * 4]);
      const float qv[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
      const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) c[u][v] = fmaf(qv[u], av[v], c[u][v]);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) two_sum_acc(hi[u][v], lo[u][v], c[u][v]);
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int a = ta * 8 + u;
    if (a < kept) {
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int cc = tc * 4 + v;
        if (cc < ncol) R[(int64_t)(i + a) * ldr + p0 + cc] = (double)hi[u][v] + (double)lo[u][v];
      }
    }
  }
}

// P2 on the CUDA cores (the CUDA-core variant; the default is k_resid_update_tc):
// A_res(:, p) -= Q_blk W(:, p) and the partial squared norms of the updated
// columns (double-float sums), for 64 positions x one row range per CTA.  Warp w
// owns 8 columns, lane l four consecutive rows of every 128-row stage (16-byte
// loads and stores, coalesced along the column).  Row ranges of the same columns
// are summed by k_norm_reduce.  W comes from R (written by k_proj_w).
constexpr int P2_COLS = 64;
constexpr int P2_ROWS = 128;
constexpr int P2_MAX_SPLIT = 8;
constexpr int P2_THREADS = 256;
constexpr size_t P2_SMEM = sizeof(float) * (size_t)MAXB * (P2_COLS + 2 * P2_ROWS);   // W + two basis stages

// 16-byte asynchronous copy global -> shared; bytes beyond src_bytes are zero-filled
__device__ __forceinline__ void upd_cp16(float* smem, const float* gmem, int src_bytes) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void upd_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void upd_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__global__ void __launch_bounds__(P2_THREADS, 2)
k_resid_update(const float* __restrict__ Qb, int64_t ldq, float* __restrict__ Ares, int64_t ld,
               const State* __restrict__ st, int m, int n, int rows_per_split, const double* __restrict__ R,
               int64_t ldr, double* __restrict__ part_norm) {
  extern __shared__ __align__(16) float p2_smem[];
  float* Ws = p2_smem;                       // Ws[a * P2_COLS + c]
  float* Qbuf = p2_smem + MAXB * P2_COLS;    // two stages of Qs[a * P2_ROWS + rr]
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int i = st->i, kept = st->bs;
  const int p0 = i + kept + blockIdx.x * P2_COLS;
  if (kept == 0 || p0 >= n) return;
  const int ncol = min(P2_COLS, n - p0);
  const int rb = blockIdx.y * rows_per_split, re = min(m, rb + rows_per_split);
  for (int idx = tid; idx < kept * P2_COLS; idx += P2_THREADS) {
    const int a = idx / P2_COLS, c = idx % P2_COLS;
    Ws[idx] = c < ncol ? (float)R[(int64_t)(i + a) * ldr + p0 + c] : 0.f;
  }
  DF nrm[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) nrm[c].hi = nrm[c].lo = 0.f;
  // basis stage of rows [r0, r0 + P2_ROWS) into dst by cp.async; rows at or past re read as zero
  auto load_q = [&](int r0, float* dst) {
    for (int idx = tid; idx < kept * (P2_ROWS / 4); idx += P2_THREADS) {
      const int a = idx / (P2_ROWS / 4), j = idx % (P2_ROWS / 4), rq = r0 + 4 * j;
      const int bytes = 4 * max(0, min(4, re - rq));
      upd_cp16(dst + a * P2_ROWS + 4 * j, bytes > 0 ? Qb + rq + (int64_t)a * ldq : Qb, bytes);
    }
    upd_commit();
  };
  load_q(rb, Qbuf);
  int stage = 0;
  for (int r0 = rb; r0 < re; r0 += P2_ROWS, ++stage) {
    const float* Qs = Qbuf + (stage & 1) * MAXB * P2_ROWS;
    // this thread's residual values, fetched before the products so the loads
    // are in flight during the stage's FMA work
    const int r = r0 + 4 * lane;
    const bool vec_ok = r + 3 < re;
    float4 xa[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int cc = w * 8 + c;
      xa[c] = (vec_ok && cc < ncol) ? *reinterpret_cast<const float4*>(Ares + (int64_t)(p0 + cc) * ld + r)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // the next stage's basis goes into the other buffer, whose last readers passed the
    // barrier that ended the previous stage
    if (r0 + P2_ROWS < re) {
      load_q(r0 + P2_ROWS, Qbuf + ((stage + 1) & 1) * MAXB * P2_ROWS);
      upd_wait<1>();
    } else {
      upd_wait<0>();
    }
    __syncthreads();
    float acc[4][8];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[u][c] = 0.f;
#pragma unroll 4
    for (int a = 0; a < kept; ++a) {
      const float4 q4 = reinterpret_cast<const float4*>(Qs + a * P2_ROWS)[lane];
      const float4* w4 = reinterpret_cast<const float4*>(Ws + a * P2_COLS + w * 8);
      const float4 x0 = w4[0], x1 = w4[1];
      const float qv[4] = {q4.x, q4.y, q4.z, q4.w};
      const float wv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[u][c] = fmaf(qv[u], wv[c], acc[u][c]);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int cc = w * 8 + c;
      if (cc < ncol) {
        float* col = Ares + (int64_t)(p0 + cc) * ld;
        if (vec_ok) {
          float4 x = xa[c];
          x.x -= acc[0][c];
          x.y -= acc[1][c];
          x.z -= acc[2][c];
          x.w -= acc[3][c];
          *reinterpret_cast<float4*>(col + r) = x;
          // FP32 sum of the 4 squares (positive terms, relative error < 3e-7), folded
          // into the double-float norm by TwoSum
          const float q4 = fmaf(x.w, x.w, fmaf(x.z, x.z, fmaf(x.y, x.y, x.x * x.x)));
          const float t = nrm[c].hi + q4;
          const float bb = t - nrm[c].hi;
          nrm[c].lo += (nrm[c].hi - (t - bb)) + (q4 - bb);
          nrm[c].hi = t;
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (r + u < re) {
              const float x = col[r + u] - acc[u][c];
              col[r + u] = x;
              df_add_sq(nrm[c], x);
            }
          }
        }
      }
    }
    __syncthreads();   // every warp is done with this stage's basis before it is refilled
  }
  // warp sums of the double-float norms on the FP32 pipe; lane 0 converts once per column
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    dfl v = df_two_sum(nrm[c].hi, nrm[c].lo);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      v = df_add(v, {__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
    const int cc = w * 8 + c;
    if (lane == 0 && cc < ncol) part_norm[(int64_t)blockIdx.y * n + p0 + cc] = (double)v.hi + (double)v.lo;
  }
}

// diags(p) = sum over row ranges of the partial norms; per-CTA residual sums and
// positive counts for k_finish.
__global__ void __launch_bounds__(256)
k_norm_reduce(const double* __restrict__ part_norm, int nsplit, int n, const State* __restrict__ st,
              double* __restrict__ diags, double* __restrict__ part_res, int* __restrict__ part_nnz) {
  __shared__ double shd[32];
  __shared__ int shi[32];
  const int p = st->i + st->bs + blockIdx.x * 256 + threadIdx.x;
  double d = 0.0;
  if (st->bs > 0 && p < n) {
    for (int z = 0; z < nsplit; ++z) d += part_norm[(int64_t)z * n + p];
    diags[p] = d;
  }
  const double s = block_sum(d, shd);
  const int c = block_sum((int)(d > 0.0), shi);
  if (threadIdx.x == 0) {
    part_res[blockIdx.x] = s;
    part_nnz[blockIdx.x] = c;
  }
}

// ===========================================================================
// a8 + a9 + a12: residual, stopping rule and per-block trace.  One CTA.
// ===========================================================================
__global__ void __launch_bounds__(1024)
k_finish(State* st, const double* __restrict__ part_res, const int* __restrict__ part_nnz, int nparts,
         double* __restrict__ diags, const int* __restrict__ js, int n, int kmax, double tol,
         int* __restrict__ trace_rank, double* __restrict__ trace_err, int* __restrict__ trace_samp) {
  __shared__ double shd[32];
  __shared__ int shi[32];
  __shared__ int s_done, s_zero, s_i, s_bs, s_bss;
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_done = st->done;
    s_zero = st->zero_panel;
    s_i = st->i;
    s_bs = st->bs;
    s_bss = st->bs_sampled;
  }
  __syncthreads();
  if (s_done) return;
  if (tid == 0) st->attempts += 1;
  if (s_zero) {
    // numerically zero panel: drop the sampled columns' weights and go on
    if (tid < s_bss) diags[js[tid]] = 0.0;
    __syncthreads();
    double s = 0.0;
    int c = 0;
    for (int p = s_i + tid; p < n; p += blockDim.x) {
      const double d = diags[p];
      s += d;
      c += d > 0.0;
    }
    s = block_sum(s, shd);
    c = block_sum(c, shi);
    if (tid == 0) {
      st->residual = s;
      st->nnz_rem = c;
      st->zero_panel = 0;
      if (c == 0 || s_bss == 0) st->done = 1;  // nothing left that can be sampled
    }
    return;
  }
  // residual and nonzero count: strided partial sums, then a fixed-order block tree
  double s = 0.0;
  int c = 0;
  for (int z = tid; z < nparts; z += blockDim.x) { s += part_res[z]; c += part_nnz[z]; }
  s = block_sum(s, shd);
  c = block_sum(c, shi);
  if (tid == 0) {
    const int i = s_i + s_bs;
    const int nb = st->nblocks;
    st->i = i;
    st->residual = s;
    st->nnz_rem = c;
    trace_rank[nb] = i;
    trace_err[nb] = st->res0 > 0.0 ? s / st->res0 : 0.0;
    trace_samp[nb] = s_bss;
    st->nblocks = nb + 1;
    if ((tol > 0.0 && s < st->res0 * tol) || c == 0 || i >= kmax || !(s == s)) st->done = 1;
    if (!(s == s) && st->status == 0) st->status = ST_ERR_NUMERIC;  // an earlier status (a timeout) stays
  }
}

}  // namespace
}  // namespace rbrp
