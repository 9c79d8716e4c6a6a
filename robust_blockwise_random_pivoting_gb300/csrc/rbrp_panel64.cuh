// rbrp_panel64.cuh - panel kernels of the FP64 form: block Gram-Schmidt, panel CPQR
// (pivoted Cholesky of the Gram matrix with the robust filter) and CholQR2.
//
// GB300 retires 1.6 FP64 FMAs per clock and SM (a warp's FMA takes 20 clocks), so these
// kernels are laid out by what that pipe has to do: tiles small enough that every SM has
// one, triangles computed once and mirrored, the 64 x 64 factorisations on 1024 threads
// over the rows still active.  Every sum runs in one fixed order whatever the tiles are
// (a column of Q times a column of A over fixed row ranges, 64-row Gram partials, one
// subtraction after the other in the triangular solves): late blocks draw by weights that
// are small differences, and the order of a sum would move which column they draw.
#pragma once
#include <type_traits>

#include "rbrp_common.cuh"
#include "rbrp_pchol_df.cuh"

namespace rbrp {
namespace {

// ===========================================================================
// a3: block Gram-Schmidt against the current basis (one CGS pass, as
// python/RBRP.ipynb cell 11 line 120 and matlab/RBRP.m:55).
// ===========================================================================
// Cpart[z][a * MAXB + c] = sum over rows of split z of Q(r, a) * A(r, cols[c]), 32 basis
// vectors x 16 columns per CTA.
constexpr int COEF_COLS = 16;
__global__ void __launch_bounds__(256)
k_cgs_coef(const double* __restrict__ Q, int64_t ldq, const double* __restrict__ A, int64_t lda,
           const int* __restrict__ cols, const State* __restrict__ st, int m, int rows_per_split, int64_t pstride,
           double* __restrict__ Cpart) {
  __shared__ double Qs[32][33];
  __shared__ double As[32][COEF_COLS + 1];
  __shared__ int cs[COEF_COLS];
  const int tid = threadIdx.x;
  const int i = st->i, bss = st->bs_sampled;
  const int a0 = blockIdx.x * 32, c0 = blockIdx.y * COEF_COLS;
  const int rb = blockIdx.z * rows_per_split, re = min(m, rb + rows_per_split);
  if (tid < COEF_COLS) cs[tid] = c0 + tid < bss ? cols[c0 + tid] : -1;
  const int al = tid >> 3, cl = tid & 7;
  double acc[2] = {0.0, 0.0};
  if (c0 < bss) {
    for (int r0 = rb; r0 < re; r0 += 32) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int idx = tid + 256 * q, kk = idx & 31, aa = idx >> 5;
        const int r = r0 + kk, a = a0 + aa;
        Qs[kk][aa] = (r < re && a < i) ? Q[r + (int64_t)a * ldq] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int idx = tid + 256 * q, kk = idx & 31, cc = idx >> 5;
        const int r = r0 + kk, c = cs[cc];
        As[kk][cc] = (r < re && c >= 0) ? A[r + (int64_t)c * lda] : 0.0;
      }
      __syncthreads();
#pragma unroll 8
      for (int kk = 0; kk < 32; ++kk) {
        const double qa = Qs[kk][al];
        acc[0] = fma(qa, As[kk][cl], acc[0]);
        acc[1] = fma(qa, As[kk][cl + 8], acc[1]);
      }
    }
  }
  const int a = a0 + al;
  if (a < i) {   // columns past the CTAs of b are never read
    double* out = Cpart + (int64_t)blockIdx.z * pstride + (int64_t)a * MAXB + c0;
    out[cl] = acc[0];
    out[cl + 8] = acc[1];
  }
}

// C(a, c) = R(a, js[c]): the same coefficients Q(:, a)^T A(:, cols[c]) where the projection of
// block a's basis left them in R (runs that need not keep k_cgs_coef's order of sums).
__global__ void __launch_bounds__(256)
k_gather_coef(const double* __restrict__ R, int64_t ldr, const int* __restrict__ js, const State* __restrict__ st,
              double* __restrict__ C) {
  const int a = blockIdx.x * 4 + (threadIdx.x >> 6), c = threadIdx.x & 63;
  if (a >= st->i) return;
  C[a * MAXB + c] = c < st->bs_sampled ? R[(int64_t)a * ldr + js[c]] : 0.0;
}

// Thread map of the row kernels: row = tid % TR of the tile, column group g = tid / TR,
// columns g + v 256 / TR.  A warp covers 32 / TR neighbouring groups.
template <int TR>
struct RowMap {
  static constexpr int NG = 256 / TR;      // column groups
  static constexpr int NV = MAXB / NG;     // columns per thread at the most
};

// V(r, c) = A(r, cols[c]) - sum_a Q(r, a) C(a, c) for TR rows.
template <int TR>
__global__ void __launch_bounds__(256)
k_cgs_panel(const double* __restrict__ A, int64_t lda, const int* __restrict__ cols, const double* __restrict__ Q,
            int64_t ldq, const double* __restrict__ C, const State* __restrict__ st, int m, double* __restrict__ V) {
  constexpr int NG = RowMap<TR>::NG, NV = RowMap<TR>::NV, KA = 32;
  __shared__ double Qs[KA][TR + 1];
  __shared__ double Cs[KA][MAXB];
  const int tid = threadIdx.x, row = tid % TR, g = tid / TR;
  const int i = st->i, bss = st->bs_sampled;
  const int r0 = blockIdx.x * TR, r = r0 + row;
  // columns this warp has, as a uniform count: predicated-off FP64 FMAs would still take the pipe
  const int g0 = (tid & ~31) / TR;
  const int nv = bss > g0 ? (bss - g0 + NG - 1) / NG : 0;
  double x[NV], acc[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = g + NG * v;
    x[v] = (r < m && c < bss) ? A[r + (int64_t)cols[c] * lda] : 0.0;
    acc[v] = 0.0;
  }
  for (int a0 = 0; a0 < i; a0 += KA) {
    __syncthreads();
    for (int t = tid; t < KA * TR; t += 256) {
      const int rr = t % TR, aa = t / TR;
      Qs[aa][rr] = (r0 + rr < m && a0 + aa < i) ? Q[r0 + rr + (int64_t)(a0 + aa) * ldq] : 0.0;
    }
    for (int t = tid; t < KA * MAXB; t += 256)
      (&Cs[0][0])[t] = a0 + t / MAXB < i ? C[(int64_t)a0 * MAXB + t] : 0.0;
    __syncthreads();
    auto fmas = [&](auto nvc) {
      constexpr int N = decltype(nvc)::value;
#pragma unroll 4
      for (int aa = 0; aa < KA; ++aa) {
        const double q = Qs[aa][row];
#pragma unroll
        for (int v = 0; v < N; ++v) acc[v] = fma(q, Cs[aa][g + NG * v], acc[v]);
      }
    };
    if (nv == 1) fmas(std::integral_constant<int, 1>{});
    else if (nv == 2) fmas(std::integral_constant<int, 2>{});
    else if (nv > 2 && nv <= 4) fmas(std::integral_constant<int, (NV < 4 ? NV : 4)>{});
    else if (nv > 4 && nv <= 6) fmas(std::integral_constant<int, (NV < 6 ? NV : 6)>{});
    else if (nv > 6) fmas(std::integral_constant<int, NV>{});
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = g + NG * v;
    if (r < m && c < bss) V[r + (int64_t)c * m] = x[v] - acc[v];
  }
}

// Gram partials of the first bs_sampled (or kept) columns of V (ld = m) over 64 rows
// (gridDim.x) for a fifth of the pairs (gridDim.y), packed.
constexpr int GRAM_PARTS = 5;
constexpr int GRAM_PAIRS = NPAIR / GRAM_PARTS;
static_assert(GRAM_PARTS * GRAM_PAIRS == NPAIR, "pair split");
__global__ void __launch_bounds__(256)
k_gram64(const double* __restrict__ V, int m, const State* __restrict__ st, int kept_cols,
         double* __restrict__ part) {
  __shared__ double Vs[MAXB][65];
  const int tid = threadIdx.x;
  const int w = kept_cols ? st->bs : st->bs_sampled;
  const int np = w * (w + 1) / 2, x0 = blockIdx.y * GRAM_PAIRS, x1 = min(np, x0 + GRAM_PAIRS);
  if (x0 >= x1) return;
  const int r0 = blockIdx.x * 64;
  for (int t = tid; t < 64 * w; t += 256) {
    const int rr = t & 63, c = t >> 6;
    Vs[c][rr] = r0 + rr < m ? V[r0 + rr + (int64_t)c * m] : 0.0;
  }
  __syncthreads();
  for (int x = x0 + tid; x < x1; x += 256) {
    int a, b;
    tri_pair(x, w, a, b);
    double s = 0.0;
#pragma unroll 8
    for (int r = 0; r < 64; ++r) s = fma(Vs[a][r], Vs[b][r], s);
    part[(int64_t)blockIdx.x * NPAIR + x] = s;
  }
}

// G = sum of the packed partials in row order, both triangles.
__global__ void __launch_bounds__(64)
k_reduce_gram(const double* __restrict__ part, int nparts, const State* __restrict__ st, int kept_cols,
              double* __restrict__ G) {
  const int n = kept_cols ? st->bs : st->bs_sampled;
  const int x = blockIdx.x * 64 + threadIdx.x;
  if (x >= n * (n + 1) / 2) return;
  double s = 0.0;
#pragma unroll 8
  for (int z = 0; z < nparts; ++z) s += part[(int64_t)z * NPAIR + x];
  int a, b;
  tri_pair(x, n, a, b);
  G[a * MAXB + b] = s;
  G[b * MAXB + a] = s;
}

// ===========================================================================
// a4 + a5: panel CPQR and robust filter.
// CPQR of the m x bs panel V is computed as pivoted Cholesky of its Gram
// matrix in shared memory: at step t the Schur complement's diagonal holds the
// squared norms of the panel columns orthogonalised against the t pivots, so
// the argmax is the CPQR pivot (LAPACK dgeqp3's greedy rule, swap semantics,
// first index among ties), and its trace is the reverse cumulative sum of the
// squared row norms of R that the robust filter tests
// (python/RBRP.ipynb cell 11 lines 69-73, 122-123):
//   keep t rows <=> trace_t / trace_0 >= tol_loc for every earlier step.
// Q is then V_p R^{-1}, made orthonormal by a second CholQR pass (CholQR2).
// ===========================================================================
struct Panel64Smem {
  double S[MAXB][MAXB + 1];   // Schur complement: entry (a, b) of panel columns at [min][max]
  double R[MAXB][MAXB + 1];   // R[t][c]: row t of the factor, by panel column c
  int ord[MAXB];              // slot -> panel column
  int J[MAXB], K1[MAXB], K2[MAXB], inblk[MAXB], Tperm[MAXB];
  int nK, stop;
};

// Cholesky factorisation of the nb x nb matrix in sm.S, 1024 threads.  With PIVOT each
// step takes the largest remaining diagonal entry (swaps are virtual: ord maps slot ->
// column) and stops by the robust filter.  Returns the number of steps taken.
//
// A step: warp 0 finds the pivot (integer comparisons: the diagonal is positive where it
// matters) and scales its row, warp 1 sums the trace for the filter; a barrier; warp w
// updates the active slots t + 1 + w and t + 33 + w, lanes over the row from the diagonal;
// a barrier.  The chain is the square root, the division and two barriers; one warp doing
// all of it took 389 us at 64 columns, now 105.
template <bool PIVOT>
__device__ int chol64(Panel64Smem& sm, int nb, int rows, double tol_loc) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid < MAXB) sm.ord[tid] = tid;
  if (tid == 0) sm.stop = 0;
  // warp 1: slot s of lane and lane + 32 counted from t, as the filter sums them
  double total = 0.0;
  int o0 = lane, o1 = lane + 32;   // its own copy of the slot map (warp 0 is moving the shared one)
  __syncthreads();
  if (PIVOT && w == 1) {
    double d = 0.0;
    if (lane < nb) d += sm.S[lane][lane];
    if (lane + 32 < nb) d += sm.S[lane + 32][lane + 32];
    total = __shfl_sync(0xffffffffu, warp_sum(d), 0);
  }
  for (int t = 0; t < rows; ++t) {
    if (w == 0) {
      int pv = t;
      if (PIVOT) {
        // (value, lowest slot) of the largest positive diagonal entry among the slots >= t
        const int c0 = sm.ord[lane], c1 = sm.ord[lane + 32];
        const double d0 = lane >= t && lane < nb ? sm.S[c0][c0] : 0.0;
        const double d1 = lane + 32 >= t && lane + 32 < nb ? sm.S[c1][c1] : 0.0;
        const double best = d1 > d0 ? d1 : d0;
        const unsigned hi = best > 0.0 ? (unsigned)__double2hiint(best) : 0u;
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh && hi ? (unsigned)__double2loint(best) : 0u);
        const double mx = __hiloint2double((int)mh, (int)ml);
        const unsigned b0 = __ballot_sync(0xffffffffu, d0 == mx), b1 = __ballot_sync(0xffffffffu, d1 == mx);
        const bool none = mh == 0u && ml == 0u;
        const int slot = none ? t : b0 ? __ffs(b0) - 1 : 31 + __ffs(b1);
        const int o = sm.ord[t];
        pv = sm.ord[slot];
        __syncwarp();
        if (lane == 0) {
          if (none) sm.stop = 1;
          sm.ord[t] = pv;
          sm.ord[slot] = o;
        }
        __syncwarp();
      }
      const double rtt = sqrt(PIVOT ? sm.S[pv][pv] : fmax(sm.S[pv][pv], 0.0));
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int s = lane + 32 * u;
        if (s > t && s < nb) {
          const int c = sm.ord[s];
          sm.R[t][c] = sm.S[min(pv, c)][max(pv, c)] / rtt;
        }
      }
      if (lane == 0) sm.R[t][pv] = rtt;
    } else if (PIVOT && w == 1) {
      // slots t + lane, then t + lane + 32, in the order of the slots after the swaps so far
      const int s0 = t + lane, s1 = t + lane + 32;
      const int q0 = __shfl_sync(0xffffffffu, o0, s0 & 31), q1 = __shfl_sync(0xffffffffu, o1, s0 & 31);
      double rem = 0.0;
      if (s0 < nb) {
        const int c = s0 < 32 ? q0 : q1;
        rem += sm.S[c][c];
      }
      if (s1 < nb) rem += sm.S[q1][q1];   // s1 >= 32, and s1 & 31 == s0 & 31
      rem = warp_sum(rem);
      if (lane == 0 && (!(total > 0.0) || rem / total < tol_loc)) sm.stop = 1;
    }
    __syncthreads();
    if (PIVOT && sm.stop) return t;
    if (PIVOT && w == 1) {
      o0 = sm.ord[lane];
      o1 = sm.ord[lane + 32];
    }
    for (int ss = t + 1 + w; ss < nb; ss += 32) {
      const int c = sm.ord[ss];
      const double rc = sm.R[t][c];
      for (int s2 = ss + lane; s2 < nb; s2 += 32) {
        const int c2 = sm.ord[s2];
        double& x = sm.S[min(c, c2)][max(c, c2)];
        x = fma(-rc, sm.R[t][c2], x);
      }
    }
    __syncthreads();
  }
  return rows;
}

// k_pchol (one CTA): CPQR pivots and the robust filter from the panel's Gram matrix;
// publishes the pivots (ord), the kept count and R11 in slot order, and swaps the block in
// perm and diags (matlab/RBRP.m:81-99: K1 = block positions not kept, ascending; K2 = kept
// positions outside the block, in pivot order).
__global__ void __launch_bounds__(1024)
k_pchol(const double* __restrict__ G, int m, State* st, double tol_loc, const int* __restrict__ js,
        int* __restrict__ perm, double* __restrict__ diags, double* __restrict__ R11g, int* __restrict__ ordg,
        int* __restrict__ Jg, int* __restrict__ K1g, int* __restrict__ K2g) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  Panel64Smem& sm = *reinterpret_cast<Panel64Smem*>(dyn_smem);
  const int tid = threadIdx.x;
  const int nb = st->bs_sampled, i = st->i;
  for (int x = tid; x < MAXB * MAXB; x += 1024) {
    const int a = x / MAXB, c = x % MAXB;
    sm.S[a][c] = (a < nb && c < nb) ? G[x] : 0.0;
  }
  const int kept = chol64<true>(sm, nb, min(nb, m), tol_loc);
  for (int x = tid; x < MAXB * MAXB; x += 1024) {
    const int a = x / MAXB, c = x % MAXB;
    R11g[x] = (c < kept && a <= c) ? sm.R[a][sm.ord[c]] : 0.0;
  }
  if (tid < MAXB) ordg[tid] = sm.ord[tid];
  block_swap_parallel<MAXB>(sm, i, kept, js, perm, diags, Jg, K1g, K2g, st);
}

// Out(:, out0 + s) = In(:, ord) F^{-1} for TR rows (ord NULL: as stored), F upper triangular
// kept x kept: forward substitution with the columns still to come updated as soon as an
// entry is known, so a tile's TR x 64 entries work at once and each is reduced in column
// order.  One barrier per column; the division is the owning warp's alone.
template <int TR>
__global__ void __launch_bounds__(256)
k_panel_solve(const double* __restrict__ In, int m, const State* __restrict__ st, const double* __restrict__ Fg,
              const int* __restrict__ ordg, double* __restrict__ Out, int64_t ldo, int out_at_i) {
  constexpr int NG = RowMap<TR>::NG, NV = RowMap<TR>::NV;
  __shared__ double Fs[MAXB][MAXB + 1];
  __shared__ double ws[2][TR];
  const int tid = threadIdx.x, row = tid % TR, g = tid / TR;
  const int kept = st->bs;
  if (kept == 0) return;
  const int r = blockIdx.x * TR + row;
  for (int x = tid; x < kept * MAXB; x += 256) Fs[x / MAXB][x % MAXB] = Fg[x];
  double x[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = g + NG * v;
    x[v] = (r < m && c < kept) ? In[r + (int64_t)(ordg ? ordg[c] : c) * m] : 0.0;
  }
  __syncthreads();
  const int glast = (tid | 31) / TR;   // the warp's last column group
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    for (int gg = 0; gg < NG; ++gg) {
      const int u = gg + NG * v;       // the column that becomes known
      if (u >= kept) break;
      if (g == gg) {
        x[v] = x[v] / Fs[u][u];
        ws[u & 1][row] = x[v];
      }
      __syncthreads();
      const double wv = ws[u & 1][row];
#pragma unroll
      for (int q = v; q < NV; ++q) {
        if (glast + NG * q > u && (g & ~(32 / TR - 1)) + NG * q < kept) {
          const int c = g + NG * q;
          const double y = fma(-wv, Fs[u][c], x[q]);
          x[q] = c > u ? y : x[q];
        }
      }
    }
  }
  const int o = out_at_i ? st->i : 0;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = g + NG * v;
    if (r < m && c < kept) Out[r + (int64_t)(o + c) * ldo] = x[v];
  }
}

// k_chol2 (one CTA): R2 = chol(Q1^T Q1), upper, for the second row solve.
__global__ void __launch_bounds__(1024)
k_chol2(const double* __restrict__ G2, const State* __restrict__ st, double* __restrict__ R2g) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  Panel64Smem& sm = *reinterpret_cast<Panel64Smem*>(dyn_smem);
  const int tid = threadIdx.x;
  const int kept = st->bs;
  if (kept == 0) return;
  for (int x = tid; x < MAXB * MAXB; x += 1024) {
    const int a = x / MAXB, c = x % MAXB;
    sm.S[a][c] = (a < kept && c < kept) ? G2[x] : 0.0;
  }
  chol64<false>(sm, kept, kept, 0.0);
  for (int x = tid; x < MAXB * MAXB; x += 1024) {
    const int a = x / MAXB, c = x % MAXB;
    R2g[x] = (c < kept && a <= c) ? sm.R[a][c] : 0.0;
  }
}

// The panel R = R2 R11 into R(I2, I2) (matlab/RBRP.m:78), four rows per CTA.
__global__ void __launch_bounds__(256)
k_panel_r(const State* __restrict__ st, const double* __restrict__ R11g, const double* __restrict__ R2g,
          double* __restrict__ R, int64_t ldr) {
  const int kept = st->bs, i = st->i;
  const int a = blockIdx.x * 4 + (threadIdx.x >> 6), c = threadIdx.x & 63;
  if (a >= kept || c >= kept) return;
  double v = 0.0;
#pragma unroll 4
  for (int u = a; u <= c; ++u) v = fma(R2g[a * MAXB + u], R11g[u * MAXB + c], v);
  R[(int64_t)(i + a) * ldr + (i + c)] = v;
}

}  // namespace
}  // namespace rbrp
