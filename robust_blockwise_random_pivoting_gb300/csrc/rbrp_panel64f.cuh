// rbrp_panel64f.cuh - the FP64 panel where the order of its sums is free (everything but
// random draws to a squared tolerance below 1e-8, which keep the kernels of
// rbrp_panel64.cuh): no less accurate, with shorter chains on the FP64 pipe.
//
//   Gram partials per row tile of the kernel that writes the rows, summed in eight groups;
//   L D L^T instead of Cholesky, with L^{-1} carried along, so no square root or division
//   by it sits in the chain of steps and the row solves become products;
//   the second CholQR pass from G2 = I + E directly where E is small.
// 2000 x 64 panels of condition 2 to 10^8 (model): |Q^T Q - I| 5e-16 to 8e-16, with substitutions and the
// second pass in FP64 6e-16 to 9e-16; |Q R - V| per column 1.0e-15 to 1.2e-15, for 0.7e-15 to 0.9e-15.
// 500 x 2000, b = 30, rank 270: 3.3 ms a run in fixed order, 2.4 here; 8192 x 8192, b = 64, rank
// 640: 13.2 and 11.6.
#pragma once
#include "rbrp_panel64.cuh"

namespace rbrp {
namespace {

// Gram partial of a tile held column by column (T[c][r], stride LD), upper triangle, packed.
template <int TR, int LD>
__device__ __forceinline__ void tile_gram(const double (*T)[LD], int w, double* __restrict__ out) {
  for (int x = threadIdx.x; x < w * (w + 1) / 2; x += 256) {
    int a, b;
    tri_pair(x, w, a, b);
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < TR; ++r) s = fma(T[a][r], T[b][r], s);
    out[x] = s;
  }
}

// Gram partials of V (ld = m), TR rows per CTA.
template <int TR>
__global__ void __launch_bounds__(256)
k_gram_tiles(const double* __restrict__ V, int m, const State* __restrict__ st, double* __restrict__ Gpart) {
  __shared__ double Vs[MAXB][TR + 1];
  const int bss = st->bs_sampled, r0 = blockIdx.x * TR;
  for (int t = threadIdx.x; t < bss * TR; t += 256) {
    const int rr = t % TR, c = t / TR;
    Vs[c][rr] = r0 + rr < m ? V[r0 + rr + (int64_t)c * m] : 0.0;
  }
  __syncthreads();
  tile_gram<TR, TR + 1>(Vs, bss, Gpart + (int64_t)blockIdx.x * NPAIR);
}

// G = sum of the packed partials (of the bs_sampled or kept columns), both triangles: 32
// pairs per CTA, eight groups of partials summed in a fixed order.
__global__ void __launch_bounds__(256)
k_reduce_gram_fast(const double* __restrict__ part, int nparts, const State* __restrict__ st, int kept_cols,
              double* __restrict__ G) {
  __shared__ double sh[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n = kept_cols ? st->bs : st->bs_sampled;
  const int x = blockIdx.x * 32 + lane;
  const bool in = x < n * (n + 1) / 2;
  double s = 0.0;
  if (in) {
#pragma unroll 4
    for (int z = w; z < nparts; z += 8) s += part[(int64_t)z * NPAIR + x];
  }
  sh[w][lane] = s;
  __syncthreads();
  if (w == 0 && in) {
    for (int q = 1; q < 8; ++q) s += sh[q][lane];
    int a, b;
    tri_pair(x, n, a, b);
    G[a * MAXB + b] = s;
    G[b * MAXB + a] = s;
  }
}

struct LdlSmem {
  double S[MAXB][MAXB + 1];   // Schur complement: entry (a, b) of panel columns at [min][max]
  double U[MAXB][MAXB + 1];   // U[t][c]: row t of D L^T, by panel column c
  double M[MAXB][MAXB + 1];   // M[c][s]: entry s of the row of L^{-1} that column c has so far
  double l[MAXB], d[MAXB], rs[MAXB];
  int ord[MAXB];
  int J[MAXB], K1[MAXB], K2[MAXB], inblk[MAXB], Tperm[MAXB];
  int nK, stop, piv;
  float emax[32];
  unsigned cmax[MAXB];        // k_chol2_fast: largest upper word of |R11(:, c)|
};

// Warp 0 of ldl64: the diagonal by stored column (lane, lane + 32) in registers, with the
// columns' slots, and the next pivot: the largest active entry, lowest slot on ties (integer
// reductions: the diagonal is positive where it matters).
struct Pivot64 {
  double d0, d1;
  int s0, s1;
  bool a0, a1;
  double best;      // the pivot's diagonal entry
  int pv, slot;     // its column and slot
  bool none;
  __device__ void find() {
    const int lane = threadIdx.x & 31;
    double v = 0.0;
    int s = 64, c = 0;
    if (a0) { v = d0; s = s0; c = lane; }
    if (a1 && (s == 64 || d1 > v || (d1 == v && s1 < s))) { v = d1; s = s1; c = lane + 32; }
    const bool pos = s < 64 && v > 0.0;
    const unsigned hi = pos ? (unsigned)__double2hiint(v) : 0u, lo = pos ? (unsigned)__double2loint(v) : 0u;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    none = mh == 0u && ml == 0u;
    const unsigned key =
        __reduce_min_sync(0xffffffffu, pos && hi == mh && lo == ml ? ((unsigned)s << 6) | (unsigned)c : 0xffffffffu);
    slot = (int)(key >> 6);
    pv = (int)(key & 63u);
    best = __hiloint2double((int)mh, (int)ml);
  }
  // the pivot of step t is gone: the column of slot t has its slot
  __device__ void taken(int t) {
    const int lane = threadIdx.x & 31;
    a0 = a0 && pv != lane;
    a1 = a1 && pv != lane + 32;
    if (s0 == t) s0 = slot;
    if (s1 == t) s1 = slot;
  }
};

// L D L^T of the nb x nb matrix in sm.S with L^{-1} carried along, 1024 threads.  With
// PIVOT the step takes the largest remaining diagonal entry (LAPACK dgeqp3's rule on the
// panel, first slot on ties; swaps are virtual: ord maps slot -> column) and stops where
// the remaining trace falls below tol_loc of the whole (python/RBRP.ipynb cell 11 lines
// 69-73).  Returns the number of steps taken; R = D^{1/2} L^T and R^{-1} = L^{-T} D^{-1/2}
// follow from U, M and d, so no square root sits in the chain of steps.
//
// A step: warp 0 scales the pivot's row, warp 1 applies the filter; a barrier; warps 2 .. 31
// update the active rows (slots), lanes over the row's entries of L^{-1} and of the Schur
// complement together, while warps 0 and 1, which carry the diagonal in registers, find the
// next pivot with its reciprocal and the remaining trace; a barrier.  k_pchol_ldl at 64
// columns: 103 us with the pivot found at the start of the step, now 89.
template <bool PIVOT>
__device__ int ldl64(LdlSmem& sm, int nb, int rows, double tol_loc) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  Pivot64 pz;
  pz.a0 = lane < nb;
  pz.a1 = lane + 32 < nb;
  pz.d0 = pz.d1 = 0.0;
  pz.s0 = lane;
  pz.s1 = lane + 32;
  pz.none = false;
  pz.slot = 0;
  double thr = 0.0, rem = 0.0, inv = 0.0;
  if (tid < MAXB) sm.ord[tid] = tid;
  if (tid == 0) sm.stop = 0;
  __syncthreads();
  // the pivot of step t is known: its reciprocal
  auto next = [&](int t) {
    if (PIVOT) {
      pz.find();
    } else if (t < nb) {   // natural order
      pz.pv = pz.slot = t;
      pz.best = __shfl_sync(0xffffffffu, t < 32 ? pz.d0 : pz.d1, t & 31);
    }
    inv = 1.0 / pz.best;
  };
  if (w < 2) {
    if (pz.a0) pz.d0 = sm.S[lane][lane];
    if (pz.a1) pz.d1 = sm.S[lane + 32][lane + 32];
    if (w == 0) next(0);
    if (PIVOT && w == 1) {
      rem = __shfl_sync(0xffffffffu, warp_sum(pz.d0 + pz.d1), 0);
      thr = tol_loc * rem;
      if (!(rem > 0.0)) thr = INFINITY;   // a zero or NaN panel keeps nothing
    }
  }
  for (int t = 0; t < rows; ++t) {
    if (w == 0) {
      const int pv = pz.pv;
      if (PIVOT && pz.none) {
        if (lane == 0) sm.stop = 1;
      } else {
        if (lane == 0) {
          const int o = sm.ord[t];
          sm.ord[t] = pv;
          sm.ord[pz.slot] = o;
          sm.piv = pv;
          sm.d[t] = pz.best;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = lane + 32 * u;
          if ((u ? pz.a1 : pz.a0) && c != pv) {
            const double v = sm.S[min(pv, c)][max(pv, c)];
            sm.U[t][c] = v;
            sm.l[c] = v * inv;
          }
        }
      }
    } else if (PIVOT && w == 1) {
      if (lane == 0 && !(rem >= thr)) sm.stop = 1;
    }
    __syncthreads();
    if (sm.stop) return t;
    const int pv = sm.piv;
    if (w < 2) {
      if (w == 1) pz.pv = pv;
      pz.taken(t);
      if (pz.a0) pz.d0 = fma(-sm.l[lane], sm.U[t][lane], pz.d0);
      if (pz.a1) pz.d1 = fma(-sm.l[lane + 32], sm.U[t][lane + 32], pz.d1);
      if (w == 0) next(t + 1);
      else if (PIVOT) rem = warp_sum((pz.a0 ? pz.d0 : 0.0) + (pz.a1 ? pz.d1 : 0.0));
    } else {
      for (int ss = t + w - 1; ss < nb; ss += 30) {
        const int c = sm.ord[ss];
        const double lc = sm.l[c];
        const int len = t + nb - ss;               // t entries of L^{-1}, then the slots ss .. nb - 1
        for (int e = lane; e < len; e += 32) {
          double *p, q;
          if (e < t) {
            p = &sm.M[c][e];
            q = sm.M[pv][e];
          } else {
            const int c2 = sm.ord[ss + e - t];
            p = &sm.S[min(c, c2)][max(c, c2)];
            q = sm.U[t][c2];
          }
          *p = fma(-lc, q, *p);
        }
        if (lane == 0) sm.M[c][t] = -lc;
      }
    }
    __syncthreads();
  }
  return rows;
}

// k_pchol_ldl (one CTA): CPQR pivots and the robust filter from the panel's Gram matrix;
// publishes the pivots (ord), R11 and its inverse in slot order and swaps the block in
// perm and diags (matlab/RBRP.m:81-99).
__global__ void __launch_bounds__(1024)
k_pchol_ldl(const double* __restrict__ G, int m, State* st, double tol_loc, const int* __restrict__ js,
        int* __restrict__ perm, double* __restrict__ diags, double* __restrict__ R11g, double* __restrict__ X11g,
        int* __restrict__ ordg, int* __restrict__ Jg, int* __restrict__ K1g, int* __restrict__ K2g) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  LdlSmem& sm = *reinterpret_cast<LdlSmem*>(dyn_smem);
  const int tid = threadIdx.x;
  const int nb = st->bs_sampled, i = st->i;
  for (int x = tid; x < MAXB * MAXB; x += 1024) {
    const int a = x / MAXB, c = x % MAXB;
    sm.S[a][c] = (a < nb && c < nb) ? G[x] : 0.0;
  }
  __syncthreads();
  const int kept = ldl64<true>(sm, nb, min(nb, m), tol_loc);
  if (tid < kept) sm.rs[tid] = 1.0 / sqrt(sm.d[tid]);
  __syncthreads();
  for (int x = tid; x < MAXB * MAXB; x += 1024) {
    const int a = x / MAXB, c = x % MAXB;
    double r = 0.0, y = 0.0;
    if (c < kept && a == c) {
      r = sqrt(sm.d[a]);
      y = sm.rs[a];
    } else if (c < kept && a < c) {
      r = sm.U[a][sm.ord[c]] * sm.rs[a];
      y = sm.M[sm.ord[c]][a] * sm.rs[c];
    }
    R11g[x] = r;
    X11g[x] = y;
  }
  if (tid < MAXB) ordg[tid] = sm.ord[tid];
  block_swap_parallel<MAXB>(sm, i, kept, js, perm, diags, Jg, K1g, K2g, st);
}

// Rows [r0, r0 + TR) of In(:, ord) (ord NULL: as stored) into Is[s][row]; zero past m.
template <int TR>
__device__ __forceinline__ void load_rows(double (*Is)[TR + 1], const double* __restrict__ In, int m, int r0, int kept,
                                          const int* __restrict__ ord) {
  for (int t = threadIdx.x; t < kept * TR; t += 256) {
    const int rr = t % TR, s = t / TR;
    Is[s][rr] = r0 + rr < m ? In[r0 + rr + (int64_t)(ord ? ord[s] : s) * m] : 0.0;
  }
}

// acc(v) = sum_{s <= c} Is(s, row) X(s, c), c = g + NG v, for the warp's columns
template <int TR>
__device__ __forceinline__ void rows_times_upper(const double (*Is)[TR + 1], const double (*Xs)[MAXB + 1], int kept,
                                                 double (&acc)[RowMap<TR>::NV]) {
  constexpr int NG = RowMap<TR>::NG, NV = RowMap<TR>::NV;
  const int tid = threadIdx.x, row = tid % TR, g = tid / TR, gl = (tid | 31) / TR;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    acc[v] = 0.0;
    const int send = min(kept, gl + NG * v + 1);   // the warp's last column needs s <= c (X is zero beyond)
    if (g - (g % (32 / TR)) + NG * v < kept) {
#pragma unroll 4
      for (int s = 0; s < send; ++s) acc[v] = fma(Is[s][row], Xs[s][g + NG * v], acc[v]);
    }
  }
}

// Q1 = V(:, ord) R11^{-1} for TR rows, and the Gram partial of Q1.
template <int TR>
__global__ void __launch_bounds__(256)
k_panel1_fast(const double* __restrict__ V, int m, const State* __restrict__ st, const double* __restrict__ X11g,
         const int* __restrict__ ordg, double* __restrict__ Q1, double* __restrict__ G2part) {
  constexpr int NG = RowMap<TR>::NG, NV = RowMap<TR>::NV;
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  double(*Xs)[MAXB + 1] = reinterpret_cast<double(*)[MAXB + 1]>(dyn_smem);
  double(*Is)[TR + 1] = reinterpret_cast<double(*)[TR + 1]>(dyn_smem + sizeof(double) * MAXB * (MAXB + 1));
  const int tid = threadIdx.x, kept = st->bs;
  if (kept == 0) return;
  const int r0 = blockIdx.x * TR, row = tid % TR, g = tid / TR, r = r0 + row;
  for (int x = tid; x < MAXB * MAXB; x += 256) Xs[x / MAXB][x % MAXB] = X11g[x];
  load_rows<TR>(Is, V, m, r0, kept, ordg);
  __syncthreads();
  double acc[NV];
  rows_times_upper<TR>(Is, Xs, kept, acc);
  __syncthreads();
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = g + NG * v;
    if (c < kept) {
      Is[c][row] = acc[v];
      if (r < m) Q1[r + (int64_t)c * m] = acc[v];
    }
  }
  __syncthreads();
  tile_gram<TR, TR + 1>(Is, kept, G2part + (int64_t)blockIdx.x * NPAIR);
}

// The second pass of CholQR2 starts from G2 = Q1^T Q1 = I + E.  Where every |E| <= 2^-38
// (a panel of condition up to some 200; the filter admits little more), R2 = I + U with
// U = triu(E), its diagonal halved, to 64 |E|^2 <= 2^-70, and R2^{-1} = I - U.  The products
// with U add less than 2^-32 of the entries they correct, so FP32 leaves errors below
// 2^-56 of them.  Otherwise R2 and its inverse come from a Cholesky factorisation.
constexpr float CHOL2_SMALL = 0x1.0p-38f;

// k_chol2_fast (one CTA): the panel R = R2 R11 into R(I2, I2) (matlab/RBRP.m:78), and for the
// second row pass either U (FP32, *full = 0) or R2^{-1} (*full = 1).
__global__ void __launch_bounds__(1024)
k_chol2_fast(const double* __restrict__ G2, const State* __restrict__ st, const double* __restrict__ R11g,
        double* __restrict__ Y2g, float* __restrict__ U2g, int* __restrict__ full, double* __restrict__ R,
        int64_t ldr) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  LdlSmem& sm = *reinterpret_cast<LdlSmem*>(dyn_smem);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int kept = st->bs, i = st->i;
  if (kept == 0) return;
  float em = 0.f;
  if (tid < MAXB) sm.cmax[tid] = 0u;
  __syncthreads();
  for (int x = tid; x < MAXB * MAXB; x += 1024) {
    const int a = x / MAXB, c = x % MAXB;
    const bool in = a < kept && c < kept;
    const double v = in ? G2[x] : 0.0;
    sm.S[a][c] = v;
    atomicMax(&sm.cmax[c], (unsigned)__double2hiint(R11g[x]) & 0x7FFFFFFFu);
    if (in) {
      const float e = fabsf((float)(a == c ? v - 1.0 : v));
      em = e <= em ? em : e;   // (a NaN may get lost, and then spreads in either branch)
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float f = __shfl_xor_sync(0xffffffffu, em, o);
    em = f <= em ? em : f;
  }
  if (lane == 0) sm.emax[w] = em;
  __syncthreads();
  bool small = true;
  for (int x = 0; x < 32; ++x) small = small && sm.emax[x] <= CHOL2_SMALL;
  if (tid == 0) *full = small ? 0 : 1;
  if (small) {
    float(*Uf)[MAXB + 1] = reinterpret_cast<float(*)[MAXB + 1]>(&sm.U[0][0]);
    float(*Rf)[MAXB + 1] = reinterpret_cast<float(*)[MAXB + 1]>(&sm.M[0][0]);
    for (int x = tid; x < MAXB * MAXB; x += 1024) {
      const int a = x / MAXB, c = x % MAXB;
      float u = 0.f;
      if (a < kept && c < kept && a <= c) u = a == c ? 0.5f * (float)(sm.S[a][a] - 1.0) : (float)sm.S[a][c];
      Uf[a][c] = u;
      // R11 leaves FP32's range with its columns' scale: a power of two per column
      Rf[a][c] = (float)ldexp(R11g[x], 1022 - (int)(sm.cmax[c] >> 20));
      U2g[x] = u;
    }
    __syncthreads();
    for (int x = tid; x < kept * kept; x += 1024) {
      const int a = x / kept, c = x % kept;
      double v = 0.0;
      if (c >= a) {
        float s = 0.f;
        for (int u = a; u <= c; ++u) s = fmaf(Uf[a][u], Rf[u][c], s);
        v = R11g[a * MAXB + c] + ldexp((double)s, (int)(sm.cmax[c] >> 20) - 1022);
      }
      R[(int64_t)(i + a) * ldr + (i + c)] = v;
    }
    return;
  }
  ldl64<false>(sm, kept, kept, 0.0);
  if (tid < kept) sm.rs[tid] = 1.0 / sqrt(fmax(sm.d[tid], 0.0));
  __syncthreads();
  for (int x = tid; x < MAXB * MAXB; x += 1024) {
    const int a = x / MAXB, c = x % MAXB;
    double y = 0.0;
    if (c < kept && a <= c) y = a == c ? sm.rs[c] : sm.M[c][a] * sm.rs[c];
    Y2g[x] = y;
  }
  for (int x = tid; x < kept * kept; x += 1024) {
    const int a = x / kept, c = x % kept;
    double v = 0.0;
    if (c >= a) {
      v = sqrt(fmax(sm.d[a], 0.0)) * R11g[a * MAXB + c];
      for (int u = a + 1; u <= c; ++u) v = fma(sm.U[a][u] * sm.rs[a], R11g[u * MAXB + c], v);
    }
    R[(int64_t)(i + a) * ldr + (i + c)] = v;
  }
}

// Second CholQR pass: Q_blk = Q1 R2^{-1}, TR rows per CTA.
template <int TR>
__global__ void __launch_bounds__(256)
k_panel2_fast(const double* __restrict__ Q1, int m, const State* __restrict__ st, const double* __restrict__ Y2g,
         const float* __restrict__ U2g, const int* __restrict__ full, double* __restrict__ Q, int64_t ldq) {
  constexpr int NG = RowMap<TR>::NG, NV = RowMap<TR>::NV;
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  double(*Xs)[MAXB + 1] = reinterpret_cast<double(*)[MAXB + 1]>(dyn_smem);
  double(*Is)[TR + 1] = reinterpret_cast<double(*)[TR + 1]>(dyn_smem + sizeof(double) * MAXB * (MAXB + 1));
  const int tid = threadIdx.x, kept = st->bs, i = st->i;
  if (kept == 0) return;
  const int r0 = blockIdx.x * TR, row = tid % TR, g = tid / TR, r = r0 + row;
  load_rows<TR>(Is, Q1, m, r0, kept, nullptr);
  double out[NV];
  if (*full) {
    for (int x = tid; x < MAXB * MAXB; x += 256) Xs[x / MAXB][x % MAXB] = Y2g[x];
    __syncthreads();
    rows_times_upper<TR>(Is, Xs, kept, out);
  } else {
    float(*Uf)[MAXB] = reinterpret_cast<float(*)[MAXB]>(dyn_smem);
    float(*If)[TR + 1] = reinterpret_cast<float(*)[TR + 1]>(dyn_smem + sizeof(float) * MAXB * MAXB);
    for (int x = tid; x < MAXB * MAXB; x += 256) (&Uf[0][0])[x] = U2g[x];
    __syncthreads();
    for (int x = tid; x < kept * TR; x += 256) If[x / TR][x % TR] = (float)Is[x / TR][x % TR];
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c = g + NG * v;
      float s = 0.f;
      if (c < kept) {
        for (int u = 0; u <= c; ++u) s = fmaf(If[u][row], Uf[u][c], s);
        out[v] = Is[c][row] - (double)s;
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = g + NG * v;
    if (r < m && c < kept) Q[r + (int64_t)(i + c) * ldq] = out[v];
  }
}

template <int TR>
constexpr size_t panel_rows_smem() { return sizeof(double) * (MAXB * (MAXB + 1) + MAXB * (TR + 1)); }

}  // namespace
}  // namespace rbrp
