// rbrp_pchol_df.cuh - double-float pivoted Cholesky with the robust filter
// and the block swap, for panels of up to BB columns (BB = 16, 32 or 64).
// Used by the one-matrix panel kernel (BB = 64) and the batched kernel.
#pragma once
#include "rbrp_common.cuh"
#include "rbrp_df.cuh"

namespace rbrp {
namespace {

template <int BB>
struct PcholDfSmemT {
  dfl S[BB][BB + 1];  // Schur complement, indexed by panel column
  dfl R[BB][BB + 1];  // R[t][j]: row t of the factor, by panel column j
  int ord[BB];        // slot -> panel column
  int alive[BB];
  int J[BB], K1[BB], K2[BB], inblk[BB], Tperm[BB];
  int stop, piv, nK;
  dfl inv;
};

// Block swap of perm and diags (matlab/RBRP.m:81-99), in parallel: K1 = block
// positions not kept (ascending), K2 = kept positions outside the block (pivot
// order), compacted with warp ballots.  All threads call it after `kept` is known.
template <int BB, typename Smem>
__device__ void block_swap_parallel(Smem& sm, int i, int kept, const int* __restrict__ js,
                                    int* __restrict__ perm, double* __restrict__ diags, int* __restrict__ Jg,
                                    int* __restrict__ K1g, int* __restrict__ K2g, State* st) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid < BB) sm.inblk[tid] = 0;
  __syncthreads();
  if (tid < kept) {
    const int p = js[sm.ord[tid]];
    sm.J[tid] = p;
    Jg[tid] = p;
    if (p >= i && p < i + kept) sm.inblk[p - i] = 1;
    sm.Tperm[tid] = perm[p];
  }
  __syncthreads();
  if (wid < 2) {
    // warp 0: K1 (block positions not kept), warp 1: K2 (kept positions outside the block)
    int count = 0;
    for (int base = 0; base < kept; base += 32) {
      const int t = base + lane;
      bool flag = false;
      int val = 0;
      if (t < kept) {
        if (wid == 0) { flag = !sm.inblk[t]; val = i + t; }
        else { const int p = sm.J[t]; flag = p < i || p >= i + kept; val = p; }
      }
      const unsigned bal = __ballot_sync(0xffffffffu, flag);
      if (flag) {
        const int slot = count + __popc(bal & ((1u << lane) - 1u));
        if (wid == 0) sm.K1[slot] = val; else sm.K2[slot] = val;
      }
      count += __popc(bal);
    }
    if (wid == 1 && lane == 0) sm.nK = count;
  }
  __syncthreads();
  const int nK = sm.nK;
  if (tid < nK) {  // perm(K2) = perm(K1), diags(K2) = diags(K1): K1 inside the block, K2 outside
    const int a = sm.K1[tid], b = sm.K2[tid];
    const int pa = perm[a];
    const double da = diags[a];
    perm[b] = pa;
    diags[b] = da;
    K1g[tid] = a;
    K2g[tid] = b;
  }
  __syncthreads();
  if (tid < kept) perm[i + tid] = sm.Tperm[tid];
  if (tid == 0) {
    st->bs = kept;
    st->nK = nK;
    st->zero_panel = kept == 0;
  }
}

// Pivoted Cholesky of a panel Gram matrix with the robust filter, in
// double-float, by 256 threads.  On entry sm.S holds the nb x nb Gram matrix
// (zero elsewhere), sm.ord the identity and sm.alive[j] = (j < nb).  Pivots
// follow LAPACK dgeqp3 (the first slot of maximal Schur diagonal); the filter
// (python/RBRP.ipynb cell 11 lines 69-73) stops once the remaining trace falls
// below tol_loc of the total.  Swaps are virtual (ord maps slot -> panel
// column), so sm.R[t][j] holds row t of the factor by panel column j.
// Returns the number of kept pivots.
template <int BB>
__device__ int pchol_filter_df(PcholDfSmemT<BB>& sm, int nb, int rows, double tol_loc) {
  constexpr int U = BB / 16;  // U x U Schur entries per thread: rows ty*U+u, columns tx*U+v
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int ty = tid >> 4, tx = tid & 15;
  // trace(G) and the stop threshold tol_loc * trace as a double-float, used by warp 0:
  // the per-step test rem < thr stays on the FP32 pipe (rem / trace < tol_loc, no FP64 divide)
  bool have_total = false;
  dfl thr = {0.f, 0.f};
  if (wid == 0) {
    dfl t = {0.f, 0.f};
    for (int s2 = 0; s2 < nb; ++s2) t = df_add(t, sm.S[s2][s2]);
    const double total = df_dbl(t);
    have_total = total > 0.0;
    thr = df_of(tol_loc * total);
  }
  int kept = rows;
  for (int t = 0; t < rows; ++t) {
    if (wid == 0) {
      // remaining trace and the first maximal slot (LAPACK dgeqp3 order)
      dfl rem = {0.f, 0.f}, best = {-1.f, 0.f};
      int bs = nb;
      for (int s2 = t + lane; s2 < nb; s2 += 32) {
        const dfl d = sm.S[sm.ord[s2]][sm.ord[s2]];
        rem = df_add(rem, d);
        if (df_gt(d, best)) { best = d; bs = s2; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const dfl orem = {__shfl_down_sync(0xffffffffu, rem.hi, o), __shfl_down_sync(0xffffffffu, rem.lo, o)};
        rem = df_add(rem, orem);
        const dfl ob = {__shfl_down_sync(0xffffffffu, best.hi, o), __shfl_down_sync(0xffffffffu, best.lo, o)};
        const int oi = __shfl_down_sync(0xffffffffu, bs, o);
        if (df_gt(ob, best) || (df_eq(ob, best) && oi < bs)) { best = ob; bs = oi; }
      }
      if (lane == 0) {
        const bool stop = !have_total || df_gt(thr, rem) || !(best.hi > 0.f);
        sm.stop = stop;
        if (!stop) {
          const int o = sm.ord[t];
          sm.ord[t] = sm.ord[bs];
          sm.ord[bs] = o;
          const int pv = sm.ord[t];
          sm.alive[pv] = 0;
          const dfl r = df_sqrt(sm.S[pv][pv]);
          sm.R[t][pv] = r;
          sm.inv = df_recip(r);
          sm.piv = pv;
        }
      }
    }
    __syncthreads();
    if (sm.stop) { kept = t; break; }
    const int pv = sm.piv;
    const dfl inv = sm.inv;
    if (tid < nb && sm.alive[tid]) sm.R[t][tid] = df_mul(sm.S[pv][tid], inv);
    __syncthreads();
    dfl ru[U], rv[U];
    bool au[U], av[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = ty * U + u;
      au[u] = j < nb && sm.alive[j];
      ru[u] = sm.R[t][j];
      const int c = tx * U + u;
      av[u] = c < nb && sm.alive[c];
      rv[u] = sm.R[t][c];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int v = 0; v < U; ++v)
        if (au[u] && av[v]) sm.S[ty * U + u][tx * U + v] = df_fms(sm.S[ty * U + u][tx * U + v], ru[u], rv[v]);
    __syncthreads();
  }
  return kept;
}

// The same factorization and filter as pchol_filter_df<64>, by 1024 threads
// (LEAN_THREADS).  A step: warp 0 scales the pivot's row, warp 1 applies the filter; a
// barrier; warps 2 .. 31 update the active slots, lanes over the columns as they are
// stored (active ones; by slot, the permuted columns cost several shared-memory
// wavefronts), while warps 0 and 1, which carry the diagonal in registers, find the next
// pivot with its square root and reciprocal (reductions of the bit patterns, first slot on
// ties) and the remaining trace; a barrier.  Each Schur entry gets the same double-float
// operation on the same inputs as in the 256-thread form, both triangles (the
// low parts of an entry and its mirror differ with the order of the factors).
// Square root and reciprocal start from the correctly rounded FP32 intrinsics.
// Latency bound on one SM: 64 steps of two barriers and the pivot's chain.  With
// every thread scaling its own rows, a pivot search by shuffles and no
// compaction a step took 4,000 clocks, with the pivot found at its start 3,300, now 2,800
// (an adjoint call's 64 panels at 8192 rows: 11.0 -> 9.9 ms).
constexpr int LEAN_THREADS = 1024;

__device__ __forceinline__ dfl df_sqrt_lean(dfl a) {
  if (!(a.hi > 0.0f)) return {0.0f, 0.0f};
  const float sq = __fsqrt_rn(a.hi);
  const dfl e = df_add(a, df_neg(df_mul({sq, 0.0f}, {sq, 0.0f})));  // a - sq^2
  return df_fast(sq, e.hi * (0.5f * __frcp_rn(sq)));
}
__device__ __forceinline__ dfl df_recip_lean(dfl b) {
  const float q = __frcp_rn(b.hi);
  const dfl r = df_add({1.0f, 0.0f}, df_neg(df_mul({q, 0.0f}, b)));  // 1 - q b
  return df_fast(q, q * r.hi);
}

__device__ int pchol_filter_df_lean(PcholDfSmemT<64>& sm, int nb, int rows, double tol_loc) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  bool a0 = lane < nb, a1 = lane + 32 < nb;   // the lane's columns still active
  // warps 0 and 1: the lane's diagonal entries, kept up beside the update of the matrix, so
  // that the next pivot and the remaining trace are found while the other warps update
  dfl d0 = {0.f, 0.f}, d1 = {0.f, 0.f};
  int s0 = lane, s1 = lane + 32;              // warp 0: the slots of the lane's columns
  int pv = 0, bs = 0;                         // warp 0: the next pivot column and its slot
  bool none = false;
  dfl r = {0.f, 0.f}, inv = {0.f, 0.f}, rem = {0.f, 0.f}, thr = {0.f, 0.f};
  bool have_total = false;
  auto trace = [&]() {   // remaining trace, valid in lane 0
    dfl t = {0.f, 0.f};
    if (a0) t = df_add(t, d0);
    if (a1) t = df_add(t, d1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      t = df_add(t, {__shfl_down_sync(0xffffffffu, t.hi, o), __shfl_down_sync(0xffffffffu, t.lo, o)});
    return t;
  };
  auto find = [&]() {    // largest active diagonal entry, lowest slot on ties
    dfl best = {-1.f, 0.f};
    int slot = 64, col = 0;
    if (a0) { best = d0; slot = s0; col = lane; }
    if (a1 && (slot == 64 || df_gt(d1, best) || (df_eq(d1, best) && s1 < slot))) { best = d1; slot = s1; col = lane + 32; }
    const unsigned hi = best.hi > 0.f ? __float_as_uint(best.hi) : 0u;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lb = __float_as_uint(best.lo + 0.f);   // -0 as +0
    const unsigned lo = hi == mh ? ((lb & 0x80000000u) ? ~lb : (lb | 0x80000000u)) : 0u;
    const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
    const bool mine = hi == mh && lo == ml;
    const unsigned key = __reduce_min_sync(0xffffffffu, mine ? ((unsigned)slot << 6) | (unsigned)col : 0xffffffffu);
    none = mh == 0u;
    bs = (int)(key >> 6);
    pv = (int)(key & 63u);
    // every matching lane holds the same value
    const int src = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
    const dfl v = {__shfl_sync(0xffffffffu, best.hi, src), __shfl_sync(0xffffffffu, best.lo, src)};
    r = df_sqrt_lean(v);
    inv = df_recip_lean(r);
  };
  if (tid == 0) sm.stop = 0;
  __syncthreads();
  if (w < 2) {
    if (a0) d0 = sm.S[lane][lane];
    if (a1) d1 = sm.S[lane + 32][lane + 32];
    if (w == 0) find();
    if (w == 1) {
      rem = trace();
      const double total = __shfl_sync(0xffffffffu, df_dbl(rem), 0);
      have_total = total > 0.0;
      thr = df_of(tol_loc * total);
    }
  }
  for (int t = 0; t < rows; ++t) {
    if (w == 0) {
      if (none) {
        if (lane == 0) sm.stop = 1;
      } else {
        if (lane == 0) {
          // LAPACK order: the pivot column moves to slot t, slot t's column to the pivot's slot
          const int o = sm.ord[t];
          sm.ord[t] = pv;
          sm.ord[bs] = o;
          sm.piv = pv;
        }
        if (a0) sm.R[t][lane] = pv == lane ? r : df_mul(sm.S[pv][lane], inv);
        if (a1) sm.R[t][lane + 32] = pv == lane + 32 ? r : df_mul(sm.S[pv][lane + 32], inv);
      }
    } else if (w == 1) {
      if (lane == 0 && (!have_total || df_gt(thr, rem))) sm.stop = 1;
    }
    __syncthreads();
    if (sm.stop) return t;
    a0 = a0 && sm.piv != lane;
    a1 = a1 && sm.piv != lane + 32;
    const dfl g0 = a0 ? sm.R[t][lane] : dfl{0.f, 0.f}, g1 = a1 ? sm.R[t][lane + 32] : dfl{0.f, 0.f};
    if (w < 2) {
      if (a0) d0 = df_fms(d0, g0, g0);
      if (a1) d1 = df_fms(d1, g1, g1);
      if (w == 0) {
        if (s0 == t) s0 = bs;   // slot t's column took the pivot's slot
        if (s1 == t) s1 = bs;
        find();
      } else {
        rem = trace();
      }
    } else {
      for (int ss = t + w - 1; ss < nb; ss += LEAN_THREADS / 32 - 2) {
        const int c = sm.ord[ss];
        const dfl f = sm.R[t][c];
        dfl x0 = {0.f, 0.f}, x1 = {0.f, 0.f};
        if (a0) x0 = sm.S[c][lane];
        if (a1) x1 = sm.S[c][lane + 32];
        if (a0) sm.S[c][lane] = df_fms(x0, f, g0);
        if (a1) sm.S[c][lane + 32] = df_fms(x1, f, g1);
      }
    }
    __syncthreads();
  }
  return rows;
}

}  // namespace
}  // namespace rbrp
