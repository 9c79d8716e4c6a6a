// rbrp_fixed.cuh - FP64-accurate products of narrow blocks (b <= 8) in fixed point.
//
// Greedy b = 1 is column-pivoted QR: each step multiplies one basis vector with every
// remaining column, 8 bytes of A per FMA.  On the FP64 pipe (1.6 FMAs per clock and SM) that
// takes 2.5 times the time of reading A.  Here an entry x of a column with |x| < 2^e is the
// integer X = rint(x 2^(54 - e)) = h 2^28 + l (|h| <= 2^26, |l| <= 2^27), and the products
// h h', h l' + l h' and l l' accumulate exactly in 64-bit integers (IMAD.WIDE): 55 bits below
// each column's largest entry, rounded once at the end.  A is converted once per run, into a
// copy of the same size: converting where it is read took 40 integer instructions per entry,
// as long as the FP64 pipe.  8192 x 8192: 200 us a step on the FP64 pipe, 100 here, 81 at the
// HBM copy rate.
#pragma once
#include "rbrp_slices.cuh"

namespace rbrp {
namespace {

constexpr int FIX_MAX_ROWS = 32768;   // sum of h h' over the m / 32 rows of a lane below 2^62

// Limbs of x for |x| < 2^e.
__device__ __forceinline__ void fixed_limbs(double x, int e, int& h, int& l) {
  const unsigned hw = (unsigned)__double2hiint(x), lw = (unsigned)__double2loint(x);
  const int ex = (int)((hw >> 20) & 0x7FFu);
  const unsigned mh = (hw & 0xFFFFFu) | (ex ? 0x100000u : 0u);
  // |X| = mant 2^sh, sh <= 1: the mantissa shifted left by 2, then right by r >= 1 less one
  // place, rounded there
  const int r = 1023 + e - (ex ? ex : 1);            // = 2 - sh >= 1
  unsigned uh = __funnelshift_l(lw, mh, 2), ul = lw << 2;
  const int q = r - 1;
  if (q >= 32) { ul = uh; uh = 0u; }
  if (q >= 64) ul = 0u;
  const unsigned sl = __funnelshift_r(ul, uh, q & 31), shh = uh >> (q & 31);
  unsigned long long X = ((unsigned long long)shh << 32) | sl;
  X = (X + 1) >> 1;
  const long long S = (int)hw < 0 ? -(long long)X : (long long)X;
  l = ((int)((unsigned)S << 4)) >> 4;
  h = (int)((S - l) >> 28);
}

// Limbs (h, l) of A's columns, columns as they are stored, m pairs each.
__global__ void __launch_bounds__(256)
k_fix_cols(const double* __restrict__ A, int64_t lda, int m, int n, const int* __restrict__ exA,
           int2* __restrict__ X) {
  const int lane = threadIdx.x & 31, c = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (c >= n) return;
  const int e = exA[c];
  const double* col = A + (int64_t)c * lda;
  int2* x = X + (int64_t)c * m;
#pragma unroll 4
  for (int r = lane; r < m; r += 32) {
    int h, l;
    fixed_limbs(col[r], e, h, l);
    x[r] = make_int2(h, l);
  }
}

// Limbs and exponents of the block's basis columns: FIX layout [column][limb][row].  Columns that
// are not finite end the run as in k_slice_q.
__global__ void __launch_bounds__(256)
k_fix_q(const double* __restrict__ Q, int64_t ldq, int m, int n, State* __restrict__ st, int* __restrict__ lim,
        int* __restrict__ exps) {
  __shared__ unsigned s_mx[8];
  const int tid = threadIdx.x, a = blockIdx.x;
  if (a >= st->bs) return;
  const double* col = Q + (int64_t)(st->i + a) * ldq;
  unsigned mx = 0u;
  for (int r = tid; r < m; r += 256) mx = max(mx, (unsigned)__double2hiint(col[r]) & 0x7FFFFFFFu);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((tid & 31) == 0) s_mx[tid >> 5] = mx;
  __syncthreads();
  for (int w = 0; w < 8; ++w) mx = max(mx, s_mx[w]);
  const int e = tc::slice_exponent(mx);
  if (tid == 0 && mx >= 0x7FF00000u && st->i + st->bs < n) atomicCAS(&st->status, 0, ST_ERR_NUMERIC);
  if (tid == 0) exps[a] = e;
  for (int r = tid; r < m; r += 256) {
    int h, l;
    fixed_limbs(col[r], e, h, l);
    lim[(int64_t)(2 * a) * m + r] = h;
    lim[(int64_t)(2 * a + 1) * m + r] = l;
  }
}

// a7 + a8 for b <= 8 (k_project_skinny's work): each warp streams CW whole columns, coalesced
// over rows, against the limbs of KB basis vectors in shared memory; a lane's exact partial sums
// are combined by a butterfly.
template <int KB>
struct FixTile {
  static constexpr int CW = KB <= 1 ? 4 : KB <= 4 ? 2 : 1;   // columns per warp: 3 sums of 64 bits each
  static constexpr int COLS = 8 * CW;                        // positions per CTA
  static constexpr int MC = KB <= 1 ? 1024 : 256;            // rows per stage
};

template <int KB>
__global__ void __launch_bounds__(256)
k_project_fix(const int* __restrict__ lim, const int* __restrict__ exQ, const int2* __restrict__ X,
              const int* __restrict__ exA, const int* __restrict__ perm, const State* __restrict__ st, int m, int n,
              double* __restrict__ R, int64_t ldr, double* __restrict__ diags, double* __restrict__ part_res,
              int* __restrict__ part_nnz) {
  constexpr int CW = FixTile<KB>::CW, MC = FixTile<KB>::MC, NW = 8;
  __shared__ int Qs[KB][2][MC];
  __shared__ double red_s[NW];
  __shared__ int red_c[NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i = st->i, kept = min(st->bs, KB);   // kept <= b <= KB by the host's choice
  const int pbase = i + st->bs + blockIdx.x * FixTile<KB>::COLS;
  if (kept == 0 || pbase >= n) {
    if (tid == 0) { part_res[blockIdx.x] = 0.0; part_nnz[blockIdx.x] = 0; }
    return;
  }
  const int2* col[CW];
  int ex[CW];
#pragma unroll
  for (int c = 0; c < CW; ++c) {
    const int p = pbase + warp * CW + c;
    const int pc = p < n ? perm[p] : perm[n - 1];
    col[c] = X + (int64_t)pc * m;
    ex[c] = exA[pc];
  }
  long long hh[CW][KB], hl[CW][KB], ll[CW][KB];
#pragma unroll
  for (int c = 0; c < CW; ++c)
#pragma unroll
    for (int a = 0; a < KB; ++a) hh[c][a] = hl[c][a] = ll[c][a] = 0;
  for (int r0 = 0; r0 < m; r0 += MC) {
    __syncthreads();
    for (int x = tid; x < KB * 2 * MC; x += 256) {
      const int a = x / (2 * MC), k = x / MC & 1, rr = x % MC;
      Qs[a][k][rr] = (a < kept && r0 + rr < m) ? lim[(int64_t)(2 * a + k) * m + r0 + rr] : 0;
    }
    __syncthreads();
    // 4 rows of every column in flight per lane
#pragma unroll 2
    for (int r4 = 0; r4 < MC; r4 += 128) {
      int2 v[4][CW];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int c = 0; c < CW; ++c) {
          const int r = r0 + r4 + 32 * u + lane;
          v[u][c] = r < m ? __ldg(col[c] + r) : make_int2(0, 0);
        }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int rr = r4 + 32 * u + lane;
#pragma unroll
        for (int c = 0; c < CW; ++c) {
          const int h = v[u][c].x, l = v[u][c].y;
#pragma unroll
          for (int a = 0; a < KB; ++a) {
            const int qh = Qs[a][0][rr], ql = Qs[a][1][rr];
            hh[c][a] += (long long)h * qh;
            hl[c][a] += (long long)h * ql;
            hl[c][a] += (long long)l * qh;
            ll[c][a] += (long long)l * ql;
          }
        }
      }
    }
    if (((r0 / MC + 1) * MC & 8191) == 0) {   // 256 rows a lane: the middle sum stays below 2^63
#pragma unroll
      for (int c = 0; c < CW; ++c)
#pragma unroll
        for (int a = 0; a < KB; ++a) {
          hl[c][a] += ll[c][a] >> 28;
          ll[c][a] &= 0xFFFFFFF;
          hh[c][a] += hl[c][a] >> 28;
          hl[c][a] &= 0xFFFFFFF;
        }
    }
  }
  double dsum = 0.0;
  int dcnt = 0;
#pragma unroll
  for (int c = 0; c < CW; ++c) {
    const int p = pbase + warp * CW + c;
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < KB; ++a) {
      // carries up first, so that the lanes' sums cannot overflow: t 2^84 + z 2^56 + y 2^28 + x
      // in units 2^(ex + eq - 108)
      long long x = ll[c][a], y = hl[c][a] + (x >> 28), z = hh[c][a] + (y >> 28), t = z >> 28;
      x &= 0xFFFFFFF;
      y &= 0xFFFFFFF;
      z &= 0xFFFFFFF;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
        z += __shfl_xor_sync(0xffffffffu, z, o);
        t += __shfl_xor_sync(0xffffffffu, t, o);
      }
      if (lane == 0 && p < n && a < kept) {
        // over 2^40: (t 2^20) 2^24 + z 2^16 + (y 2^28 + x) / 2^40
        const double w = tc::slice_value(t << 20, (z << 16) + (((y << 28) + x) >> 40), ex[c] + exQ[a] - 68);
        R[(int64_t)(i + a) * ldr + p] = w;
        s = fma(w, w, s);
      }
    }
    if (lane == 0 && p < n) {
      double d = diags[p] - s;
      d = d > 0.0 ? d : (d == d ? 0.0 : d);
      diags[p] = d;
      dsum += d;
      dcnt += d > 0.0;
    }
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

// The panel of one column (b = 1), one CTA: its norm, the two passes of CholQR2, the block
// swap, R(i, i) and the limbs of the new basis vector - what k_gram64, k_pchol, k_panel_solve,
// k_chol2 and k_panel_r do for wider blocks in ten launches.
__global__ void __launch_bounds__(1024)
k_panel_one(const double* __restrict__ V, int m, State* st, double tol_loc, const int* __restrict__ js,
            int* __restrict__ perm, double* __restrict__ diags, double* __restrict__ Q, int64_t ldq,
            double* __restrict__ R, int64_t ldr, int* __restrict__ lim, int* __restrict__ exps, int* __restrict__ Jg,
            int* __restrict__ K1g, int* __restrict__ K2g) {
  __shared__ double sh[32];
  __shared__ unsigned s_mx[32];
  const int tid = threadIdx.x, i = st->i, nb = st->bs_sampled;
  double g = 0.0;
  if (nb > 0)
    for (int r = tid; r < m; r += 1024) g = fma(V[r], V[r], g);
  g = block_sum(g, sh);
  const bool keep = nb > 0 && g > 0.0 && !(1.0 < tol_loc);
  if (tid == 0) {
    if (keep) {
      const int p = js[0], pp = perm[p];
      Jg[0] = p;
      if (p != i) {
        K1g[0] = i;
        K2g[0] = p;
        perm[p] = perm[i];
        diags[p] = diags[i];
        perm[i] = pp;
      }
      st->nK = p != i;
    } else {
      st->nK = 0;
    }
    st->bs = keep ? 1 : 0;
    st->zero_panel = keep ? 0 : 1;
  }
  if (!keep) return;
  const double r11 = sqrt(g), x11 = 1.0 / r11;
  double* q = Q + (int64_t)i * ldq;
  double g2 = 0.0;
  for (int r = tid; r < m; r += 1024) {
    const double y = V[r] * x11;
    q[r] = y;
    g2 = fma(y, y, g2);
  }
  g2 = block_sum(g2, sh);
  const double r2 = sqrt(g2), x2 = 1.0 / r2;
  unsigned mx = 0u;
  for (int r = tid; r < m; r += 1024) {
    const double y = q[r] * x2;
    q[r] = y;
    mx = max(mx, (unsigned)__double2hiint(y) & 0x7FFFFFFFu);
  }
  if (tid == 0) R[(int64_t)i * ldr + i] = r2 * r11;
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((tid & 31) == 0) s_mx[tid >> 5] = mx;
  __syncthreads();
  for (int w = 0; w < 32; ++w) mx = max(mx, s_mx[w]);
  const int e = tc::slice_exponent(mx);
  if (tid == 0) exps[0] = e;
  for (int r = tid; r < m; r += 1024) {
    int h, l;
    fixed_limbs(q[r], e, h, l);
    lim[r] = h;
    lim[m + r] = l;
  }
}

}  // namespace
}  // namespace rbrp
