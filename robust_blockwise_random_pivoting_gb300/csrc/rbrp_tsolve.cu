// rbrp_tsolve.cu - the interpolation matrix T = R11^{-1} R12 (a10).
#include <algorithm>

#include <cuda.h>

#include "../../include/rbrp_gb300_testing.h"
#include "rbrp_internal.h"
#include "rbrp_slices.cuh"

namespace rbrp {

// ===========================================================================
// a10: T = R11^{-1} R12 (matlab/driver.m:86; gpu/interp.cu:45-105 solves the
// same triangular system after re-factoring a sketch; gpu/id_cpqr.cu:133-136).
// R is the RBRP factor (row major, ld = n, indexed by position): R11 =
// R[:k, :k] upper triangular, R12 = R[:k, k:].  T is k x (n-k), column major.
// ===========================================================================
__global__ void k_gather_T(const double* __restrict__ R, int64_t ldr, int k, int ncols, double* __restrict__ T) {
  __shared__ double tile[32][33];
  const int c0 = blockIdx.x * 32, a0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int q = 0; q < 32; q += 8) {
    const int a = a0 + ty + q, c = c0 + tx;
    tile[ty + q][tx] = (a < k && c < ncols) ? R[(int64_t)a * ldr + k + c] : 0.0;
  }
  __syncthreads();
  for (int q = 0; q < 32; q += 8) {
    const int c = c0 + ty + q, a = a0 + tx;
    if (a < k && c < ncols) T[a + (int64_t)c * k] = tile[tx][ty + q];
  }
}

struct TrsmSmem {
  double Rs[64][65];
  double Xs[64][33];
  double Acc[64][33];
};

// Block back substitution, 32 right-hand sides per CTA, 64-row diagonal blocks
// from the bottom; the update of a row block by the solved blocks below it is a
// 64 x 64 x 32 product per step.
__global__ void __launch_bounds__(256) k_trsm_T(const double* __restrict__ R, int64_t ldr, int k, int ncols,
                                                double* __restrict__ T) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  TrsmSmem& sm = *reinterpret_cast<TrsmSmem*>(dyn_smem);
  const int tid = threadIdx.x;
  const int c0 = blockIdx.x * 32;
  const int nc = min(32, ncols - c0);
  const int nbk = (k + 63) / 64;
  const int x = tid >> 2;  // output row of this thread in the 64 x 32 tile
  for (int bi = nbk - 1; bi >= 0; --bi) {
    const int b0 = bi * 64, bl = min(64, k - b0);
    for (int idx = tid; idx < 64 * 32; idx += 256) {
      const int xr = idx & 63, c = idx >> 6;
      sm.Acc[xr][c] = (xr < bl && c < nc) ? T[(b0 + xr) + (int64_t)(c0 + c) * k] : 0.0;
    }
    double acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = 0.0;
    for (int bj = bi + 1; bj < nbk; ++bj) {
      const int cr = bj * 64, cl = min(64, k - cr);
      __syncthreads();
      for (int idx = tid; idx < 64 * 64; idx += 256) {
        const int y = idx & 63, xr = idx >> 6;
        sm.Rs[xr][y] = (xr < bl && y < cl) ? R[(int64_t)(b0 + xr) * ldr + cr + y] : 0.0;
      }
      for (int idx = tid; idx < 64 * 32; idx += 256) {
        const int y = idx & 63, c = idx >> 6;
        sm.Xs[y][c] = (y < cl && c < nc) ? T[(cr + y) + (int64_t)(c0 + c) * k] : 0.0;
      }
      __syncthreads();
#pragma unroll 4
      for (int y = 0; y < 64; ++y) {
        const double r = sm.Rs[x][y];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = fma(r, sm.Xs[y][(tid & 3) + 4 * q], acc[q]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) sm.Acc[x][(tid & 3) + 4 * q] -= acc[q];
    for (int idx = tid; idx < 64 * 64; idx += 256) {
      const int y = idx & 63, xr = idx >> 6;
      sm.Rs[xr][y] = (xr < bl && y < bl && y >= xr) ? R[(int64_t)(b0 + xr) * ldr + b0 + y] : 0.0;
    }
    __syncthreads();
    if (tid < nc) {
      for (int xr = bl - 1; xr >= 0; --xr) {
        double v = sm.Acc[xr][tid];
        for (int y = xr + 1; y < bl; ++y) v = fma(-sm.Rs[xr][y], sm.Acc[y][tid], v);
        sm.Acc[xr][tid] = v / sm.Rs[xr][xr];
      }
    }
    __syncthreads();
    for (int idx = tid; idx < 64 * 32; idx += 256) {
      const int xr = idx & 63, c = idx >> 6;
      if (xr < bl && c < nc) T[(b0 + xr) + (int64_t)(c0 + c) * k] = sm.Acc[xr][c];
    }
    __syncthreads();
  }
}

// Back substitution for small ranks, k <= 32 NR: a warp per right-hand side, row 32 q + lane in
// register q, R11 in shared memory with its rows divided by their diagonal, so that a step is a
// shuffle and the updates.  Bound by the FP64 pipe, about ncols k^2 / 10^6 us, or the load of R11 and the
// chain of k steps (k = 64, 500 columns: 17 us).  The slice products below take some ten launches.
constexpr int TS_SMALL = 128;
template <int NR>
__global__ void __launch_bounds__(256)
k_trsm_small(const double* __restrict__ R, int64_t ldr, int k, int ncols, double* __restrict__ T) {
  extern __shared__ __align__(16) double small_smem[];
  constexpr int LD = 32 * NR + 1;
  double(*Rs)[LD] = reinterpret_cast<double(*)[LD]>(small_smem);              // [row][column], k rows
  double(*Bs)[LD] = reinterpret_cast<double(*)[LD]>(small_smem + k * LD);     // [right-hand side][row]
  double* ri = small_smem + (k + 8) * LD;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, c0 = blockIdx.x * 8;
  if (tid < k) ri[tid] = 1.0 / R[(int64_t)tid * ldr + tid];
  __syncthreads();
  for (int x = tid; x < k * k; x += 256) {
    const int a = x / k, j = x % k;
    if (j > a) Rs[a][j] = R[(int64_t)a * ldr + j] * ri[a];
  }
  for (int x = tid; x < 8 * k; x += 256) {
    const int a = x / 8, c = x % 8;
    Bs[c][a] = c0 + c < ncols ? R[(int64_t)a * ldr + k + c0 + c] * ri[a] : 0.0;
  }
  __syncthreads();
  if (c0 + w >= ncols) return;
  double x[NR];
#pragma unroll
  for (int q = 0; q < NR; ++q) x[q] = 32 * q + lane < k ? Bs[w][32 * q + lane] : 0.0;
#pragma unroll
  for (int r = NR - 1; r >= 0; --r) {
    for (int jj = min(31, k - 1 - 32 * r); jj >= 0; --jj) {
      const int j = 32 * r + jj;
      const double xj = __shfl_sync(0xffffffffu, x[r], jj);
#pragma unroll
      for (int q = 0; q < r; ++q) x[q] = fma(-Rs[32 * q + lane][j], xj, x[q]);
      if (lane < jj) x[r] = fma(-Rs[32 * r + lane][j], xj, x[r]);
    }
  }
#pragma unroll
  for (int q = 0; q < NR; ++q)
    if (32 * q + lane < k) T[32 * q + lane + (int64_t)(c0 + w) * k] = x[q];
}

// ===========================================================================
// The same solve as slice products (rbrp_slices.cuh): blocks of 256 (or 128) rows from the bottom up,
// X_J = inv(R11(J, J)) B_J and then B(0:j0) -= R11(0:j0, J) X_J, both on the tensor cores.
//
// A slice keeps 55 bits below the largest entry of its row (M) or column (N).  The skeleton's
// columns may differ in size by any factor and nearly depend on one another, so the terms of a
// product are brought to one size first, by what the data are: term a of the solve by the power
// of two of the largest entry of B_J(a, :), term j of the update by that of X_J(j, :).  A row i of
// X then carries 2^-55 of max_a |inv(i, a)| |B_J(a, :)|, and where that is not much more than
// |X_J(i, :)| it is as good as a substitution's.  Where it is (2^6 and more: the inverse's
// products cancel), one step of refinement for the block, X_J += inv (B_J - R11(J, J) X_J); past
// 2^44, and where something is not finite, the substitution on the FP64 pipe solves anew
// (State::t_hard).  Residuals |R11 T - R12| against |R11| |T| of kernel, Gaussian, sparse and
// nearly dependent skeletons, and of columns scaled from 2^0 to 2^60: at most 2e-15, of the FP64
// substitution 5e-16, of the 48-bit one 3e-15.  Scaled by R11's diagonal instead, which supposes
// that its rows and columns are ordered by size, a skeleton of pairs 1e-8 apart had 1e-9.
//
// What bounds it: a 128 x 64 tile over 256 values of k is 18,000 clocks of MMAs, which its
// epilogue (one FP64 subtraction per entry) runs beside; the double-float solve needed 12 FP32 operations per
// product and a warp per column in the diagonal blocks (k = 2000, 14,384 columns: 15.9 ms,
// now 3.1; k = 1000, 64,536 columns: 19.5, now 3.9; 0.4 and 0.5 of these are the scales, the
// copies of X and the launches of a refinement that is not needed).
// ===========================================================================
namespace tc {
namespace {

constexpr int TS_OB = 256;            // rows per block at the most
constexpr int TS_CHUNK = 65536;       // columns of T per pass: bounds the sliced copy to 235 MB
constexpr int TS_REFINE = 6;          // log2 of the cancellation from which X_J is refined
constexpr int TS_HARD = 44;           // and from which the FP64 pipe solves

__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }

// Exponent of a row from the upper word of its largest entry; 0 for a zero row.
__device__ __forceinline__ int row_exponent(unsigned hi) { return hi ? slice_exponent(hi) : 0; }

// T(a, c) = R(a, c0 + c), transposed; the rows' largest entries (upper words) into rho from row a_rho on.
__global__ void k_ts_gather(const double* __restrict__ R, int64_t ldr, int k, int ncols, double* __restrict__ T,
                            int a_rho, unsigned* __restrict__ rho) {
  __shared__ double tile[32][33];
  const int c0 = blockIdx.x * 32, a0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int q = 0; q < 32; q += 8) {
    const int a = a0 + ty + q, c = c0 + tx;
    tile[ty + q][tx] = (a < k && c < ncols) ? R[(int64_t)a * ldr + c] : 0.0;
  }
  __syncthreads();
  const int a = a0 + tx;
  if (a >= k) return;
  unsigned mx = 0u;
  for (int q = 0; q < 32; q += 8) {
    const int c = c0 + ty + q;
    const double v = tile[tx][ty + q];
    mx = max(mx, abs_hi(v));
    if (c < ncols) T[a + (int64_t)c * k] = v;
  }
  if (a >= a_rho) atomicMax(rho + a, mx);
}

// Inverses of the diagonal blocks, row major (ld ldi): CTA (g, J) finds columns 8g ..
// 8g + 7 of block J by back substitution, thread = row, the columns still to come updated
// as soon as an entry is known.
__global__ void __launch_bounds__(TS_OB)
k_ts_inv(const double* __restrict__ R, int64_t ldr, int k, double* __restrict__ inv, int ldi) {
  __shared__ double xs[2][8];
  const int ob = blockDim.x, a = threadIdx.x, j0 = blockIdx.y * ob, len = min(ob, k - j0);
  const int cb = blockIdx.x * 8;
  const bool row = a < len;
  if (cb >= len) {   // padding of the last block's K
    if (row)
      for (int q = 0; q < 8; ++q) inv[(int64_t)(j0 + a) * ldi + cb + q] = 0.0;
    return;
  }
  const double* Ra = R + (int64_t)(j0 + a) * ldr + j0;
  const double rinv = row ? 1.0 / Ra[a] : 0.0;
  double x[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) x[q] = a == cb + q ? 1.0 : 0.0;
  const int w0 = a & ~31;
  double r[8];
  for (int jt = cb; jt >= 0; jt -= 8) {      // columns jt .. jt + 7 of R, from the last
    if (w0 < jt + 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) r[u] = (row && jt + u < len && a < jt + u) ? Ra[jt + u] : 0.0;
    }
#pragma unroll
    for (int u = 7; u >= 0; --u) {
      const int j = jt + u;
      if (a == j) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          x[q] = x[q] * rinv;
          xs[u & 1][q] = x[q];
        }
      }
      __syncthreads();
      if (w0 < j) {
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = fma(-r[u], xs[u & 1][q], x[q]);
      }
    }
  }
  if (row) {
#pragma unroll
    for (int q = 0; q < 8; ++q)
      inv[(int64_t)(j0 + a) * ldi + cb + q] = (cb + q < len && a <= cb + q) ? x[q] : 0.0;
  }
}

// Vectors of up to 256 FP64 values (rows of R11 or of an inverse for M, columns of T for N) whose
// entry u is taken times 2^(sign * row_exponent(scale[u])), as slices of kpad values.
struct TsVec {
  const double* src;
  int64_t ld;
  int count;               // vectors
  int sign;
  int tri;                 // vector c starts at entry c - tri (rows of R11 from its diagonal on)
  bool n_operand;          // rows (64-column tile, half, slice, column within the half), else slice by slice
  int64_t rows;            // M: vectors per slice
  unsigned short* out;
  int* exps;
  double* copy;            // N: the values themselves too (or NULL), ld ldc
  int64_t ldc;
};

// What a launch has to know of the refinement of its block.
struct TsNeed {
  int* flag;               // NULL: no condition
  const int* eI;           // not NULL: find the flag from the inverse's exponents and X's rows
  const unsigned* sig;
};

// One warp per vector, its entries in registers; first the M vectors' CTAs, then the N vectors'.
__global__ void __launch_bounds__(256)
k_ts_slices(TsVec vm, TsVec vn, const unsigned* __restrict__ scale, int len, int kpad, TsNeed need,
            State* __restrict__ st) {
  bool refine = false;
  if (need.eI) {           // every CTA for itself, the first one for the launches to come
    const int t = threadIdx.x;
    const int kappa = t < len && need.sig[t] ? need.eI[t] - slice_exponent(need.sig[t]) : 0;
    refine = __syncthreads_or(kappa > TS_REFINE);
    const bool hard = __syncthreads_or(kappa > TS_HARD);
    if (blockIdx.x == 0 && t == 0) {
      *need.flag = refine;
      if (hard) st->t_hard = 1;
    }
  } else if (need.flag && *need.flag == 0) {
    return;
  }
  const int mctas = (vm.count + 7) / 8;
  const bool m_part = (int)blockIdx.x < mctas;
  const TsVec& v = m_part ? vm : vn;
  const int lane = threadIdx.x & 31;
  const int c = ((int)blockIdx.x - (m_part ? 0 : mctas)) * 8 + (threadIdx.x >> 5);
  if (c >= v.count) return;
  const double* src = v.src + (int64_t)c * v.ld;
  constexpr int NONE = -8192;
  double x[8];
  int f[8];
  int mx = NONE;
  bool bad = false;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int a = 8 * lane + u;
    const bool in = a < len && a >= c - v.tri;
    x[u] = in ? src[a] : 0.0;
    f[u] = in ? v.sign * row_exponent(scale[a]) : 0;
    const unsigned hi = abs_hi(x[u]);
    bad = bad || hi >= 0x7FF00000u;
    if (x[u] != 0.0) mx = max(mx, slice_exponent(hi) + f[u]);
  }
  if (v.copy && !refine) {   // coalesced, the values once more from the cache
    double* dst = v.copy + (int64_t)c * v.ldc;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (lane + 32 * u < len) dst[lane + 32 * u] = src[lane + 32 * u];
  }
  if (bad) st->t_hard = 1;
  mx = __reduce_max_sync(0xffffffffu, mx);
  const int e = mx == NONE ? 0 : mx;
  if (lane == 0) v.exps[c] = e;
  if (8 * lane >= kpad) return;
  unsigned short d[8][SL];
#pragma unroll
  for (int u = 0; u < 8; ++u) slice_digits(x[u], max(e - f[u], -1021), d[u]);
  const int64_t step = (v.n_operand ? SL_HALF : v.rows) * (int64_t)kpad;
  const int64_t at = v.n_operand ? (int64_t)(c / SL_HALF) * SL * SL_HALF + c % SL_HALF : (int64_t)c;
  unsigned short* dst = v.out + at * kpad + 8 * lane;
#pragma unroll
  for (int s = 0; s < SL; ++s) store_slice8(dst + s * step, d, s);
}

// M = rows row0 .. row0 + rows of the sliced matrix, N = columns of T, K = a block's rows; row
// p of the product at T(p, :), stored, subtracted from it or added to it.  The rows' largest
// entries into mx(p) for p >= mx0.
enum { TS_SET, TS_SUB, TS_ADD };
struct TsEpi {
  static constexpr bool A_M_MAJOR = false;
  State* st;
  double* T;
  int64_t ldt;
  int row0, rows, ncols, nst, mode;
  const int* exM;
  const int* exX;
  int mx0;
  unsigned* mx;
  const int* flag;         // not NULL: only where it is set
  __device__ int mtiles() const { return (rows + BM - 1) / BM; }
  __device__ int init() const { return flag && *flag == 0 ? 0 : ncols > SL_HALF ? 2 : 1; }
  __device__ bool tile(int t, int& p0, int& brow, int& s0, int& n, int& ax) const {
    const int y = t / mtiles();
    p0 = row0 + (t - y * mtiles()) * BM;
    brow = y * 2 * SL * SL_HALF;
    s0 = ax = 0;
    n = nst;
    return y * 64 < ncols;
  }
  __device__ void part(int t, int p, int a0, const long long (&hi)[SL_HALF], const long long (&lo)[SL_HALF]) const {
    if (p >= row0 + rows) return;
    const int c0 = t / mtiles() * 64 + a0, e = exM[p] - 60;
    double* x = T + p + (int64_t)c0 * ldt;
    unsigned m = 0u;
#pragma unroll
    for (int j0 = 0; j0 < SL_HALF; j0 += 8) {
      double old[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) old[j] = mode != TS_SET && c0 + j0 + j < ncols ? x[(int64_t)(j0 + j) * ldt] : 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c0 + j0 + j < ncols) {
          double v = slice_value(hi[j0 + j], lo[j0 + j], e + exX[c0 + j0 + j]);
          if (mode != TS_SET) v = mode == TS_SUB ? old[j] - v : old[j] + v;
          x[(int64_t)(j0 + j) * ldt] = v;
          m = max(m, abs_hi(v));
        }
    }
    if (p >= mx0) atomicMax(mx + p, m);
  }
  __device__ void timeout() const { atomicExch(&st->status, ST_ERR_TIMEOUT); }
};

}  // namespace
}  // namespace tc

rbrp_status solve_T_fp64(rbrp_handle h, int k, int n, int* launches) {
  const int ncols = n - k;
  cudaStream_t st = h->stream;
  *launches += 2;
  h->form |= RBRP_FORM_T_FP64;
  k_gather_T<<<dim3((ncols + 31) / 32, (k + 31) / 32), dim3(32, 8), 0, st>>>(h->R, n, k, ncols, h->T);
  rbrp_status s = cuda_check(h, cudaFuncSetAttribute(k_trsm_T, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)sizeof(TrsmSmem)), "cudaFuncSetAttribute(k_trsm_T)");
  if (s != RBRP_OK) return s;
  k_trsm_T<<<(ncols + 31) / 32, 256, sizeof(TrsmSmem), st>>>(h->R, n, k, ncols, h->T);
  return cuda_check(h, cudaGetLastError(), "T solve launch");
}

template <int NR>
static rbrp_status solve_T_small(rbrp_handle h, int k, int n, int* launches) {
  const size_t smem = ((size_t)(k + 8) * (32 * NR + 1) + k) * sizeof(double);
  const rbrp_status s =
      cuda_check(h, cudaFuncSetAttribute(k_trsm_small<NR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(((32 * NR + 8) * (32 * NR + 1) + 32 * NR) * sizeof(double))),
                 "cudaFuncSetAttribute(k_trsm_small)");
  if (s != RBRP_OK) return s;
  *launches += 1;
  h->form |= RBRP_FORM_T_FP64;
  k_trsm_small<NR><<<(n - k + 7) / 8, 256, smem, h->stream>>>(h->R, n, k, n - k, h->T);
  return cuda_check(h, cudaGetLastError(), "T solve launch");
}

rbrp_status solve_T(rbrp_handle h, int k, int n, int* launches) {
  *launches = 0;
  const size_t bytes = (size_t)k * (size_t)(n - k) * sizeof(double);
  if (bytes > h->T_bytes) {
    if (h->T) cudaFree(h->T);
    h->T = nullptr;
    h->T_bytes = 0;
    rbrp_status s = device_alloc(h, (void**)&h->T, bytes, "cudaMalloc(T)");
    if (s != RBRP_OK) return s;
    h->T_bytes = bytes;
  }
  if (h->tsolve_fp64) return solve_T_fp64(h, k, n, launches);
  const int ncols = n - k;
  // where the FP64 pipe is the shorter way (us, substitution and slice products): k = 16, 500 columns 8 and
  // 67, 64, 500 columns 17 and 100, 20,000 140 and 192, 128, 2000 71 and 155, 5000 162 and 167, 10,000 285
  // and 202, 100, 10,000 186 and 177
  if (k <= TS_SMALL && (double)ncols * k * k <= 9e7)
    return k <= 32   ? solve_T_small<1>(h, k, n, launches)
           : k <= 64 ? solve_T_small<2>(h, k, n, launches)
           : k <= 96 ? solve_T_small<3>(h, k, n, launches)
                     : solve_T_small<4>(h, k, n, launches);
  cudaStream_t st = h->stream;
  rbrp_status s;
  using namespace tc;
  // blocks of 256 rows, but two or three of 128 where those shorten the chain of steps in the
  // inverses and the columns are too few to hide it (ms with 128 and with 256): k = 208, 4747 columns
  // 0.25 and 0.24, 256 0.25 and 0.29, 384, 3000 columns 0.32 and 0.35, 385 0.39 and 0.36, 1000, 15,000
  // columns 1.69 and 1.30; 60,000 columns, 256 0.88 and 0.85, 384 1.37 and 1.26
  const int ob = k > 208 && k <= 384 && ncols <= 32768 ? TS_OB / 2 : TS_OB;
  const int nblk = (k + ob - 1) / ob;
  const size_t ldi = std::min((size_t)ob, ((size_t)k + 63) / 64 * 64);
  const size_t chunk = std::min(ncols, TS_CHUNK), cpad = (chunk + 63) / 64 * 64;
  struct Item {
    void** ptr;
    size_t bytes;
  };
  unsigned *rho, *rho2, *sig;   // largest entries of the rows of B, of a block's residual, of X
  int *flag, *eR, *eI, *eX;
  unsigned short *sR, *sI, *sX;
  double *inv, *X;
  Item items[] = {
      {(void**)&rho, (size_t)k * 4},
      {(void**)&rho2, (size_t)k * 4},
      {(void**)&sig, (size_t)k * 4},
      {(void**)&flag, 4},
      {(void**)&eR, (size_t)k * 4},
      {(void**)&eI, ldi * 4},
      {(void**)&eX, cpad * 4},
      {(void**)&sR, (size_t)SL * k * ldi * 2},
      {(void**)&inv, (size_t)k * ldi * 8},
      {(void**)&sI, (size_t)SL * ldi * ldi * 2},
      {(void**)&sX, (size_t)SL * cpad * ldi * 2},
      {(void**)&X, cpad * ldi * 8},
  };
  size_t need = 0;
  for (auto& it : items) need += (it.bytes + 255) & ~(size_t)255;
  if (need > h->ts_bytes) {
    if (h->ts_ws) cudaFree(h->ts_ws);
    h->ts_ws = nullptr;
    h->ts_bytes = 0;
    if (device_alloc(h, &h->ts_ws, need, "cudaMalloc(T solve operands)") != RBRP_OK) {
      h->ts_ws = nullptr;   // no room for them: the substitution needs none
      return solve_T_fp64(h, k, n, launches);
    }
    h->ts_bytes = need;
  }
  char* base = static_cast<char*>(h->ts_ws);
  for (auto& it : items) {
    *it.ptr = base;
    base += (it.bytes + 255) & ~(size_t)255;
  }
  CUtensorMap tmR, tmI, tmX;
  s = make_tmap_bf16(h, &tmI, sI, ldi, (uint64_t)SL * ldi, BM);
  if (s == RBRP_OK) s = make_tmap_bf16(h, &tmR, sR, ldi, (uint64_t)SL * k, BM);
  if (s == RBRP_OK) s = make_tmap_bf16(h, &tmX, sX, ldi, (uint64_t)SL * cpad, SL * SL_HALF);
  if (s == RBRP_OK)
    s = cuda_check(h, cudaFuncSetAttribute(k_gemm_slices<TsEpi>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)SL_SMEM), "cudaFuncSetAttribute(k_gemm_slices)");
  if (s != RBRP_OK) return s;
  const long long budget = h->wait_budget > 0 ? h->wait_budget : kWaitBudgetDefault;
  const int kpad = (int)ldi;
  k_ts_inv<<<dim3(kpad / 8, nblk), ob, 0, st>>>(h->R, n, k, inv, kpad);
  *launches += 1;
  for (int c0 = 0; c0 < ncols; c0 += TS_CHUNK) {
    const int nc = std::min(TS_CHUNK, ncols - c0), ntile = (nc + 63) / 64;
    double* T = h->T + (size_t)c0 * k;
    const int jlast = (nblk - 1) * ob;
    // rho, rho2 and sig lie together
    cudaMemsetAsync(rho, 0, (size_t)((char*)flag - (char*)rho), st);
    k_ts_gather<<<dim3((nc + 31) / 32, (k + 31) / 32), dim3(32, 8), 0, st>>>(h->R + k + c0, n, k, nc, T, jlast, rho);
    *launches += 1;
    for (int J = nblk - 1; J >= 0; --J) {
      const int j0 = J * ob, len = std::min(ob, k - j0), nst = (len + SL_BK - 1) / SL_BK;
      auto slices = [&](const TsVec& vm, const TsVec& vn, const unsigned* scale, const TsNeed& nd) {
        k_ts_slices<<<(vm.count + 7) / 8 + (vn.count + 7) / 8, 256, 0, st>>>(vm, vn, scale + j0, len, kpad, nd, h->st);
      };
      auto gemm = [&](const CUtensorMap& tm, int64_t a_rows, const TsEpi& e) {
        k_gemm_slices<<<std::min(h->sms, (e.rows + BM - 1) / BM * ntile), SL_THREADS, SL_SMEM, st>>>(tm, tmX, a_rows,
                                                                                                    budget, e);
      };
      const TsVec vI{inv + (size_t)j0 * ldi, (int64_t)ldi, len, 1, len, false, (int64_t)ldi, sI, eI, nullptr, 0};
      const TsVec vB{T + j0, k, nc, -1, nc, true, 0, sX, eX, nullptr, 0};
      const TsVec vR{h->R + j0, n, j0 + len, 1, j0, false, k, sR, eR, nullptr, 0};
      const TsVec vX{X, (int64_t)ldi, nc, -1, nc, true, 0, sX, eX, T + j0, k};
      TsVec none = vI;
      none.count = 0;
      // X = inv B_J, and from it the flag and the operands of the update; T takes X if it stands
      slices(vI, vB, rho, TsNeed{nullptr, nullptr, nullptr});
      gemm(tmI, (int64_t)ldi, TsEpi{h->st, X, (int64_t)ldi, 0, len, nc, nst, TS_SET, eI, eX, 0, sig + j0, nullptr});
      slices(vR, vX, sig, TsNeed{flag, eI, sig + j0});
      // the refinement: launches that return at once where the flag is not set
      gemm(tmR, k, TsEpi{h->st, T, k, j0, len, nc, nst, TS_SUB, eR, eX, 0, rho2, flag});
      slices(vI, vB, rho2, TsNeed{flag, nullptr, nullptr});
      gemm(tmI, (int64_t)ldi, TsEpi{h->st, X, (int64_t)ldi, 0, len, nc, nst, TS_ADD, eI, eX, len, nullptr, flag});
      slices(none, vX, sig, TsNeed{flag, nullptr, nullptr});
      if (J > 0)
        gemm(tmR, k, TsEpi{h->st, T, k, 0, j0, nc, nst, TS_SUB, eR, eX, j0 - ob, rho, nullptr});
      *launches += J > 0 ? 8 : 7;
    }
  }
  return cuda_check(h, cudaGetLastError(), "T solve launch");
}

}  // namespace rbrp
