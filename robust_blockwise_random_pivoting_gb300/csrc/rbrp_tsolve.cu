// rbrp_tsolve.cu - the interpolation matrix T = R11^{-1} R12 (a10).
#include <algorithm>

#include <cuda.h>

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

// ===========================================================================
// The same solve as slice products (rbrp_slices.cuh): blocks of 256 (or 128) rows from the bottom up,
// X_J = inv(R11(J, J)) B_J and then B(0:j0) -= R11(0:j0, J) X_J, both on the tensor cores.
// Rows are scaled by the power of two of their diagonal entry (which leaves T alone), so the
// entries of the scaled R11, of its blocks' inverses and of T are of one size and a slice
// loses nothing: 55 bits below each row's largest entry, where the double-float solve this
// replaces carried 48 throughout.
//
// What bounds it: a 128 x 64 tile over 256 values of k is 18,000 clocks of MMAs, which its
// epilogue (one FP64 subtraction per entry) runs beside; the double-float solve needed 12 FP32 operations per
// product and a warp per column in the diagonal blocks (k = 2000, 14,384 columns: 15.9 ms,
// now 2.7; k = 1000, 64,536 columns: 19.5, now 3.4).
// ===========================================================================
namespace tc {
namespace {

constexpr int TS_OB = 256;            // rows per block at the most
constexpr int TS_CHUNK = 65536;       // columns of T per pass: bounds the sliced copy to 235 MB

__device__ __forceinline__ int diag_exponent(const double* R, int64_t ldr, int a) {
  return slice_exponent((unsigned)__double2hiint(R[(int64_t)a * ldr + a]) & 0x7FFFFFFFu);
}

// T(a, c) = R(a, k + c) 2^(-e_a), transposed; e_a into ed.
__global__ void k_ts_gather(const double* __restrict__ R, int64_t ldr, int k, int ncols, double* __restrict__ T,
                            int* __restrict__ ed) {
  __shared__ double tile[32][33];
  const int c0 = blockIdx.x * 32, a0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int q = 0; q < 32; q += 8) {
    const int a = a0 + ty + q, c = c0 + tx;
    tile[ty + q][tx] = (a < k && c < ncols) ? R[(int64_t)a * ldr + k + c] : 0.0;
  }
  __syncthreads();
  const int a = a0 + tx;
  if (a >= k) return;
  const int e = diag_exponent(R, ldr, a);
  if (blockIdx.x == 0 && ty == 0) ed[a] = e;
  // 2^(-e) as an FP64 value (a subnormal one only beside a diagonal of 2^1022 and more)
  const double sc = ldexp(1.0, -e);
  for (int q = 0; q < 32; q += 8) {
    const int c = c0 + ty + q;
    if (c < ncols) T[a + (int64_t)c * k] = tile[tx][ty + q] * sc;
  }
}

// Slices of R11's rows right of their own block of ob rows (one warp per row), K-major; the
// exponents are those of the scaled rows.
__global__ void __launch_bounds__(256)
k_ts_slice_r(const double* __restrict__ R, int64_t ldr, int k, int ob, int64_t ldk, unsigned short* __restrict__ out,
             int* __restrict__ exps) {
  const int lane = threadIdx.x & 31;
  const int a = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int jb = (a / ob + 1) * ob;
  if (a >= k || jb >= k) return;
  const double* row = R + (int64_t)a * ldr;
  unsigned mx = 0u;
  for (int j = jb + lane; j < k; j += 32) mx = max(mx, (unsigned)__double2hiint(row[j]) & 0x7FFFFFFFu);
  mx = __reduce_max_sync(0xffffffffu, mx);
  const int e = slice_exponent(mx);
  if (lane == 0) exps[a] = e - diag_exponent(R, ldr, a);
  for (int j0 = jb + 8 * lane; j0 < ldk; j0 += 256) {
    unsigned short d[8][SL];
#pragma unroll
    for (int u = 0; u < 8; ++u) slice_digits(j0 + u < k ? row[j0 + u] : 0.0, e, d[u]);
#pragma unroll
    for (int s = 0; s < SL; ++s) store_slice8(out + ((int64_t)s * k + a) * ldk + j0, d, s);
  }
}

// Inverses of the scaled diagonal blocks, row major (ld ldi): CTA (g, J) finds columns 8g ..
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
  const double sc = row ? ldexp(1.0, -diag_exponent(R, ldr, j0 + a)) : 0.0;
  const double rinv = row ? 1.0 / (Ra[a] * sc) : 0.0;
  double x[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) x[q] = a == cb + q ? 1.0 : 0.0;
  const int w0 = a & ~31;
  double r[8];
  for (int jt = cb; jt >= 0; jt -= 8) {      // columns jt .. jt + 7 of R, from the last
    if (w0 < jt + 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) r[u] = (row && jt + u < len && a < jt + u) ? Ra[jt + u] * sc : 0.0;
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

// Slices of rows j0 .. j0 + len of T's columns (one warp per column, its entries in registers)
// as the N operand: rows (64-column tile, half, slice, column within the half), ldk values.
__global__ void __launch_bounds__(256)
k_ts_slice_x(const double* __restrict__ T, int64_t ldt, int j0, int len, int ncols, int ldk,
             unsigned short* __restrict__ out, int* __restrict__ exps) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (c >= ncols) return;
  const double* col = T + (int64_t)c * ldt + j0;
  double x[8];
  unsigned mx = 0u;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    x[u] = 8 * lane + u < len ? col[8 * lane + u] : 0.0;
    mx = max(mx, (unsigned)__double2hiint(x[u]) & 0x7FFFFFFFu);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  const int e = slice_exponent(mx);
  if (lane == 0) exps[c] = e;
  if (8 * lane >= ldk) return;
  unsigned short d[8][SL];
#pragma unroll
  for (int u = 0; u < 8; ++u) slice_digits(x[u], e, d[u]);
  unsigned short* dst = out + ((int64_t)(c / SL_HALF) * SL * SL_HALF + c % SL_HALF) * ldk + 8 * lane;
#pragma unroll
  for (int s = 0; s < SL; ++s) store_slice8(dst + (int64_t)s * SL_HALF * ldk, d, s);
}

// M = rows row0 .. row0 + rows of the sliced matrix (its K starts at column ax), N = columns
// of T; stores the product in T, or subtracts it (sub).
struct TsEpi {
  static constexpr bool A_M_MAJOR = false;
  State* st;
  double* T;
  int64_t ldt;
  int row0, rows, ncols, nst, ax, sub;
  const int* exM;
  const int* exX;
  __device__ int mtiles() const { return (rows + BM - 1) / BM; }
  __device__ int init() const { return ncols > SL_HALF ? 2 : 1; }
  __device__ bool tile(int t, int& p0, int& brow, int& s0, int& n, int& a_x) const {
    const int y = t / mtiles();
    p0 = row0 + (t - y * mtiles()) * BM;
    brow = y * 2 * SL * SL_HALF;
    s0 = 0;
    n = nst;
    a_x = ax;
    return y * 64 < ncols;
  }
  __device__ void part(int t, int p, int a0, const long long (&hi)[SL_HALF], const long long (&lo)[SL_HALF]) const {
    if (p >= row0 + rows) return;
    const int c0 = t / mtiles() * 64 + a0, e = exM[p] - 60;
    double* x = T + p + (int64_t)c0 * ldt;
#pragma unroll
    for (int j0 = 0; j0 < SL_HALF; j0 += 8) {
      double old[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) old[j] = sub && c0 + j0 + j < ncols ? x[(int64_t)(j0 + j) * ldt] : 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c0 + j0 + j < ncols) {
          const double v = slice_value(hi[j0 + j], lo[j0 + j], e + exX[c0 + j0 + j]);
          x[(int64_t)(j0 + j) * ldt] = sub ? old[j] - v : v;
        }
    }
  }
  __device__ void timeout() const { atomicExch(&st->status, ST_ERR_TIMEOUT); }
};

}  // namespace
}  // namespace tc

rbrp_status solve_T(rbrp_handle h, int k, int n) {
  const size_t bytes = (size_t)k * (size_t)(n - k) * sizeof(double);
  if (bytes > h->T_bytes) {
    if (h->T) cudaFree(h->T);
    h->T = nullptr;
    h->T_bytes = 0;
    rbrp_status s = device_alloc(h, (void**)&h->T, bytes, "cudaMalloc(T)");
    if (s != RBRP_OK) return s;
    h->T_bytes = bytes;
  }
  const int ncols = n - k;
  cudaStream_t st = h->stream;
  rbrp_status s;
  if (h->tsolve_fp64) {
    dim3 g1((ncols + 31) / 32, (k + 31) / 32), b1(32, 8);
    k_gather_T<<<g1, b1, 0, st>>>(h->R, n, k, ncols, h->T);
    s = cuda_check(h, cudaFuncSetAttribute(k_trsm_T, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sizeof(TrsmSmem)), "cudaFuncSetAttribute(k_trsm_T)");
    if (s != RBRP_OK) return s;
    k_trsm_T<<<(ncols + 31) / 32, 256, sizeof(TrsmSmem), st>>>(h->R, n, k, ncols, h->T);
    return cuda_check(h, cudaGetLastError(), "T solve launch");
  }
  using namespace tc;
  // the chain of ob steps of the inverses against fewer, larger products: k = 270, 1730 columns:
  // 0.26 ms with blocks of 128, 0.34 with 256; 640, 7552: 0.61 and 0.63; 900, 300: 0.54 and 0.50;
  // 2000, 14384: 5.7 and 3.9 (before the grid was persistent)
  const int ob = k <= 640 ? TS_OB / 2 : TS_OB;
  const int nblk = (k + ob - 1) / ob;
  const size_t ldk = ((size_t)k + 63) / 64 * 64, ldi = std::min((size_t)ob, ldk);
  const size_t chunk = std::min(ncols, TS_CHUNK), cpad = (chunk + 63) / 64 * 64;
  struct Item {
    void** ptr;
    size_t bytes;
  };
  int *ed, *eR, *eI, *eX;
  unsigned short *sR, *sI, *sX;
  double* inv;
  Item items[] = {
      {(void**)&ed, (size_t)k * 4},
      {(void**)&eR, (size_t)k * 4},
      {(void**)&eI, (size_t)k * 4},
      {(void**)&eX, cpad * 4},
      {(void**)&sR, nblk > 1 ? (size_t)SL * k * ldk * 2 : 0},
      {(void**)&inv, (size_t)k * ldi * 8},
      {(void**)&sI, (size_t)SL * k * ldi * 2},
      {(void**)&sX, (size_t)SL * cpad * ldi * 2},
  };
  size_t need = 0;
  for (auto& it : items) need += (it.bytes + 255) & ~(size_t)255;
  if (need > h->ts_bytes) {
    if (h->ts_ws) cudaFree(h->ts_ws);
    h->ts_ws = nullptr;
    h->ts_bytes = 0;
    s = device_alloc(h, &h->ts_ws, need, "cudaMalloc(T solve operands)");
    if (s != RBRP_OK) return s;
    h->ts_bytes = need;
  }
  char* base = static_cast<char*>(h->ts_ws);
  for (auto& it : items) {
    *it.ptr = base;
    base += (it.bytes + 255) & ~(size_t)255;
  }
  CUtensorMap tmR, tmI, tmX;
  s = make_tmap_bf16(h, &tmI, sI, ldi, (uint64_t)SL * k, BM);
  if (s == RBRP_OK && nblk > 1) s = make_tmap_bf16(h, &tmR, sR, ldk, (uint64_t)SL * k, BM);
  if (s == RBRP_OK) s = make_tmap_bf16(h, &tmX, sX, ldi, (uint64_t)SL * cpad, SL * SL_HALF);
  if (s == RBRP_OK)
    s = cuda_check(h, cudaFuncSetAttribute(k_gemm_slices<TsEpi>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)SL_SMEM), "cudaFuncSetAttribute(k_gemm_slices)");
  if (s != RBRP_OK) return s;
  const long long budget = h->wait_budget > 0 ? h->wait_budget : kWaitBudgetDefault;
  k_ts_gather<<<dim3((ncols + 31) / 32, (k + 31) / 32), dim3(32, 8), 0, st>>>(h->R, n, k, ncols, h->T, ed);
  if (nblk > 1) k_ts_slice_r<<<(k + 7) / 8, 256, 0, st>>>(h->R, n, k, ob, ldk, sR, eR);
  k_ts_inv<<<dim3((int)ldi / 8, nblk), ob, 0, st>>>(h->R, n, k, inv, (int)ldi);
  k_slice_cols<<<(k + 7) / 8, 256, 0, st>>>(inv, ldi, (int)ldi, k, k, ldi, sI, eI);
  for (int c0 = 0; c0 < ncols; c0 += TS_CHUNK) {
    const int nc = std::min(TS_CHUNK, ncols - c0), ntile = (nc + 63) / 64;
    double* T = h->T + (size_t)c0 * k;
    for (int J = nblk - 1; J >= 0; --J) {
      const int j0 = J * ob, len = std::min(ob, k - j0), nst = (len + SL_BK - 1) / SL_BK;
      k_ts_slice_x<<<(nc + 7) / 8, 256, 0, st>>>(T, k, j0, len, nc, (int)ldi, sX, eX);
      k_gemm_slices<<<std::min(h->sms, (len + BM - 1) / BM * ntile), SL_THREADS, SL_SMEM, st>>>(
          tmI, tmX, (int64_t)k, budget, TsEpi{h->st, T, k, j0, len, nc, nst, 0, 0, eI, eX});
      if (J > 0) {
        k_ts_slice_x<<<(nc + 7) / 8, 256, 0, st>>>(T, k, j0, len, nc, (int)ldi, sX, eX);
        k_gemm_slices<<<std::min(h->sms, j0 / BM * ntile), SL_THREADS, SL_SMEM, st>>>(
            tmR, tmX, (int64_t)k, budget, TsEpi{h->st, T, k, 0, j0, nc, nst, j0, 1, eR, eX});
      }
    }
  }
  return cuda_check(h, cudaGetLastError(), "T solve launch");
}

}  // namespace rbrp
