// rbrp_slices.cuh - FP64-accurate products on the tcgen05 tensor cores (sm_103a), by
// exact integer slices (the splitting of Ozaki, Ogita, Oishi and Rump, 2012).
//
// A row x of an operand (K values, |x| < 2^e) is held as X = rint(x 2^(54 - e)) in
// balanced base-256 digits, X = sum_s d_s 256^(6 - s) with |d_0| <= 64 and
// -128 <= d_s <= 127: seven slices of exact BF16 integers.  Then
//   sum_k x(k) y(k) = 2^(ex + ey - 60) sum_c S_c 256^(6 - c),   S_c = sum_{i + j = c} sum_k d_i(k) e_j(k),
// and every S_c is a sum of integer products that FP32 accumulates without rounding as
// long as |S_c| <= 2^24.  Classes c <= 7 are taken (34 slice products).  Over a chunk of
// 192 values of k, S_0 .. S_5 stay below 2^24 for any data; S_6 and S_7 can pass it only
// by 1.13x, where a rounding of a unit or two is 2^-60 of max|x| max|y|.  After each
// chunk the sums are folded into 64-bit integers, so the result carries no rounding
// that grows with K: what is left is the operands' representation (2^-55 of each row's
// largest entry per value) and the dropped classes (about 2^-62 per value), against
// 2^-53 of every partial sum in an FP64 FMA chain.  Both are bounds by the operands' columns:
// an entry far below its column's largest has that many digits fewer, and none 2^-55 below, where
// an FMA chain keeps it if nothing larger is added to it.  With rows graded over 2^60 the error of
// T (400 x 300, rank 60) is a quarter to a half of the FP64 pipe's.
//
// Why: GB300 retires about 1.6 FP64 FMAs per clock and SM, the BF16 tensor pipe some 3,100
// (cuBLAS's rate): 58 times as many over 34 slice products.  A block of 64 columns of an
// 8192 x 8192 matrix takes 0.23 ms for 8.8 on the FP64 pipe.
#pragma once
#include "rbrp_tc.cuh"

namespace rbrp {
namespace tc {
namespace {

constexpr int SL = 7;                        // slices per operand
constexpr int SL_BK = 64;                    // values of k per stage: one 128-byte swizzle row of BF16
constexpr int SL_CHUNK = 3;                  // stages between drains (192 values of k)
constexpr int SL_HALF = 32;                  // N per accumulator set
constexpr int SL_CLASSES = 8;
constexpr int SL_A_BYTES = BM * SL_BK * 2;              // one slice of the M operand: 16 KB
constexpr int SL_B_BYTES = SL * SL_HALF * SL_BK * 2;    // seven slices of one half of the N operand: 28 KB
constexpr int SL_DRAIN = 256;                           // 8 drain warps
constexpr int SL_THREADS = 64 + SL_DRAIN;

// Balanced base-256 digits of x 2^(-e) for |x| < 2^e, as BF16 bit patterns.
// The integer comes from the bits of x: the FP64 pipe is 1/64 of the integer pipe's rate.
__device__ __forceinline__ void slice_digits(double x, int e, unsigned short (&d)[SL]) {
  const long long bits = __double_as_longlong(x);
  const int ex = (int)((bits >> 52) & 0x7FF);
  long long mant = bits & 0xFFFFFFFFFFFFFll;
  if (ex) mant |= 1ll << 52;
  // x = mant 2^(max(ex, 1) - 1075); X = mant 2^sh, sh <= 1 because |x| < 2^e
  const int sh = (ex ? ex : 1) - 1075 + 54 - e;
  long long X;
  if (sh >= 0) {
    X = mant << sh;
  } else {
    const int r = -sh;
    X = r > 60 ? 0 : (mant + (1ll << (r - 1))) >> r;   // nearest, ties away from zero
  }
  if (bits < 0) X = -X;
#pragma unroll
  for (int s = SL - 1; s >= 0; --s) {
    const int v = s ? (int)(signed char)(X & 0xFF) : (int)X;
    X = (X - v) >> 8;
    // float(v) by the 1.5 * 2^23 bias; at most 8 significant bits, so its upper half is the BF16
    const float f = __int_as_float(0x4B400000 + v) - 12582912.0f;
    d[s] = (unsigned short)(__float_as_uint(f) >> 16);
  }
}

// Exponent e with |x| < 2^e from the largest |x| of a row, given as the upper 32 bits
// of its FP64 pattern; zero and subnormal rows take the smallest normal one.
__device__ __forceinline__ int slice_exponent(unsigned hi) {
  const int ex = (int)((hi >> 20) & 0x7FF);
  return (ex ? ex : 1) - 1022;
}

// Slice s of eight consecutive values, 16 bytes.
__device__ __forceinline__ void store_slice8(unsigned short* dst, const unsigned short (&d)[8][SL], int s) {
  uint4 v;
  v.x = d[0][s] | ((unsigned)d[1][s] << 16);
  v.y = d[2][s] | ((unsigned)d[3][s] << 16);
  v.z = d[4][s] | ((unsigned)d[5][s] << 16);
  v.w = d[6][s] | ((unsigned)d[7][s] << 16);
  *reinterpret_cast<uint4*>(dst) = v;
}

// Slices of the columns of an FP64 matrix: column c into rows s * srows + c of out
// (ldk BF16 values each, zero past m), its exponent into ex[c].  One warp per column:
// a pass for the largest entry, then a second one (L2) that writes 16 bytes per lane
// and slice.  HBM bound: reads 8 and writes 14 bytes per entry (8192 x 8192: 0.36 ms,
// 4.1 TB/s of those 22 bytes).
__global__ void __launch_bounds__(256)
k_slice_cols(const double* __restrict__ A, int64_t lda, int m, int n, int64_t srows, int64_t ldk,
             unsigned short* __restrict__ out, int* __restrict__ exps) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (c >= n) return;
  const double* col = A + (int64_t)c * lda;
  unsigned mx = 0u;
  for (int r = lane; r < m; r += 32) mx = max(mx, (unsigned)__double2hiint(col[r]) & 0x7FFFFFFFu);
  mx = __reduce_max_sync(0xffffffffu, mx);
  const int e = slice_exponent(mx);
  if (lane == 0) exps[c] = e;
  for (int r0 = 8 * lane; r0 < ldk; r0 += 256) {
    unsigned short d[8][SL];
#pragma unroll
    for (int u = 0; u < 8; ++u) slice_digits(r0 + u < m ? col[r0 + u] : 0.0, e, d[u]);
#pragma unroll
    for (int s = 0; s < SL; ++s) store_slice8(out + ((int64_t)s * srows + c) * ldk + r0, d, s);
  }
}

// Slices of the block's basis columns Q(:, i .. i + kept) as the N operand: rows
// (half, slice, column within the half), zero beyond the kept columns (up to 32, or 64
// where more than 32 are kept).  One CTA per column.  Also into row i + a of the basis
// history (hist_rows per slice; its rows up to the next multiple of 64 are zeroed: the
// Gram-Schmidt products read whole stages).  A column that is not finite has no digits: the run
// ends with the status that its products would have brought about (remaining positions: n).
__global__ void __launch_bounds__(256)
k_slice_q(const double* __restrict__ Q, int64_t ldq, int m, int n, State* __restrict__ st, int64_t ldk,
          unsigned short* __restrict__ out, int* __restrict__ exps, unsigned short* __restrict__ hist, int hist_rows,
          int* __restrict__ hist_exps) {
  __shared__ unsigned s_mx[8];
  const int tid = threadIdx.x, a = blockIdx.x, i = st->i, kept = st->bs;
  const bool oper = a < (kept > SL_HALF ? 2 * SL_HALF : SL_HALF);
  const bool keep = i + a < hist_rows && i + a < (i + kept + 63) / 64 * 64;
  if (kept == 0 || (!oper && !keep)) return;
  unsigned short* hdst = hist + (int64_t)(i + a) * ldk;
  unsigned short* dst = out + ((int64_t)(a / SL_HALF) * SL * SL_HALF + a % SL_HALF) * ldk;
  const double* col = Q + (int64_t)(i + (a < kept ? a : 0)) * ldq;
  unsigned mx = 0u;
  if (a < kept)
    for (int r = tid; r < m; r += 256) mx = max(mx, (unsigned)__double2hiint(col[r]) & 0x7FFFFFFFu);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((tid & 31) == 0) s_mx[tid >> 5] = mx;
  __syncthreads();
  for (int w = 0; w < 8; ++w) mx = max(mx, s_mx[w]);
  const int e = slice_exponent(mx);
  if (tid == 0 && mx >= 0x7FF00000u && i + kept < n) atomicCAS(&st->status, 0, ST_ERR_NUMERIC);
  if (tid == 0 && oper) exps[a] = e;
  if (tid == 0 && keep) hist_exps[i + a] = e;
  for (int r0 = 2 * tid; r0 < ldk; r0 += 512) {
    unsigned short d0[SL], d1[SL];
    slice_digits(a < kept && r0 < m ? col[r0] : 0.0, e, d0);
    slice_digits(a < kept && r0 + 1 < m ? col[r0 + 1] : 0.0, e, d1);
#pragma unroll
    for (int s = 0; s < SL; ++s) {
      const unsigned v = d0[s] | ((unsigned)d1[s] << 16);
      if (oper) *reinterpret_cast<unsigned*>(dst + (int64_t)s * SL_HALF * ldk + r0) = v;
      if (keep) *reinterpret_cast<unsigned*>(hdst + (int64_t)s * hist_rows * ldk + r0) = v;
    }
  }
}

// Slices of the sampled columns' coefficients R(0:i, js[c]) as the N operand of Q C, K = the
// basis index, each scaled by its basis column's exponent (2^ex of the history's rows).  One CTA
// per column, zero beyond the sampled ones.
__global__ void __launch_bounds__(256)
k_slice_coef(const double* __restrict__ R, int64_t ldr, const int* __restrict__ js, const State* __restrict__ st,
             const int* __restrict__ hist_exps, int64_t ldk, unsigned short* __restrict__ out, int* __restrict__ exps) {
  __shared__ int s_mx[8];
  const int tid = threadIdx.x, c = blockIdx.x, i = st->i;
  const bool in = c < st->bs_sampled;
  unsigned short* dst = out + ((int64_t)(c / SL_HALF) * SL * SL_HALF + c % SL_HALF) * ldk;
  const double* col = R + (in ? js[c] : 0);
  int mx = -4096;
  for (int a = tid; a < i && in; a += 256)
    mx = max(mx, slice_exponent((unsigned)__double2hiint(col[(int64_t)a * ldr]) & 0x7FFFFFFFu) + hist_exps[a]);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((tid & 31) == 0) s_mx[tid >> 5] = mx;
  __syncthreads();
  for (int w = 0; w < 8; ++w) mx = max(mx, s_mx[w]);
  if (tid == 0) exps[c] = mx;
  const int kend = (i + SL_BK - 1) / SL_BK * SL_BK;
  for (int a = tid; a < kend; a += 256) {
    unsigned short d[SL];
    const bool ok = in && a < i;
    slice_digits(ok ? col[(int64_t)a * ldr] : 0.0, ok ? mx - hist_exps[a] : 0, d);
#pragma unroll
    for (int s = 0; s < SL; ++s) dst[(int64_t)s * SL_HALF * ldk + a] = d[s];
  }
}

// Block swap of the sliced columns (they stay in position order, as perm):
// columns K2 take the slices and exponents of K1.
__global__ void __launch_bounds__(256)
k_swap_slices(unsigned short* __restrict__ out, int64_t srows, int64_t ldk, int* __restrict__ exps,
              const State* __restrict__ st, const int* __restrict__ K1g, const int* __restrict__ K2g) {
  const int t = blockIdx.x;
  if (t >= st->nK) return;
  const int a = K1g[t], b = K2g[t];
  const uint4* src = reinterpret_cast<const uint4*>(out + ((int64_t)blockIdx.y * srows + a) * ldk);
  uint4* dst = reinterpret_cast<uint4*>(out + ((int64_t)blockIdx.y * srows + b) * ldk);
  for (int64_t x = threadIdx.x; x < ldk / 8; x += 256) dst[x] = src[x];
  if (blockIdx.y == 0 && threadIdx.x == 0) exps[b] = exps[a];
}

// A tile stored [k][128-byte row of 64 values of M] (two such blocks, 64 k rows each): the
// descriptor of an M-major operand, 128-byte swizzle.  Leading offset: the next 64 values of
// M; stride offset: the next 8 values of k.
__device__ __forceinline__ uint64_t sw128_desc_m(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((SL_BK * 128) >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

template <bool A_M_MAJOR>
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, int n, uint32_t accumulate) {
  // D = F32 (bits 4-5 = 1), A = B = BF16 (bits 7-9, 10-12 = 1), A K-major or M-major (bit 15),
  // B K-major, N >> 3, M >> 4
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (A_M_MAJOR ? 1u << 15 : 0u) |
                         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4]) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = __uint_as_float(r[j]);
}

// (hi 2^24 + lo) 2^e rounded to the nearest FP64 value (ties away from zero), on 32-bit
// words: conversions on the FP64 pipe would cost 25,000 clocks per 128 x 64 tile, and 64-bit
// shifts with a normalisation by cases did cost 20,000 (T solve, k = 2000, 14,384 columns:
// 3.9 ms; 2.7 with this and the persistent grid).
__device__ __forceinline__ double slice_value(long long hi, long long lo, int e) {
  hi += lo >> 24;
  // |hi 2^32 + (lo mod 2^24) 2^8| as three words
  unsigned w2 = (unsigned)((unsigned long long)hi >> 32), w1 = (unsigned)hi, w0 = (unsigned)lo << 8;
  const unsigned neg = (unsigned)((int)w2 >> 31);
  w0 = (w0 ^ neg) - neg;
  const unsigned c0 = neg & (w0 == 0u ? 1u : 0u);   // the carry of -x = ~x + 1
  w1 = (w1 ^ neg) + c0;
  const unsigned c1 = c0 & (w1 == 0u ? 1u : 0u);
  w2 = (w2 ^ neg) + c1;
  // leading one into bit 31 of w2
  int p = 95;
  if (w2 == 0u) { w2 = w1; w1 = w0; w0 = 0u; p -= 32; }
  if (w2 == 0u) { w2 = w1; w1 = 0u; p -= 32; }
  const int n = __clz((int)w2);
  w2 = __funnelshift_lc(w1, w2, n);
  w1 = __funnelshift_lc(w0, w1, n);
  // 53 bits of w2 : w1, rounded; a carry out of them raises the exponent by itself
  const unsigned r = (w1 >> 10) & 1u;
  unsigned ml = __funnelshift_r(w1, w2, 11), mh = w2 >> 11;
  ml += r;
  mh += r & (ml == 0u ? 1u : 0u);
  const int be = 1023 + p - n - 8 + e;
  if (w2 == 0u) return 0.0;
  if (be < 1 || be > 2045) return ldexp(__hiloint2double((int)(mh + (1022u << 20) | (neg & 0x80000000u)), (int)ml), be - 1023);
  return __hiloint2double((int)((mh + ((unsigned)(be - 1) << 20)) | (neg & 0x80000000u)), (int)ml);
}

// Shared memory: the seven slices of the stage's M tile, each its own slot of a ring,
// and two stages of the N operand's halves.
struct __align__(1024) SliceSmem {
  uint8_t as[SL][SL_A_BYTES];
  uint8_t bs[2][2][SL_B_BYTES];             // [stage parity][half]
  unsigned long long afull[SL], aempty[SL], bfull[2], bempty[2], accf[2], acce[2], mmadone;
  uint32_t tmem_base;
  int abort;
};
constexpr size_t SL_SMEM = sizeof(SliceSmem) + 1024;
static_assert(SL_SMEM <= 232448, "227 KB of shared memory per CTA");

// Tiles of 128 x 64 (128 x 32 where one half holds every column) of D(p, a), each over the
// stages [s0, s0 + nst) of 64 values of k: a persistent grid, tile t = blockIdx.x, + gridDim.x, ...
//
//   warp 0    TMA: per stage the N operand's halves, then the M operand's slices.
//   warp 1    MMAs.  Slice i of M meets slices 0 .. min(6, 7 - i) of N at once: those sit
//             in consecutive rows, so one MMA of N = 32 x (slices) adds classes i, i + 1, ...
//             in consecutive accumulator columns.  An accumulator set (8 classes x 32
//             columns) holds one half; tensor memory holds two sets, whose chunks are
//             staggered by a stage, and the half that starts a chunk is issued last, so
//             that its drain hides behind the other's MMAs.  With one half, chunks
//             alternate between the sets.
//   warps 2-9 drain a set each (four lane quarters): FP32 integers to int, folded into
//             two 64-bit integers per column (weights 256^3 and 1, in units of class 6);
//             with one half, warps 2-5 drain both sets.  A tile's results leave the
//             registers while the next tile's MMAs run.
//
// What bounds it, 8192 x 8192, 64 columns (230 us a block): the MMAs are 568 clocks per 16 values of k
// and half (N = 32 x 34 classes at half a clock per column, or the shared-memory reads of the
// short ones), 115 us, the 964 MB of slices from HBM 145 us at the copy rate.  Counters: tensor pipe 57%
// active, DRAM 4.2 TB/s, issue slots 16%; neither is full, with one stage of slices (112 KB)
// in flight per SM.  1000 x 1000, 40 columns: 0.034 ms a block against 0.61 on the FP64 pipe.
//
// The M operand is K-major (slices of rows along k), or M-major (Epi::A_M_MAJOR: slices of
// columns along M, k the slice's row).
//
// epi.init(): halves of every tile, 0 for nothing to do; epi.tile(t, ...): the t-th tile,
// false past the last; epi.part(t, p, a0, hi, lo): the thread's 32 columns a0 .. a0 + 31 of
// row p, with D = 2^(ex + ey - 60) (hi 2^24 + lo).
template <typename Epi>
__global__ void __launch_bounds__(SL_THREADS, 1)
k_gemm_slices(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int64_t a_rows,
              long long budget, Epi epi) {
  extern __shared__ uint8_t sl_raw[];
  SliceSmem& sm = *reinterpret_cast<SliceSmem*>((reinterpret_cast<uintptr_t>(sl_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nh = epi.init();
  int p0, brow, s0, nst, ax;   // first M row, first N row, stage range, M's first value of k
  if (nh == 0 || !epi.tile(blockIdx.x, p0, brow, s0, nst, ax)) return;  // uniform over the CTA
  volatile int* abort = &sm.abort;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SL; ++s) {
      mbar_init(&sm.afull[s], 1);
      mbar_init(&sm.aempty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.bfull[b], 1);
      mbar_init(&sm.bempty[b], 1);
      mbar_init(&sm.accf[b], 1);
      mbar_init(&sm.acce[b], SL_DRAIN / 2);
    }
    mbar_init(&sm.mmadone, 1);
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = sm.tmem_base;
  int g = 0;                     // stages so far, over the tiles (ring positions)
  int aissued = 0, bissued = 0;  // producer: slices and N stages whose loads were issued
  bool ok = true;

  // chunk of half h at stage s of a tile: with two halves the second one's chunks start a stage early
  auto chunk_of = [&](int h, int s) { return (s + (nh == 2 ? h : 0)) / SL_CHUNK; };

  if (warp == 0) {
    for (int t = blockIdx.x; ok && epi.tile(t, p0, brow, s0, nst, ax); t += gridDim.x) {
      for (int s = 0; s < nst && ok; ++s, ++g) {
        const int b = g & 1, x = (s0 + s) * SL_BK;
        if (g >= 2 && !mbar_wait(&sm.bempty[b], (uint32_t)((g >> 1) & 1) ^ 1, abort, budget)) { ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&sm.bfull[b], (uint32_t)(nh * SL_B_BYTES));
          for (int h = 0; h < nh; ++h)
            tma_load_2d(sm.bs[b][h], &tmB, &sm.bfull[b], x, brow + h * SL * SL_HALF);
        }
        __syncwarp();
        bissued = g + 1;
        for (int i = 0; i < SL; ++i) {
          if (g >= 1 && !mbar_wait(&sm.aempty[i], (uint32_t)(g & 1) ^ 1, abort, budget)) { ok = false; break; }
          if (elect_one()) {
            mbar_expect_tx(&sm.afull[i], SL_A_BYTES);
            if constexpr (Epi::A_M_MAJOR) {
              tma_load_2d(sm.as[i], &tmA, &sm.afull[i], p0, (int)(i * a_rows) + x);
              tma_load_2d(sm.as[i] + SL_A_BYTES / 2, &tmA, &sm.afull[i], p0 + 64, (int)(i * a_rows) + x);
            } else {
              tma_load_2d(sm.as[i], &tmA, &sm.afull[i], ax + x, (int)(i * a_rows) + p0);
            }
          }
          __syncwarp();
          aissued = g * SL + i + 1;
        }
      }
    }
  } else if (warp == 1) {
    int uses[2] = {0, 0};  // chunks started per accumulator set
    for (int t = blockIdx.x; ok && epi.tile(t, p0, brow, s0, nst, ax); t += gridDim.x) {
      for (int s = 0; s < nst && ok; ++s, ++g) {
        const int b = g & 1;
        if (!mbar_wait(&sm.bfull[b], (uint32_t)(g >> 1) & 1, abort, budget)) { ok = false; break; }
        const bool starts0 = s == 0 || chunk_of(0, s) != chunk_of(0, s - 1);
        for (int q = 0; q < nh && ok; ++q) {
          const int h = (nh == 2 && starts0) ? 1 - q : q;
          const int ck = chunk_of(h, s);
          const bool first = s == 0 || ck != chunk_of(h, s - 1);
          const bool last = s == nst - 1 || ck != chunk_of(h, s + 1);
          const int set = nh == 2 ? h : ck & 1;
          if (first) {
            const int u = set ? uses[1] : uses[0];
            if (u >= 1 && !mbar_wait(&sm.acce[set], (uint32_t)(u - 1) & 1, abort, budget)) {
              ok = false;
              break;
            }
            if (set) ++uses[1]; else ++uses[0];
          }
          const uint32_t dset = tbase + (uint32_t)(set * SL_CLASSES * SL_HALF);
          const uint64_t db = sw128_desc(smem_u32(sm.bs[b][h]));
          for (int i = 0; i < SL; ++i) {
            if (!mbar_wait(&sm.afull[i], (uint32_t)g & 1, abort, budget)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t da = Epi::A_M_MAJOR ? sw128_desc_m(smem_u32(sm.as[i])) : sw128_desc(smem_u32(sm.as[i]));
            constexpr int AK = Epi::A_M_MAJOR ? 16 * 128 / 16 : 2;   // 16 values of k further on, in 16 bytes
            const uint32_t d = dset + (uint32_t)(i * SL_HALF);
            const int nsl = i == 0 ? SL : SL_CLASSES - i;   // N slices 0 .. nsl - 1: classes i .. i + nsl - 1
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < SL_BK / 16; ++k) {        // K = 16 BF16: 32 bytes
                if (first && k == 0 && i == 1) {
                  // classes 1 .. 6 were started by slice 0; class 7 starts here
                  mma_bf16<Epi::A_M_MAJOR>(d, da, db, (SL - 1) * SL_HALF, 1u);
                  mma_bf16<Epi::A_M_MAJOR>(d + (uint32_t)((SL - 1) * SL_HALF), da,
                           db + (uint64_t)(((SL - 1) * SL_HALF * SL_BK * 2) >> 4), SL_HALF, 0u);
                } else {
                  mma_bf16<Epi::A_M_MAJOR>(d, da + AK * k, db + 2 * k, nsl * SL_HALF,
                                           (first && k == 0 && i == 0) ? 0u : 1u);
                }
              }
              if (q == nh - 1) mma_commit(&sm.aempty[i]);
              if (i == SL - 1) {
                if (last) mma_commit(&sm.accf[set]);
                if (q == nh - 1) mma_commit(&sm.bempty[b]);
              }
            }
            __syncwarp();
          }
        }
      }
    }
  } else if (nh == 2 || warp < 6) {
    const int q = warp & 3, grp = (warp - 2) >> 2;
    const uint32_t tq = tbase + ((uint32_t)(32 * q) << 16);
    int uses[2] = {0, 0};
    for (int t = blockIdx.x; ok && epi.tile(t, p0, brow, s0, nst, ax); t += gridDim.x) {
      long long hi[SL_HALF], lo[SL_HALF];
#pragma unroll
      for (int j = 0; j < SL_HALF; ++j) hi[j] = lo[j] = 0;
      const int nchunk = chunk_of(grp, nst - 1) + 1;
      for (int c = 0; c < nchunk; ++c) {
        const int set = nh == 2 ? grp : c & 1;
        const int u = set ? uses[1] : uses[0];
        if (!mbar_wait(&sm.accf[set], (uint32_t)u & 1, abort, budget)) { ok = false; break; }
        if (set) ++uses[1]; else ++uses[0];
        tc_fence_after();
        const uint32_t ta = tq + (uint32_t)(set * SL_CLASSES * SL_HALF);
#pragma unroll
        for (int j0 = 0; j0 < SL_HALF; j0 += 4) {
          float v[SL_CLASSES][4];
#pragma unroll
          for (int k = 0; k < SL_CLASSES; ++k) tmem_ld4(ta + (uint32_t)(k * SL_HALF + j0), v[k]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int s01 = __float2int_rn(v[0][j]) * 256 + __float2int_rn(v[1][j]);   // < 2^28
            const int s23 = __float2int_rn(v[2][j]) * 256 + __float2int_rn(v[3][j]);   // < 2^31
            hi[j0 + j] += (long long)s01 * 65536 + s23;
            // class 7 joins class 6, rounded to its unit
            lo[j0 + j] += (long long)__float2int_rn(v[4][j]) * 65536 + (long long)__float2int_rn(v[5][j]) * 256 +
                          __float2int_rn(fmaf(v[7][j], 0.00390625f, v[6][j]));
          }
        }
        tc_fence_before();
        mbar_arrive(&sm.acce[set]);
      }
      if (ok && !*abort) epi.part(t, p0 + 32 * q + lane, SL_HALF * grp, hi, lo);
    }
  }
  __syncthreads();
  if (*abort) {
    // as k_proj_w_tc: the CTA's own TMA copies and issued MMAs finish before TMEM is freed
    int dummy = 0;
    volatile int* never = &dummy;
    if (threadIdx.x == 0) epi.timeout();
    if (warp == 0 && lane == 0) {
      for (int x = aissued - SL > 0 ? aissued - SL : 0; x < aissued; ++x)
        mbar_wait(&sm.afull[x % SL], (uint32_t)(x / SL) & 1, never);
      for (int s = bissued - 2 > 0 ? bissued - 2 : 0; s < bissued; ++s)
        mbar_wait(&sm.bfull[s & 1], (uint32_t)(s >> 1) & 1, never);
    }
    if (warp == 1) {
      if (elect_one()) mma_commit(&sm.mmadone);
      __syncwarp();
      mbar_wait(&sm.mmadone, 0u, never);
    }
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------
// a7 of the FP64 form: W = Q_blk^T A(:, perm[p]), M = positions (the slices of A stay
// in position order), N = the block's basis columns, K = the m rows, split over
// gridDim.y; FP64 partials per row range, summed by k_proj_finish.
// ---------------------------------------------------------------------------
struct ProjEpi {
  static constexpr bool A_M_MAJOR = false;
  State* st;
  int n, nstages, sps;
  const int* exA;
  const int* exQ;
  double* Wpart;
  int pb, kept, ctiles;   // set by init
  __device__ int init() {
    kept = st->bs;
    pb = st->i + kept;
    ctiles = (n - pb + BM - 1) / BM;
    return kept == 0 || pb >= n ? 0 : kept > SL_HALF ? 2 : 1;
  }
  __device__ bool tile(int t, int& p0, int& brow, int& s0, int& nst, int& ax) const {
    const int z = t / ctiles;
    ax = brow = 0;
    p0 = pb + (t - z * ctiles) * BM;
    s0 = z * sps;
    nst = min(sps, nstages - s0);
    return nst > 0;
  }
  __device__ void part(int t, int p, int a0, const long long (&hi)[SL_HALF], const long long (&lo)[SL_HALF]) const {
    if (p >= n) return;
    const int e = exA[p] - 60;
    double* w = Wpart + ((int64_t)(t / ctiles) * MAXB + a0) * n + p;
#pragma unroll
    for (int j = 0; j < SL_HALF; ++j)
      if (a0 + j < kept) w[(int64_t)j * n] = slice_value(hi[j], lo[j], e + exQ[a0 + j]);
  }
  __device__ void timeout() const { atomicExch(&st->status, ST_ERR_TIMEOUT); }
};

// ---------------------------------------------------------------------------
// a3 of the FP64 form: V(r, c) = A(r, cols[c]) - (Q C)(r, c), M = rows (the basis history's
// columns, M-major), N = the sampled columns, K = the i basis vectors.  8192 rows, 64 columns,
// 288 basis vectors on average: 288 us on the FP64 pipe, 40 here.
// ---------------------------------------------------------------------------
struct CgsEpi {
  static constexpr bool A_M_MAJOR = true;
  State* st;
  int m;
  const double* A;
  int64_t lda;
  const int* cols;
  const int* exC;
  double* V;
  int nst, bss;   // set by init
  __device__ int init() {
    bss = st->bs_sampled;
    nst = (st->i + SL_BK - 1) / SL_BK;
    return bss == 0 || nst == 0 ? 0 : bss > SL_HALF ? 2 : 1;
  }
  __device__ bool tile(int t, int& p0, int& brow, int& s0, int& n, int& ax) const {
    p0 = t * BM;
    brow = s0 = ax = 0;
    n = nst;
    return p0 < m;
  }
  __device__ void part(int, int r, int c0, const long long (&hi)[SL_HALF], const long long (&lo)[SL_HALF]) const {
    if (r >= m) return;
#pragma unroll
    for (int j = 0; j < SL_HALF; ++j) {
      const int c = c0 + j;
      if (c < bss) V[r + (int64_t)c * m] = A[r + (int64_t)cols[c] * lda] - slice_value(hi[j], lo[j], exC[c] - 60);
    }
  }
  __device__ void timeout() const { atomicExch(&st->status, ST_ERR_TIMEOUT); }
};

// R(I2, p) = W (the row ranges summed in order), diags(p) -= ||W(:, p)||^2 clipped at zero
// (a8), and the partials of the residual and the positive count, 32 positions per CTA:
// lane = position, warp w takes the basis columns w, w + 8, ...
__global__ void __launch_bounds__(256)
k_proj_finish(const State* __restrict__ st, const double* __restrict__ Wpart, int nsplit, int n,
              double* __restrict__ R, int64_t ldr, double* __restrict__ diags, double* __restrict__ part_res,
              int* __restrict__ part_nnz) {
  __shared__ double s_sq[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = st->i, kept = st->bs;
  const int p = i + kept + blockIdx.x * 32 + lane;
  double s = 0.0;
  if (kept > 0 && p < n) {
    for (int a = w; a < kept; a += 8) {
      double v = 0.0;
      for (int z = 0; z < nsplit; ++z) v += Wpart[((int64_t)z * MAXB + a) * n + p];
      R[(int64_t)(i + a) * ldr + p] = v;
      s = fma(v, v, s);
    }
  }
  s_sq[w][lane] = s;
  __syncthreads();
  if (w == 0) {
    double d = 0.0;
    if (kept > 0 && p < n) {
      for (int x = 1; x < 8; ++x) s += s_sq[x][lane];
      d = diags[p] - s;
      d = d > 0.0 ? d : (d == d ? 0.0 : d);
      diags[p] = d;
    }
    const int c = __popc(__ballot_sync(0xffffffffu, d > 0.0));
    const double t = warp_sum(d);
    if (lane == 0) {
      part_res[blockIdx.x] = t;
      part_nnz[blockIdx.x] = c;
    }
  }
}

}  // namespace
}  // namespace tc
}  // namespace rbrp
