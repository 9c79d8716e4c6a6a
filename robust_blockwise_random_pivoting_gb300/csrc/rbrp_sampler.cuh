// rbrp_sampler.cuh - block-wide weighted sampler of one RBRP block.
//
// Shared by the one-matrix kernel (k_sample, 1024 threads) and the batched
// persistent kernel (one CTA per problem).  All state is read from and
// written to a State that may live in global or shared memory.
#pragma once
#include "rbrp_common.cuh"

namespace rbrp {
namespace {

// ===========================================================================
// a2: block sampler.  One CTA over the n - i remaining positions.
// NP: numpy Generator.choice(replace=False, p=w/sum(w)) rounds (python/RBRP.ipynb
//     cell 11 line 108): uniforms from the Philox np-compat stream, cdf by a
//     block scan, searchsorted(side='right') by binary search, first occurrences
//     kept in draw order.  (The reference CUDA sampler draws WITH replacement
//     and may return fewer indices, gpu/rbrp.cu:102-146.)
// ES: keys -log(1-u)/w (u from the exponential-key stream of the original
//     column), the bs smallest by an 8-bit radix select on the key bits.
// GREEDY: the bs largest weights (ties: lower position), same radix select.
// GIVEN: a fixed skeleton: the bs listed columns that come first in the list
//     (order_of[col] = list index, -1 for unlisted), same radix select.
// ===========================================================================
constexpr int SAMPLE_THREADS = 1024;

// Weights, probabilities and cdf values are never negative: their bit patterns order as they
// do, and a comparison on the FP64 pipe takes a warp 20 clocks.
__device__ __forceinline__ bool nonneg_gt(double a, double b) {
  return __double_as_longlong(a) > __double_as_longlong(b);
}

// block_exclusive_scan of one value per thread where `any` tells which warps hold some (the
// others' zeros would only take the FP64 pipe): the same sums in the same order.
__device__ __forceinline__ double scan_active(double v, bool any, double* sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  double x = v;
  if (any) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
  }
  __syncthreads();
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  if (wid == 0) {
    double w = lane < nw ? sh[lane] : 0.0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    sh[lane] = w;
  }
  __syncthreads();
  const double off = wid ? sh[wid - 1] : 0.0;
  __syncthreads();
  double excl = __shfl_up_sync(0xffffffffu, x, 1);
  if (lane == 0) excl = 0.0;
  return off + excl;
}

// Block-wide sampler body (any block size from 64 to MAXT); k_sample runs it with
// 1024 threads, the batched kernel with its CTA.  pre_tot / pre_pos (one entry per thread,
// or NULL): the NP sampler's probabilities are in pbuf already, with the chunk totals and
// counts (k_sample_probs, which spreads their FP64 work over 32 SMs).
template <int MAXT = SAMPLE_THREADS>
__device__ void sample_block(State* st, const double* __restrict__ diags, const int* __restrict__ perm, int n,
                             int kmax, int b, uint64_t seed, int sampler, double* __restrict__ pbuf,
                             unsigned long long* __restrict__ kbuf, int* __restrict__ js, int* __restrict__ cols,
                             const int* __restrict__ order_of = nullptr, const double* __restrict__ pre_tot = nullptr,
                             const int* __restrict__ pre_pos = nullptr) {
  __shared__ double shd[32];
  __shared__ int shi[32];
  __shared__ unsigned int hist[256];
  __shared__ int s_rel[MAXB];
  __shared__ int s_cand[MAXB];
  __shared__ unsigned long long s_key[MAXB];
  __shared__ int s_found, s_size, s_digit, s_krank, s_i, s_done;
  __shared__ unsigned long long s_draws;
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_done = st->done;
    s_i = st->i;
    s_draws = st->draws;
  }
  __syncthreads();
  if (s_done) return;
  const int i = s_i;
  const int nrem = n - i;
  const int req = min(min(kmax - i, b), st->nnz_rem);
  const int chunk = (nrem + (int)blockDim.x - 1) / (int)blockDim.x;
  const int lo = min(nrem, tid * chunk), hi = min(nrem, lo + chunk);
  const double* w = diags + i;

  if (sampler == SAMPLER_NP) {
    // p = w / sum(w)
    int npos = 0;
    if (pre_tot) {
      npos = pre_pos[tid];
    } else {
      double part = 0.0;
      for (int j = lo; j < hi; ++j) part += w[j];
      const double S = block_sum(part, shd);
      // one FP64 division for the block, shared: per-thread or per-entry divisions are
      // ~1/64-rate work on GB300
      __shared__ double s_invS;
      if (tid == 0) s_invS = 1.0 / S;
      __syncthreads();
      const double invS = s_invS;
      for (int j = lo; j < hi; ++j) {
        const double pj = w[j] * invS;
        pbuf[j] = pj;
        npos += nonneg_gt(pj, 0.0);
      }
    }
    npos = block_sum(npos, shi);
    if (tid == 0) {
      s_size = min(req, npos);
      s_found = 0;
    }
    // The cdf is never stored.  Thread t's chunk [lo, hi) keeps its total `tot`; the
    // block scan of the totals gives its offset; cdf(j) = (off + run(j)) * (1 / last),
    // run(j) the chunk-local sequential sum, last = off + tot of the chunk holding
    // index nrem - 1, whose cdf is exactly 1 (numpy's cdf /= cdf[-1]).  A draw
    // binary-searches the chunks' last cdf entries in shared memory, then scans one
    // chunk: the index searchsorted(side='right') returns on the stored cdf.
    __shared__ double s_end[MAXT];
    __shared__ double s_off[MAXT];
    __shared__ double s_last, s_inv_last;
    __shared__ unsigned s_new[2];
    double tot = pre_tot ? pre_tot[tid] : 0.0;
    const bool warp_any = (tid & ~31) * chunk < nrem;   // some thread of this warp holds entries
    __syncthreads();
    // Rejection rounds.  Each round draws at least one new index unless every
    // remaining positive weight is absorbed by rounding in the cdf; the cap
    // turns that (pathological) case into a smaller sample instead of a spin.
    for (int round = 0; s_found < s_size && round < 4096; ++round) {
      const int found = s_found, need = s_size - s_found;
      if (tid < found) {
        pbuf[s_rel[tid]] = 0.0;
        s_end[s_rel[tid] / chunk] = -1.0;   // that chunk's total is to be formed again
      }
      __syncthreads();
      // chunk totals: every chunk in the first round, afterwards the chunks holding a drawn index
      if (round == 0 ? pre_tot == nullptr : __double_as_longlong(s_end[tid]) < 0) {
        double run = 0.0;
        int j = lo;
        for (; j + 8 <= hi; j += 8) {
          double v[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) v[q] = pbuf[j + q];
#pragma unroll
          for (int q = 0; q < 8; ++q) run += v[q];
        }
        for (; j < hi; ++j) run += pbuf[j];
        tot = run;
      }
      const double off = scan_active(tot, warp_any, shd);
      if (lo < hi && hi == nrem) {
        s_last = off + tot;
        s_inv_last = 1.0 / s_last;  // once, by the thread holding the last chunk
      }
      s_off[tid] = off;
      __syncthreads();
      const double inv_last = s_inv_last;
      s_end[tid] = lo < hi ? (hi == nrem ? 1.0 : (off + tot) * inv_last) : 2.0;
      __syncthreads();
      if (tid < need) {
        const double x = np_uniform(seed, s_draws + (unsigned long long)tid);
        int a = 0, z = (int)blockDim.x;  // first chunk whose last cdf entry is > x
        while (a < z) {
          const int mid = (a + z) >> 1;
          if (!nonneg_gt(s_end[mid], x)) a = mid + 1; else z = mid;
        }
        const int t = min(a, (int)blockDim.x - 1);
        const int clo = min(nrem, t * chunk), chi = min(nrem, clo + chunk);
        const double co = s_off[t];
        int pick = chi - 1;
        double run = 0.0;
        bool hit = false;
        for (int j0 = clo; j0 < chi && !hit; j0 += 8) {
          double v[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) v[q] = j0 + q < chi ? pbuf[j0 + q] : 0.0;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int j = j0 + q;
            if (!hit && j < chi) {
              run += v[q];
              const double c = j == nrem - 1 ? 1.0 : (co + run) * inv_last;
              if (nonneg_gt(c, x)) {
                pick = j;
                hit = true;
              }
            }
          }
        }
        s_cand[tid] = pick < nrem ? pick : nrem - 1;
      }
      __syncthreads();
      // first occurrences in draw order, 64 threads side by side (one thread comparing all
      // pairs took 8 of a 64-column block's 41 us)
      bool fresh = tid < need;
      int mine = -1;
      if (tid < MAXB) {
        if (fresh) {
          mine = s_cand[tid];
          for (int u = 0; u < tid; ++u) fresh = fresh && s_cand[u] != mine;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, fresh);
        if ((tid & 31) == 0) s_new[tid >> 5] = bal;
      }
      __syncthreads();
      const unsigned n0 = s_new[0], n1 = s_new[1];
      if (fresh) {
        const unsigned before = (1u << (tid & 31)) - 1u;
        s_rel[found + (tid < 32 ? __popc(n0 & before) : __popc(n0) + __popc(n1 & before))] = mine;
      }
      if (tid == 0) {
        s_found = found + __popc(n0) + __popc(n1);
        s_draws += (unsigned long long)need;
      }
      __syncthreads();
    }
    if (tid == 0) s_size = s_found;
    __syncthreads();
  } else {
    // keys (ascending = preferred); each thread also keeps its smallest (key, position)
    int npos = 0;
    unsigned long long bk = ~0ull;
    int bj = 0x7fffffff;
    for (int j = lo; j < hi; ++j) {
      const double wj = w[j];
      unsigned long long key = ~0ull;
      if (sampler == SAMPLER_GIVEN) {
        // fixed skeleton: columns of the list (order_of[col] >= 0), earliest first
        const int o = order_of[perm[i + j]];
        if (wj > 0.0 && o >= 0) {
          ++npos;
          key = (unsigned long long)o;
        }
      } else if (wj > 0.0) {
        ++npos;
        if (sampler == SAMPLER_ES) {
          const double u = es_uniform(seed, (uint64_t)st->attempts, (uint64_t)perm[i + j]);
          const double e = -log(1.0 - u) / wj;
          key = (unsigned long long)__double_as_longlong(e);
        } else {
          key = 0x7FF0000000000000ull - (unsigned long long)__double_as_longlong(wj);
        }
      }
      kbuf[j] = key;
      if (key < bk) bk = key, bj = j;
    }
    npos = block_sum(npos, shi);
    const int size = min(req, npos);
    if (size == 1) {
      // one index (greedy b = 1 is column-pivoted QR): argmin of (key, position),
      // the element the radix select below would return
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long ok = __shfl_xor_sync(0xffffffffu, bk, o);
        const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
        if (ok < bk || (ok == bk && oj < bj)) bk = ok, bj = oj;
      }
      if ((tid & 31) == 0) {
        s_key[tid >> 5] = bk;
        s_cand[tid >> 5] = bj;
      }
      __syncthreads();
      if (tid == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
          if (s_key[w] < s_key[0] || (s_key[w] == s_key[0] && s_cand[w] < s_cand[0])) s_key[0] = s_key[w], s_cand[0] = s_cand[w];
        s_rel[0] = s_cand[0];
        s_size = 1;
        s_found = 1;
      }
      __syncthreads();
    } else {
      // radix select of the size-th smallest key
      unsigned long long prefix = 0ull, mask = 0ull;
      int krank = size;
      for (int shift = 56; shift >= 0 && size > 0; shift -= 8) {
        for (int d = tid; d < 256; d += blockDim.x) hist[d] = 0u;
        __syncthreads();
        for (int j = lo; j < hi; ++j) {
          const unsigned long long k = kbuf[j];
          if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 0xFF], 1u);
        }
        __syncthreads();
        if (tid == 0) {
          int cum = 0, d = 0;
          for (; d < 255; ++d) {
            if (cum + (int)hist[d] >= krank) break;
            cum += (int)hist[d];
          }
          s_digit = d;
          s_krank = krank - cum;
        }
        __syncthreads();
        prefix |= (unsigned long long)s_digit << shift;
        mask |= 0xFFull << shift;
        krank = s_krank;
        __syncthreads();
      }
      const unsigned long long kth = prefix;
      int nlt = 0, neq = 0;
      for (int j = lo; j < hi; ++j) {
        const unsigned long long k = kbuf[j];
        nlt += k < kth;
        neq += k == kth;
      }
      int tot_lt, tot_eq;
      const int off_lt = block_exclusive_scan(nlt, shi, &tot_lt);
      const int off_eq = block_exclusive_scan(neq, shi, &tot_eq);
      const int ties = size - tot_lt;
      int a = off_lt, e = off_eq;
      if (size > 0) {
        for (int j = lo; j < hi; ++j) {
          const unsigned long long k = kbuf[j];
          if (k < kth) {
            s_key[a] = k;
            s_cand[a] = j;
            ++a;
          } else if (k == kth) {
            if (e < ties) {
              s_key[tot_lt + e] = k;
              s_cand[tot_lt + e] = j;
            }
            ++e;
          }
        }
      }
      __syncthreads();
      if (tid < size) {
        const unsigned long long k = s_key[tid];
        const int j = s_cand[tid];
        int rank = 0;
        for (int u = 0; u < size; ++u) {
          const unsigned long long ku = s_key[u];
          rank += (ku < k) || (ku == k && s_cand[u] < j);
        }
        s_rel[rank] = j;
      }
      if (tid == 0) {
        s_size = size;
        s_found = size;
      }
      __syncthreads();
    }
  }
  const int size = s_size;
  if (tid < size) {
    const int p = i + s_rel[tid];
    js[tid] = p;
    cols[tid] = perm[p];
  }
  if (tid == 0) {
    st->bs_sampled = size;
    st->draws = s_draws;
  }
  __syncthreads();
}

// The NP sampler's FP64 passes for many columns: thread t of k_sample's 1024 owns the chunk
// [t chunk, (t + 1) chunk) of the remaining positions; here chunk t belongs to thread t % 32 of
// CTA t / 32, so the sums keep their order and take 32 SMs' FP64 pipes instead of one's.
constexpr int SAMPLE_PRE_MIN = 15 * SAMPLE_THREADS + 1;   // remaining positions from which the two launches
// pay: 16 a thread (us a block in one launch and in three: 8,300 columns 48 and 63, 13,000 61 and 66, 15,000
// 68 and 68, 15,424 104 and 65, 32,000 186 and 80)

// part[t] = sum of the chunk's weights
__global__ void __launch_bounds__(32)
k_sample_sums(const State* __restrict__ st, const double* __restrict__ diags, int n, double* __restrict__ part) {
  const int nrem = n - st->i, t = blockIdx.x * 32 + threadIdx.x;
  const int chunk = (nrem + SAMPLE_THREADS - 1) / SAMPLE_THREADS;
  const int lo = min(nrem, t * chunk), hi = min(nrem, lo + chunk);
  const double* w = diags + st->i;
  double s = 0.0;
#pragma unroll 8
  for (int j = lo; j < hi; ++j) s += w[j];
  part[t] = s;
}

// p = w / sum(w) into pbuf, chunk totals of p and counts of positive p.  Every CTA adds up the
// 1024 partial sums as block_sum does.
__global__ void __launch_bounds__(32)
k_sample_probs(const State* __restrict__ st, const double* __restrict__ diags, int n, const double* __restrict__ part,
               double* __restrict__ pbuf, double* __restrict__ tot, int* __restrict__ pos) {
  const int nrem = n - st->i, lane = threadIdx.x, t = blockIdx.x * 32 + lane;
  const int chunk = (nrem + SAMPLE_THREADS - 1) / SAMPLE_THREADS;
  const int lo = min(nrem, t * chunk), hi = min(nrem, lo + chunk);
  const double* w = diags + st->i;
  double mine = 0.0;
#pragma unroll 4
  for (int q = 0; q < 32; ++q) {
    const double s = __shfl_sync(0xffffffffu, warp_sum(part[32 * q + lane]), 0);
    if (lane == q) mine = s;
  }
  const double S = __shfl_sync(0xffffffffu, warp_sum(mine), 0);
  const double invS = 1.0 / S;
  double run = 0.0;
  int np = 0;
#pragma unroll 8
  for (int j = lo; j < hi; ++j) {
    const double pj = w[j] * invS;
    pbuf[j] = pj;
    np += nonneg_gt(pj, 0.0);
    run += pj;
  }
  tot[t] = run;
  pos[t] = np;
}

}  // namespace
}  // namespace rbrp
