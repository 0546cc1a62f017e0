// Bucket-based CSC SpMSpV: y = alpha * A * x with x sparse, written back
// without global atomics on y.
//
// The reference's bucket method (CscBasedBucketSpmspvDriver,
// DEV/csc_bucket_spmspv.cuh:768-1087) counts (row, value) pairs per
// row-block bucket and per x entry, scans and scatters them, but its
// reduction is compiled out (:999-1059) and y is never produced.  This is a
// complete design of our own:
//   1. sort:    a load-balanced pass over the pairs; each block of 2,048 work
//               items puts its pairs in bucket order (bucket = row >> rshift) in
//               shared memory and stores them at its own place in the pair
//               arrays, with the offsets of its buckets in a table;
//   2. reduce:  one CTA per bucket collects its segments of all blocks and
//               accumulates them into a dense shared-memory slice of y (shared
//               atomics), writes the slice of the dense y (no memset of y
//               needed) and, in bucket order via a decoupled look-back, the
//               touched rows as sorted (key, value).
// What bounds it: latency; each step is one pass over the pairs in a wave or two.
// x of 105,000 on the 1M Zipf matrix (1.7M pairs, 256 buckets): scan of the columns
// 9 us, sort 21, reduce 24, and the count's read-back, 87 us in all; count,
// scan, scatter of single pairs and a reduction of 256 threads took 135.
// In the reduction 15 of the 24 us are the pairs, 9 the setup, the look-back and
// the output; 1,024 threads per bucket 34 us, 16 lanes per segment 25, the
// segments laid end to end by a scan and searched per pair 29.
// Above kBucketTable buckets a block has under two pairs per bucket and the table
// would outgrow the pairs; there the pairs go to exact places instead: count
// (per-CTA histograms), scan of the counts, scatter (the pass again, each CTA
// reserving its range in every bucket), reduce.
#include "kernels.h"
#include "bucket.h"
#include "sort.h"
#include <algorithm>
#include "common.cuh"
#include "engine.h"
#include "csc_lb.cuh"

namespace spmx {

// Step 1 for at most kBucketTable buckets.  tab[i * stride + b]: first pair of
// bucket i within block b's pairs (bucket nb: their number); block b's pairs
// start at the block's first item.
template <int NT, int VT>
__global__ void __launch_bounds__(NT)
bucket_sort_kernel(CscArgs a, CscScratch s, int rshift, int nb, unsigned short* __restrict__ tab, int stride,
                   int* __restrict__ prow, float* __restrict__ pval, int cap) {
  __shared__ LbSmem<NT, VT> sh;
  __shared__ int s_hist[kBucketTable];
  __shared__ int s_wtmp[NT / 32 + 1];
  const int nblocks = lb_num_blocks(a, s, 1);
  for (int b = blockIdx.x; b < nblocks; b += gridDim.x) {
    for (int i = threadIdx.x; i < nb; i += NT) s_hist[i] = 0;
    const LbBlock bl = lb_block_setup<NT, VT>(a, s, 1, b, nblocks, sh);
    int rr[VT], at[VT];
    float vv[VT];
#pragma unroll
    for (int j = 0; j < VT; ++j) {
      const int q = threadIdx.x + j * NT;
      rr[j] = -1;
      if (q < bl.nk) {
        int k;
        lb_item<NT, VT>(a, s, bl, sh, q, k, rr[j], vv[j]);
        if ((unsigned)rr[j] >= (unsigned)a.m) {
          flag_error(a.err, kDevErrOob);
          rr[j] = -1;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < VT; ++j)
      if (rr[j] >= 0) at[j] = atomicAdd(&s_hist[rr[j] >> rshift], 1);
    __syncthreads();
    // bucket offsets: thread t owns nb / NT consecutive buckets
    const int per = (nb + NT - 1) / NT, i0 = min(nb, (int)threadIdx.x * per), i1 = min(nb, i0 + per);
    int sum = 0;
    for (int i = i0; i < i1; ++i) sum += s_hist[i];
    int total;
    int run = block_exclusive_sum<NT>(sum, s_wtmp, &total);
    for (int i = i0; i < i1; ++i) {
      const int c = s_hist[i];
      s_hist[i] = run;
      tab[(size_t)i * stride + b] = (unsigned short)run;
      run += c;
    }
    if (threadIdx.x == 0) tab[(size_t)nb * stride + b] = (unsigned short)total;
    __syncthreads();
    int* const s_row = sh.off;  // the entry tables are no longer needed
    float* const s_val = reinterpret_cast<float*>(sh.cs);
#pragma unroll
    for (int j = 0; j < VT; ++j) {
      if (rr[j] < 0) continue;
      const int p = s_hist[rr[j] >> rshift] + at[j];
      s_row[p] = rr[j];
      s_val[p] = vv[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < total; i += NT) {
      const int p = bl.k0 + i;
      if (p < cap) {
        prow[p] = s_row[i];
        pval[p] = s_val[i];
      } else {
        flag_error(a.err, kDevErrCapacity);
      }
    }
    __syncthreads();
  }
}

template <int NT, int VT>
__global__ void __launch_bounds__(NT)
bucket_count_kernel(CscArgs a, CscScratch s, int variant, int rshift, int nb,
                    int* __restrict__ gcount) {
  __shared__ LbSmem<NT, VT> sh;
  extern __shared__ int s_hist[];
  const int nblocks = lb_num_blocks(a, s, variant);
  for (int b = blockIdx.x; b < nblocks; b += gridDim.x) {
    for (int i = threadIdx.x; i < nb; i += NT) s_hist[i] = 0;
    const LbBlock bl = lb_block_setup<NT, VT>(a, s, variant, b, nblocks, sh);
    for (int q = threadIdx.x; q < bl.nk; q += NT) {
      int k, r;
      float v;
      lb_item<NT, VT>(a, s, bl, sh, q, k, r, v);
      if ((unsigned)r < (unsigned)a.m) atomicAdd(&s_hist[r >> rshift], 1);
      else flag_error(a.err, kDevErrOob);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += NT)
      if (s_hist[i]) atomicAdd(gcount + i, s_hist[i]);
    __syncthreads();
  }
}

template <int NT, int VT>
__global__ void __launch_bounds__(NT)
bucket_scatter_kernel(CscArgs a, CscScratch s, int variant, int rshift, int nb,
                      int* __restrict__ cursor, int* __restrict__ prow,
                      float* __restrict__ pval, int cap) {
  __shared__ LbSmem<NT, VT> sh;
  extern __shared__ int s_hist[];
  const int nblocks = lb_num_blocks(a, s, variant);
  for (int b = blockIdx.x; b < nblocks; b += gridDim.x) {
    for (int i = threadIdx.x; i < nb; i += NT) s_hist[i] = 0;
    const LbBlock bl = lb_block_setup<NT, VT>(a, s, variant, b, nblocks, sh);
    int rr[VT];
    float vv[VT];
#pragma unroll
    for (int j = 0; j < VT; ++j) {
      const int q = threadIdx.x + j * NT;
      rr[j] = -1;
      if (q < bl.nk) {
        int k;
        lb_item<NT, VT>(a, s, bl, sh, q, k, rr[j], vv[j]);
        if ((unsigned)rr[j] < (unsigned)a.m) atomicAdd(&s_hist[rr[j] >> rshift], 1);
        else rr[j] = -1;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += NT)
      if (s_hist[i]) s_hist[i] = atomicAdd(cursor + i, s_hist[i]);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < VT; ++j) {
      if (rr[j] >= 0) {
        const int slot = atomicAdd(&s_hist[rr[j] >> rshift], 1);
        if (slot < cap) { prow[slot] = rr[j]; pval[slot] = vv[j]; }
        else flag_error(a.err, kDevErrCapacity);
      }
    }
    __syncthreads();
  }
}

// Step 2: bucket bkt's pairs, either one range (boff) or, with a table, a segment
// of every block.
constexpr int kSegLanes = 8;
template <int NT, bool TABLE>
__global__ void __launch_bounds__(NT)
bucket_reduce_kernel(CscArgs a, CscScratch sc, int rshift, int nb, const int* __restrict__ boff,
                     const unsigned short* __restrict__ tab, int stride,
                     const int* __restrict__ prow, const float* __restrict__ pval,
                     float* __restrict__ y, int* __restrict__ ykey,
                     float* __restrict__ yval, int* d_count, LookbackState st,
                     int cap) {
  extern __shared__ float s_dyn[];
  const int m = a.m;
  int* const err = a.err;
  const int R = 1 << rshift;
  float* acc = s_dyn;
  unsigned* tbits = reinterpret_cast<unsigned*>(s_dyn + R);
  const int nwords = R >> 5;
  __shared__ int s_tile;
  __shared__ unsigned s_wtmp[NT / 32 + 1];
  __shared__ unsigned s_prefix, s_total;
  const int bkt = lb_acquire_tile(st, nb, &s_tile);
  const int tid = threadIdx.x;
  for (int i = tid; i < R; i += NT) acc[i] = 0.f;
  for (int i = tid; i < nwords; i += NT) tbits[i] = 0u;
  __syncthreads();
  const int base_row = bkt << rshift;
  const auto add = [&](int row, float v) {
    const int r = row - base_row;
    if ((unsigned)r < (unsigned)R) {
      atomicAdd(&acc[r], v);
      atomicOr(&tbits[r >> 5], 1u << (r & 31));
    } else {
      flag_error(err, kDevErrOob);
    }
  };
  if (TABLE) {
    // kLanes lanes per segment (8 pairs on average at 256 buckets), U segments of
    // each lane group in flight
    constexpr int U = 4, G = NT / kSegLanes;
    const int nblocks = lb_num_blocks(a, sc, 1);
    const int l = tid % kSegLanes;
    for (int b0 = tid / kSegLanes; b0 < nblocks; b0 += U * G) {
      int p[U], e[U], row[U];
      float v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int b = b0 + u * G;
        p[u] = e[u] = 0;
        if (b < nblocks) {
          const int lo = __ldg(tab + (size_t)bkt * stride + b), hi = __ldg(tab + (size_t)(bkt + 1) * stride + b);
          const int from = (int)((long long)b * (kCscLbNT * kCscLbVT) - __ldg(sc.bstart_mg + b));  // the block's first item
          p[u] = from + lo + l;
          e[u] = min(from + hi, cap);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        row[u] = -1;
        if (p[u] < e[u]) {
          row[u] = __ldg(prow + p[u]);
          v[u] = __ldg(pval + p[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (row[u] < 0) continue;
        add(row[u], v[u]);
        for (int q = p[u] + kSegLanes; q < e[u]; q += kSegLanes) add(__ldg(prow + q), __ldg(pval + q));
      }
    }
  } else {
    const int p0 = min(__ldg(boff + bkt), cap), p1 = min(__ldg(boff + bkt + 1), cap);
    for (int p = p0 + tid; p < p1; p += NT) add(__ldg(prow + p), __ldg(pval + p));
  }
  __syncthreads();
  const int rows_here = min(R, m - base_row);
  if (y)
    for (int i = tid; i < rows_here; i += NT) y[base_row + i] = acc[i];
  // touched rows of this bucket, in row order, after all earlier buckets: a scan
  // of the bitmap words' counts (at most NT words), then one warp per word, so
  // that a warp's stores are consecutive
  __shared__ unsigned s_word[NT];
  static_assert(NT >= 8192 / 32, "one bitmap word per thread");
  unsigned total;
  const unsigned cnt = tid < nwords ? __popc(tbits[tid]) : 0u;
  s_word[tid] = block_exclusive_sum<NT>(cnt, s_wtmp, &total);
  if (tid < 32) {
    const unsigned p = lb_warp_lookback(st, bkt, nb, total, err);
    if (tid == 0) { s_prefix = p; s_total = total; }
  }
  __syncthreads();
  if (ykey) {
    const int lane = tid & 31;
    for (int wd = tid >> 5; wd < nwords; wd += NT / 32) {
      const unsigned bits = tbits[wd];
      if (!((bits >> lane) & 1u)) continue;
      const unsigned pos = s_prefix + s_word[wd] + __popc(bits & lanemask_lt());
      ykey[pos] = base_row + wd * 32 + lane;
      yval[pos] = acc[wd * 32 + lane];
    }
  }
  if (bkt == nb - 1 && tid == 0) *d_count = (int)(s_prefix + s_total);
}

int bucket_geometry(int m, int buckets, int* rshift, int* nb) {
  if (buckets <= 0) buckets = 256;
  long long per = ((long long)m + buckets - 1) / buckets;
  int sh = 8;  // at least 256 rows per bucket
  while ((1LL << sh) < per && sh < 13) ++sh;  // at most 8192 rows per bucket
  const long long n = ((long long)m + (1LL << sh) - 1) >> sh;
  if (n > kBucketMax) return -1;
  *rshift = sh;
  *nb = (int)std::max<long long>(n, 1);
  return 0;
}

template <class K>
static void allow_smem(K kernel, int bytes) {
  kernel_smem_limit((const void*)kernel, (size_t)bytes);
}

int launch_bucket_spmspv(const CscArgs& a, const CscScratch& s, const BucketScratch& bs,
                         int variant, int rshift, int nb, float* y, int* ykey,
                         float* yval, int* d_count, ScanScratch& ls, int grid,
                         cudaStream_t st) {
  constexpr int NT = kCscLbNT, VT = kCscLbVT;
  if (nb > ls.status_len) return -1;
  LookbackState lbs{ls.status, ls.ticket};
  const int R = 1 << rshift;
  constexpr int RT = 512;  // threads of the reduction
  // the limits are per function and device: cached per device, set on each
  // device the first time it runs these kernels
  if (nb <= kBucketTable) {
    note_launch(2);
    bucket_sort_kernel<NT, VT><<<grid, NT, 0, st>>>(a, s, rshift, nb, bs.tab, s.mg_cap, bs.prow, bs.pval, bs.cap);
    allow_smem(bucket_reduce_kernel<RT, true>, 4 * (8192 + 8192 / 32));
    bucket_reduce_kernel<RT, true><<<nb, RT, 4 * (R + R / 32), st>>>(a, s, rshift, nb, nullptr, bs.tab, s.mg_cap, bs.prow,
                                                                     bs.pval, y, ykey, yval, d_count, lbs, bs.cap);
    return 0;
  }
  const int hist_bytes = 4 * nb;
  allow_smem(bucket_count_kernel<NT, VT>, 4 * kBucketMax);
  allow_smem(bucket_scatter_kernel<NT, VT>, 4 * kBucketMax);
  allow_smem(bucket_reduce_kernel<RT, false>, 4 * (8192 + 8192 / 32));
  cudaMemsetAsync(bs.gcount, 0, sizeof(int) * (size_t)nb, st);
  note_launch(3);
  bucket_count_kernel<NT, VT><<<grid, NT, hist_bytes, st>>>(a, s, variant, rshift, nb, bs.gcount);
  if (launch_scan_exclusive(bs.gcount, bs.boff, nb, bs.boff + nb, ls, a.err, st)) return -1;
  cudaMemcpyAsync(bs.cursor, bs.boff, sizeof(int) * (size_t)nb, cudaMemcpyDeviceToDevice, st);
  bucket_scatter_kernel<NT, VT><<<grid, NT, hist_bytes, st>>>(a, s, variant, rshift, nb, bs.cursor,
                                                             bs.prow, bs.pval, bs.cap);
  bucket_reduce_kernel<RT, false><<<nb, RT, 4 * (R + R / 32), st>>>(a, s, rshift, nb, bs.boff, nullptr, 0, bs.prow,
                                                                    bs.pval, y, ykey, yval, d_count, lbs, bs.cap);
  return 0;
}

}  // namespace spmx
