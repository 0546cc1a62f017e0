#include <algorithm>
// CSC SpMSpV kernels: y = alpha * A * x with x sparse (x_key, x_val).
//
// Stage 1, csc_scan_kernel: gathers the length of every selected column
//   (colptr[k+1]-colptr[k]), scans them into offsets in one pass (decoupled
//   look-back with status words, bounded waits) and, fused into the same pass,
//   writes the block-start tables of both load-balanced partitions.  This
//   replaces scanFuseKernel + DetermineBlockStarts / my_KernelMergePartition
//   (DEV/scan_kernel.cuh:12-143, DEV/csc_two_layer_load_balance.cuh:576,
//   DEV/csc_sort_load_balance.cuh:295) whose look-back spins without bound on
//   `sum[gid-1]==0` (scan_kernel.cuh:99).
//
// The dense-y (atomic) write-back of a handle, and its sorted (key, value)
// write-back up to a number of rows, need no global scan: csc_flat_kernel.
//
// Stage 2 of the sort write-back above that, and of the allocation-free entry point (the
//   bucket kernels share the block mapping), csc_lb_kernel: persistent CTAs take blocks of 2048 work items.
//   "twolayer" blocks hold 2048 nonzeros (DEV/csc_two_layer_load_balance_
//   fuse_reduction_modify.cuh:155); "merge" blocks hold 2048 merge-path items
//   = nonzeros + column ends (DEV/csc_sort_load_balance_fuse_reduction_
//   modify.cuh:7), which bounds the number of x entries per block.  Inside a
//   block the owner entry of every item comes from a max-scan over entry-start
//   marks in shared memory (no per-item search), and consecutive threads read
//   consecutive nonzeros of a column.
//
// naive: a group of G lanes per x entry walks its column (ExtractFuseKernel,
//   DEV/csc_sort_spmspv.cuh:98-119, is G = 1).
#include "kernels.h"
#include "common.cuh"
#include "csc_lb.cuh"

namespace spmx {

template <int NT, int VT>
__global__ void __launch_bounds__(NT)
csc_scan_kernel(CscArgs a, CscScratch s, LookbackState st, int ntiles) {
  constexpr long long K = kCscLbNT * kCscLbVT;  // items per block
  __shared__ int s_len[NT * VT];
  __shared__ unsigned s_wtmp[NT / 32 + 1];
  __shared__ int s_tile;
  __shared__ unsigned s_prefix;
  const int tile = lb_acquire_tile(st, ntiles, &s_tile);
  const int base = tile * NT * VT;
  const int tid = threadIdx.x;
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int i = base + j * NT + tid;
    int len = 0;
    if (i < a.x_nnz) {
      const int key = __ldg(a.x_key + i);
      int cs = 0;
      if ((unsigned)key >= (unsigned)a.n) {
        flag_error(a.err, kDevErrOob);
      } else {
        cs = __ldg(a.colptr + key);
        len = __ldg(a.colptr + key + 1) - cs;
      }
      s.colstart[i] = cs;
    }
    s_len[j * NT + tid] = len;
  }
  __syncthreads();
  unsigned lens[VT];
  unsigned sum = 0;
#pragma unroll
  for (int j = 0; j < VT; ++j) { lens[j] = (unsigned)s_len[tid * VT + j]; sum += lens[j]; }
  unsigned total;
  const unsigned ex = block_exclusive_sum<NT>(sum, s_wtmp, &total);
  if (tid < 32) {
    const unsigned p = lb_warp_lookback(st, tile, ntiles, total, a.err);
    if (tid == 0) s_prefix = p;
  }
  __syncthreads();
  unsigned prefix = s_prefix + ex;
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int i = base + tid * VT + j;
    if (i < a.x_nnz) {
      s.off[i] = (int)prefix;
      const long long p = prefix, len = lens[j];
      if (len > 0) {
        for (long long b = (p + K - 1) / K; b * K < p + len; ++b) {
          if (b < s.tl_cap) s.bstart_tl[b] = i; else flag_error(a.err, kDevErrCapacity);
        }
      }
      const long long lo = p + i, hi = p + len + i + 1;
      for (long long b = (lo + K - 1) / K; b * K < hi; ++b) {
        if (b < s.mg_cap) s.bstart_mg[b] = i; else flag_error(a.err, kDevErrCapacity);
      }
      prefix += lens[j];
    }
  }
  if (tile == ntiles - 1 && tid == 0) {
    const long long bl = (long long)s_prefix + total;
    s.off[a.x_nnz] = (int)bl;
    a.counts[kCntBinlen] = (int)bl;
    a.counts[kCntBlocksTL] = (int)((bl + K - 1) / K);
    a.counts[kCntBlocksMG] = (int)((bl + a.x_nnz + K - 1) / K);
  }
}

template <int NT, int VT, bool PAIRS>
__global__ void __launch_bounds__(NT)
csc_lb_kernel(CscArgs a, CscScratch s, int variant, float* __restrict__ y,
              int* __restrict__ prow, float* __restrict__ pval) {
  __shared__ LbSmem<NT, VT> sh;
  const int nblocks = lb_num_blocks(a, s, variant);
  for (int b = blockIdx.x; b < nblocks; b += gridDim.x) {
    const LbBlock bl = lb_block_setup<NT, VT>(a, s, variant, b, nblocks, sh);
    for (int q = threadIdx.x; q < bl.nk; q += NT) {
      int k, r;
      float v;
      lb_item<NT, VT>(a, s, bl, sh, q, k, r, v);
      if (PAIRS) {
        prow[k] = r;
        pval[k] = v;
      } else if ((unsigned)r < (unsigned)a.m) {
        atomicAdd(y + r, v);
      } else {
        flag_error(a.err, kDevErrOob);
      }
    }
    __syncthreads();
  }
}

// y is zero-filled by the grid launched before this one (zero_fill_kernel).
// With programmatic dependent launch this grid starts early: it reads x, the
// column bounds and the first row / value while y is being cleared, and waits
// (griddepcontrol.wait, a no-op without the launch attribute) only before its
// first atomic.
template <int G, int U>
__global__ void __launch_bounds__(256)
csc_naive_kernel(CscArgs a, float* __restrict__ y) {
  // G lanes per x entry; each lane group takes U entries, gid / G + u * groups,
  // whose loads are issued phase by phase (all keys, then all column bounds,
  // then all first nonzeros), so one chain of memory round trips covers U
  // entries
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long groups = (long long)gridDim.x * blockDim.x / G;
  const int g = (int)(gid % G);
  int key[U], cs[U], ce[U], r0[U];
  float xv[U], v0[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = gid / G + u * groups;
    key[u] = i < a.x_nnz ? __ldg(a.x_key + i) : -1;
    xv[u] = i < a.x_nnz ? __ldg(a.x_val + i) : 0.f;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = gid / G + u * groups;
    const bool ok = (unsigned)key[u] < (unsigned)a.n;
    if (i < a.x_nnz && !ok && g == 0) flag_error(a.err, kDevErrOob);
    cs[u] = ok ? __ldg(a.colptr + key[u]) : 0;
    ce[u] = ok ? __ldg(a.colptr + key[u] + 1) : 0;
    xv[u] = (float)(a.alpha * (double)xv[u]);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    r0[u] = -1;
    v0[u] = 0.f;
    if (cs[u] + g < ce[u]) {
      r0[u] = __ldg(a.row + cs[u] + g);
      v0[u] = __ldg(a.val + cs[u] + g);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // the next call's first grid may launch now (it waits for this one before
  // it touches memory)
  asm volatile("griddepcontrol.launch_dependents;");
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (cs[u] + g < ce[u]) {
      if ((unsigned)r0[u] < (unsigned)a.m) atomicAdd(y + r0[u], v0[u] * xv[u]);
      else flag_error(a.err, kDevErrOob);
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
#pragma unroll 4
    for (int k = cs[u] + g + G; k < ce[u]; k += G) {
      const int r = __ldg(a.row + k);
      if ((unsigned)r < (unsigned)a.m) atomicAdd(y + r, __ldg(a.val + k) * xv[u]);
      else flag_error(a.err, kDevErrOob);
    }
  }
}

static_assert(kCntLong % 2 == 0 && kCntLong + 2 <= kCntFeatSum, "an aligned 64-bit counter of its own");
__host__ __device__ __forceinline__ unsigned long long* long_count(const CscArgs& a) {
  return reinterpret_cast<unsigned long long*>(a.counts + kCntLong);
}

template <class T>
__device__ __forceinline__ void row_add(T* y, float v) {
  // v + 0.0 is never -0.0, nor is a sum that it entered
  if (sizeof(T) == 8) atomicAdd(y, (T)v + (T)0);
  else atomicAdd(y, (T)v);
}

// The warp's products r, v (r = -1: none) into y, those of one row as one.  A row
// that holds most columns otherwise takes one reduction after the other at 1.5 ns
// each: 9 nonzeros a column, one row full, x of 1M 1,570 us against 484 so; but
// without such a row 78 against 118, match_any being a loop over the distinct rows.
template <class T>
__device__ __forceinline__ void row_add_warp(T* y, int r, float v) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(FULL, r);
  double d = (double)v + 0.0;
  for (unsigned left = __ballot_sync(FULL, r >= 0 && (same & (same - 1))); left;) {
    const int src = __ffs(left) - 1;
    const unsigned grp = __shfl_sync(FULL, same, src);
    const double t = warp_sum((grp >> lane) & 1u ? d : 0.0);
    if (lane == src) d = t;
    left &= ~grp;
  }
  if (r >= 0 && lane == __ffs(same) - 1) atomicAdd(y + r, (T)d);
}

// Load-balanced SpMSpV with atomic write-back, without a scan: a warp takes E
// consecutive x entries (E = 2^elog <= 32), scans their column lengths with
// shuffles and spreads the nonzeros over its lanes, U per lane in flight; a
// column above kFlatCut nonzeros is handed to csc_flat_long_kernel in chunks, so
// no warp serialises on a hub.  Everything up to the first U nonzeros is read
// before the wait for the zero fill.  The owner of a nonzero is found by binary
// search over the lanes' prefix.
//
// What bounds it: the latency of x key -> column bounds -> nonzeros over three
// chained grids (5 us for a handful of entries), then the L2 reductions, which
// serialise on the rows of hubs.  1M-vertex Chung-Lu graph, x of 10,000 entries
// (0.3M nonzeros): 13.4 us against 43 for memset, scan, block tables and
// csc_lb_kernel (27 of it the scan in 5 CTAs); x of 100,000: 96 against 161;
// Zipf 1M, x of 105,000: 19.8 against 43.6.  Cut and chunk (10,000 / 100,000
// entries): 512 and 256 16.7 / 141 us, 256 and 256 14.7 / 106, 128 and 128 13.4 /
// 96, 64 and 64 13.6 / 85.  Two nonzeros in flight per lane instead of four 14.2 /
// 108, eight 15.6 / 122.
//
// T = double: y starts at -0.0 (row_add), so that it tells the rows reached.
template <int U, class T, bool COMBINE>
__global__ void __launch_bounds__(256)
csc_flat_kernel(CscArgs a, int elog, T* __restrict__ y, CscLong* queue, int qcap, int defer) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ unsigned s_bin[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long i = (((long long)blockIdx.x * 8 + w) << elog) + lane;
  const bool mine = lane < (1 << elog) && i < a.x_nnz;
  const int key = mine ? __ldg(a.x_key + i) : -1;
  float xv = mine ? __ldg(a.x_val + i) : 0.f;
  const bool ok = (unsigned)key < (unsigned)a.n;
  if (mine && !ok) flag_error(a.err, kDevErrOob);
  int cs = 0, len = 0;
  if (ok) {
    cs = __ldg(a.colptr + key);
    len = __ldg(a.colptr + key + 1) - cs;
  }
  xv = (float)(a.alpha * (double)xv);
  const bool is_long = defer && len > kFlatCut;
  const int flat = is_long ? 0 : len;
  const int incl = warp_inclusive_sum(flat);
  const int base = cs - (incl - flat);  // position of the warp's item q: base of its owner + q
  const int total = __shfl_sync(FULL, incl, 31);
  const unsigned bins = __reduce_add_sync(FULL, (unsigned)len);
  if (lane == 0) s_bin[w] = bins;
  int r[U];
  float v[U];
  auto load = [&](int q0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = q0 + u * 32 + lane;
      int o = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int t = __shfl_sync(FULL, incl, o + step - 1);
        if (t <= q) o += step;
      }
      const int p = __shfl_sync(FULL, base, o) + q;
      const float x = __shfl_sync(FULL, xv, o);
      r[u] = -1;
      v[u] = 0.f;
      if (q < total) {
        r[u] = __ldg(a.row + p);
        v[u] = __ldg(a.val + p) * x;
      }
    }
  };
  load(0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  for (int q0 = 0;;) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (COMBINE) {
        const bool in = (unsigned)r[u] < (unsigned)a.m;
        if (!in && q0 + u * 32 + lane < total) flag_error(a.err, kDevErrOob);
        row_add_warp(y, in ? r[u] : -1, v[u]);
        continue;
      }
      if (q0 + u * 32 + lane >= total) continue;
      if ((unsigned)r[u] < (unsigned)a.m) row_add(y + r[u], v[u]);
      else flag_error(a.err, kDevErrOob);
    }
    q0 += 32 * U;
    if (q0 >= total) break;
    load(q0);
  }
  // hand the long columns over, chunk by chunk
  for (unsigned lm = __ballot_sync(FULL, is_long); lm; lm &= lm - 1) {
    const int sl = __ffs(lm) - 1;
    const int c0 = __shfl_sync(FULL, cs, sl), c1 = c0 + __shfl_sync(FULL, len, sl);
    const float x = __shfl_sync(FULL, xv, sl);
    const int nch = (c1 - c0 + kFlatChunk - 1) / kFlatChunk;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(long_count(a), (unsigned long long)nch);
    at = __shfl_sync(FULL, at, 0);
    for (int j = lane; j < nch; j += 32) {
      const int s0 = c0 + j * kFlatChunk, s1 = min(c1, s0 + kFlatChunk);
      if (at + j < (unsigned long long)qcap) {
        queue[at + j] = CscLong{s0, s1, x};
      } else {  // only with repeated x keys: this lane's chunk on the spot
        for (int k = s0; k < s1; ++k) {
          const int rr = __ldg(a.row + k);
          if ((unsigned)rr < (unsigned)a.m) row_add(y + rr, __ldg(a.val + k) * x);
          else flag_error(a.err, kDevErrOob);
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned t = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += s_bin[q];
    if (t) atomicAdd(a.counts + kCntBinlen, (int)t);
  }
}

// the chunks of the long columns, one warp each
template <class T>
__global__ void __launch_bounds__(256)
csc_flat_long_kernel(CscArgs a, T* __restrict__ y, const CscLong* queue, int qcap) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  constexpr int U = 8;
  const int cnt = (int)min(*(volatile unsigned long long*)long_count(a), (unsigned long long)qcap);
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < cnt; c += nw) {
    const CscLong ch = queue[c];
    for (int kb = ch.k0; kb < ch.k1; kb += 32 * U) {
      int r[U];
      float v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = kb + u * 32 + lane;
        r[u] = k < ch.k1 ? __ldg(a.row + k) : -1;
        v[u] = k < ch.k1 ? __ldg(a.val + k) * ch.x : 0.f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (kb + u * 32 + lane >= ch.k1) continue;
        if ((unsigned)r[u] < (unsigned)a.m) row_add(y + r[u], v[u]);
        else flag_error(a.err, kDevErrOob);
      }
    }
  }
}

template <int G>
__global__ void __launch_bounds__(256)
csc_naive_pairs_kernel(CscArgs a, CscScratch s, int* __restrict__ prow,
                       float* __restrict__ pval) {
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(gid / G);
  const int g = (int)(gid % G);
  if (i >= a.x_nnz) return;
  const int cs = __ldg(s.colstart + i);
  const int o = __ldg(s.off + i);
  const int len = __ldg(s.off + i + 1) - o;
  const float xv = (float)(a.alpha * (double)__ldg(a.x_val + i));
  for (int q = g; q < len; q += G) {
    prow[o + q] = __ldg(a.row + cs + q);
    pval[o + q] = __ldg(a.val + cs + q) * xv;
  }
}

// --------------------------------------------------------------------------
// tiles of 512 entries, four times as many CTAs, while these are one wave (8 per
// SM) and the status array holds their look-back words: 105,000 entries 9 us
// against 14 in tiles of 2,048, 35,000 6 against 10.7; 1M entries 15 us more
int launch_csc_scan(const CscArgs& a, const CscScratch& s, ScanScratch& ls, cudaStream_t st) {
  constexpr int NT = kCscScanNT, VT = kCscScanVT, VS = 2;
  if (a.x_nnz <= 0) return 0;
  LookbackState lbs{ls.status, ls.ticket};
  const int small = (int)(((long long)a.x_nnz + NT * VS - 1) / (NT * VS));
  note_launch();
  if (small <= 148 * 8 && small <= ls.status_len) {
    csc_scan_kernel<NT, VS><<<small, NT, 0, st>>>(a, s, lbs, small);
    return 0;
  }
  const int ntiles = (a.x_nnz + NT * VT - 1) / (NT * VT);
  if (ntiles > ls.status_len) return -1;
  csc_scan_kernel<NT, VT><<<ntiles, NT, 0, st>>>(a, s, lbs, ntiles);
  return 0;
}

int launch_csc_lb(const CscArgs& a, const CscScratch& s, int variant, float* y,
                  int* pairs_row, float* pairs_val, int grid, cudaStream_t st) {
  constexpr int NT = kCscLbNT, VT = kCscLbVT;
  if (a.x_nnz <= 0 || grid <= 0) return 0;
  note_launch();
  if (pairs_row)
    csc_lb_kernel<NT, VT, true><<<grid, NT, 0, st>>>(a, s, variant, y, pairs_row, pairs_val);
  else
    csc_lb_kernel<NT, VT, false><<<grid, NT, 0, st>>>(a, s, variant, y, pairs_row, pairs_val);
  return 0;
}

#define SPMX_GROUP_SWITCH(G_, BODY)                                              \
  switch (G_) {                                                                 \
    case 1: { constexpr int G = 1; BODY; break; }                               \
    case 2: { constexpr int G = 2; BODY; break; }                               \
    case 4: { constexpr int G = 4; BODY; break; }                               \
    case 8: { constexpr int G = 8; BODY; break; }                               \
    case 16: { constexpr int G = 16; BODY; break; }                             \
    case 32: { constexpr int G = 32; BODY; break; }                             \
    default: return -1;                                                         \
  }

// y[0..m) = 0.  Launched as a programmatic dependent of the grid before it on
// the stream, it waits for that grid before its first store, and only then
// lets the next grid launch: a dependent that reads its inputs before its own
// wait (x keys, column bounds) therefore never starts while a grid that
// writes them is still running.
// c0 / c1 (optional) are cleared too: counters of the grid that follows.
// NEG: y holds m / 2 doubles (16-byte aligned), which become -0.0.
template <bool NEG>
__global__ void zero_fill_kernel(float* __restrict__ y, long long m, int* c0, unsigned long long* c1) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (c0) *c0 = 0;
    if (c1) *c1 = 0ull;
  }
  constexpr float hi = NEG ? -0.0f : 0.0f;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nt = (long long)gridDim.x * blockDim.x;
  if ((((uintptr_t)y) & 15u) == 0) {
    float4* y4 = reinterpret_cast<float4*>(y);
    const long long m4 = m >> 2;
    for (long long i = tid; i < m4; i += nt) y4[i] = make_float4(0.f, hi, 0.f, hi);
    for (long long i = (m4 << 2) + tid; i < m; i += nt) y[i] = (i & 1) ? hi : 0.f;
  } else {
    for (long long i = tid; i < m; i += nt) y[i] = (i & 1) ? hi : 0.f;
  }
}

// The zero fill opens a call, so it is launched as a programmatic dependent of
// whatever grid ran before it (the previous call's last kernel): its launch
// and CTA start-up overlap that grid's tail (2.4 -> 1.2 us per kernel boundary
// measured on B200), and its griddepcontrol.wait keeps the order.
int launch_zero_fill(float* y, long long m, int num_sms, cudaStream_t st, int* c0, unsigned long long* c1) {
  if (m <= 0 && !c0 && !c1) return 0;
  const long long blocks = std::min<long long>((m + 1023) / 1024, (long long)num_sms * 4);
  note_launch();
  return launch_pdl(zero_fill_kernel<false>, dim3((unsigned)std::max(1LL, blocks)), dim3(256), 0, st, y, m, c0, c1) ==
                 cudaSuccess
             ? 0
             : -2;
}

// A handful of x entries (one warp's worth) in one launch: every CTA owns a slice
// of y in shared memory, reads all the products (kSliceItems at most, from L2
// but for the first CTA), adds those of its rows and stores the whole slice, so
// y needs no fill before.
//
// What it saves is a launch: x of 11 entries on 1M rows 5.3 us per call from
// Python against 7.7 with the zero fill and the scatter, each of whose launches
// takes the host 2.2 us.  On the device alone the pair is faster (2.5 us per call
// enqueued ahead, against 3.0, and 3.5 for 32 entries), because the scatter
// reads x and its columns while y is being cleared, so a capture, which pays no
// launches, keeps the pair.
constexpr int kSliceNT = 256, kSliceRows = 4096, kSliceItems = 2048;
constexpr int kSliceMaxRows = 148 * 8 * kSliceRows;  // one wave of CTAs

__global__ void __launch_bounds__(kSliceNT)
csc_slice_kernel(CscArgs a, float* __restrict__ y) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ __align__(16) float s_acc[kSliceRows];
  const int tid = threadIdx.x, lane = tid & 31;
  for (int i = tid; i < kSliceRows / 4; i += kSliceNT)
    reinterpret_cast<float4*>(s_acc)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  // every warp for itself: the entries' columns and a prefix of their lengths
  const int key = lane < a.x_nnz ? a.x_key[lane] : -1;
  float xv = lane < a.x_nnz ? a.x_val[lane] : 0.f;
  const bool ok = (unsigned)key < (unsigned)a.n;
  if (lane < a.x_nnz && !ok) flag_error(a.err, kDevErrOob);
  int cs = 0, len = 0;
  if (ok) {
    cs = a.colptr[key];
    len = a.colptr[key + 1] - cs;
  }
  xv = (float)(a.alpha * (double)xv);
  const int incl = warp_inclusive_sum(len);
  const int base = cs - (incl - len);
  const int total = __shfl_sync(FULL, incl, 31);
  const int row0 = blockIdx.x * kSliceRows;
  __syncthreads();  // the slice is clear
  for (int q0 = tid & ~31; q0 < total; q0 += kSliceNT) {
    const int q = q0 + lane;
    int o = 0;  // the entry that owns item q
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (__shfl_sync(FULL, incl, o + step - 1) <= q) o += step;
    const int p = __shfl_sync(FULL, base, o) + q;
    const float x = __shfl_sync(FULL, xv, o);
    if (q < total) {
      const int r = a.row[p];
      if ((unsigned)r >= (unsigned)a.m) flag_error(a.err, kDevErrOob);
      else if ((unsigned)(r - row0) < (unsigned)kSliceRows) atomicAdd(&s_acc[r - row0], a.val[p] * x);
    }
  }
  __syncthreads();
  const int rows = min(kSliceRows, a.m - row0);
  float* const out = y + row0;
  if ((((uintptr_t)out) & 15u) == 0) {
    for (int i = tid; i < rows >> 2; i += kSliceNT)
      reinterpret_cast<float4*>(out)[i] = reinterpret_cast<const float4*>(s_acc)[i];
    for (int i = (rows & ~3) + tid; i < rows; i += kSliceNT) out[i] = s_acc[i];
  } else {
    for (int i = tid; i < rows; i += kSliceNT) out[i] = s_acc[i];
  }
}

bool csc_slice_fits(const CscArgs& a, long long col_max, cudaStream_t st) {
  if (a.x_nnz > 32 || a.m > kSliceMaxRows || col_max < 0 || a.x_nnz * col_max > kSliceItems) return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();
  return cap == cudaStreamCaptureStatusNone;
}

int launch_csc_slice(const CscArgs& a, float* y, cudaStream_t st) {
  if (a.m <= 0) return 0;
  note_launch();
  return launch_pdl(csc_slice_kernel, dim3((unsigned)((a.m + kSliceRows - 1) / kSliceRows)), dim3(kSliceNT), 0, st, a,
                    y) == cudaSuccess
             ? 0
             : -2;
}

// zero y, then the naive CSC SpMSpV as a programmatic dependent launch
int launch_csc_naive_zeroed(const CscArgs& a, int group, float* y, int num_sms, cudaStream_t st) {
  if (a.m > 0 && launch_zero_fill(y, a.m, num_sms, st)) return -2;
  if (a.x_nnz <= 0) return 0;
  // entries per lane group: enough that the grid is about one wave of
  // resident threads (2,048 per SM), at most 4
  const long long threads = (long long)a.x_nnz * group;
  const long long resident = (long long)num_sms * 2048;
  const int U = threads <= resident ? 1 : threads <= 2 * resident ? 2 : 4;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((threads + 256LL * U - 1) / (256LL * U)));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  note_launch();
  cudaError_t e = cudaSuccess;
  if (U == 1) {
    SPMX_GROUP_SWITCH(group, (e = cudaLaunchKernelEx(&cfg, csc_naive_kernel<G, 1>, a, y)));
  } else if (U == 2) {
    SPMX_GROUP_SWITCH(group, (e = cudaLaunchKernelEx(&cfg, csc_naive_kernel<G, 2>, a, y)));
  } else {
    SPMX_GROUP_SWITCH(group, (e = cudaLaunchKernelEx(&cfg, csc_naive_kernel<G, 4>, a, y)));
  }
  return e == cudaSuccess ? 0 : -2;
}

template <class T, bool COMBINE>
static int launch_flat(const CscArgs& a, const CscScratch& s, T* y, long long col_max, int num_sms, cudaStream_t st) {
  constexpr bool NEG = sizeof(T) == 8;
  const long long words = (long long)a.m * (sizeof(T) / 4);
  const long long blocks = std::min<long long>((words + 1023) / 1024, (long long)num_sms * 4);
  note_launch();
  if (launch_pdl(zero_fill_kernel<NEG>, dim3((unsigned)std::max(1LL, blocks)), dim3(256), 0, st,
                 reinterpret_cast<float*>(y), words, a.counts + kCntBinlen, long_count(a)) != cudaSuccess)
    return -2;
  if (a.x_nnz <= 0) return 0;
  // entries per warp: enough that the grid is about one wave of warps
  const long long resident = (long long)num_sms * 64;
  int elog = 0;
  while (elog < 5 && ((long long)a.x_nnz >> elog) > resident) ++elog;
  const long long warps = ((long long)a.x_nnz + (1 << elog) - 1) >> elog;
  const int defer = col_max < 0 || col_max > kFlatCut;  // the longest column, where it is known
  note_launch(1 + defer);
  cudaError_t e = launch_pdl(csc_flat_kernel<4, T, COMBINE>, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, st, a, elog, y,
                             s.longq, s.long_cap, defer);
  if (e == cudaSuccess && defer)
    e = launch_pdl(csc_flat_long_kernel<T>, dim3((unsigned)num_sms * 4), dim3(256), 0, st, a, y,
                   (const CscLong*)s.longq, s.long_cap);
  return e == cudaSuccess ? 0 : -2;
}

int launch_csc_flat(const CscArgs& a, const CscScratch& s, float* y, long long col_max, int num_sms,
                    cudaStream_t st) {
  return launch_flat<float, false>(a, s, y, col_max, num_sms, st);
}

// products that one row may get before those of a warp are combined: they take 50
// us one by one (x of 100,000, a row of 73,000: 50 us a call either way)
constexpr int kHubProducts = 32768;

int launch_csc_flat_rows(const CscArgs& a, const CscScratch& s, double* acc, long long col_max, long long row_max,
                         int num_sms, cudaStream_t st) {
  const bool combine = a.x_nnz > kHubProducts && (row_max < 0 || row_max > kHubProducts);
  return combine ? launch_flat<double, true>(a, s, acc, col_max, num_sms, st)
                 : launch_flat<double, false>(a, s, acc, col_max, num_sms, st);
}

int launch_csc_naive(const CscArgs& a, int group, float* y, cudaStream_t st) {
  if (a.x_nnz <= 0) return 0;
  const long long threads = (long long)a.x_nnz * group;
  const unsigned grid = (unsigned)((threads + 255) / 256);
  note_launch();
  SPMX_GROUP_SWITCH(group, (csc_naive_kernel<G, 1><<<grid, 256, 0, st>>>(a, y)));
  return 0;
}

int launch_csc_naive_pairs(const CscArgs& a, const CscScratch& s, int group,
                           int* pairs_row, float* pairs_val, cudaStream_t st) {
  if (a.x_nnz <= 0) return 0;
  const long long threads = (long long)a.x_nnz * group;
  const unsigned grid = (unsigned)((threads + 255) / 256);
  note_launch();
  SPMX_GROUP_SWITCH(group, (csc_naive_pairs_kernel<G><<<grid, 256, 0, st>>>(a, s, pairs_row, pairs_val)));
  return 0;
}

}  // namespace spmx

namespace spmx {
int csc_lb_blocks_per_sm() {
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &b, csc_lb_kernel<kCscLbNT, kCscLbVT, false>, kCscLbNT, 0) != cudaSuccess) {
    cudaGetLastError();
    return 2;
  }
  return b > 0 ? b : 1;
}
}  // namespace spmx
