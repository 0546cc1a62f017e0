// CSR SpMV and bitmap-gated CSR SpMSpV kernels (y = alpha * A * x).
//
// naive ("row group"): G threads per row, FP64 accumulation, shuffle reduce.
//   Replaces naive_spmv_ker / naive_spmspv_ker (DEV/naivespmv.h:13-51), which
//   is the G = 1 case.
//
// hola ("fixed nnz per CTA"): each CTA owns K = NT*VT consecutive nonzeros,
//   like hola_spmv's fixed-work blocks (DEV/holaspmv.h:2070-2220) with its
//   block-start table (DetermineBlockStarts, DEV/holaspmv.h:40-63).  The design
//   is our own: products are formed exactly in FP64 (float*float fits a
//   double), a CTA-wide FP64 prefix P[] is kept in shared memory and every row
//   inside the chunk is P[end]-P[begin], rounded once to FP32.  Rows that cross
//   chunk boundaries leave one FP64 partial per chunk; the last chunk to arrive
//   (atomic counter per row) adds the partials in chunk order and writes y, so
//   the result is deterministic and needs no zero-fill of y and no second
//   launch.
#include <algorithm>

#include "common.cuh"
#include "engine.h"
#include "kernels.h"

namespace spmx {

__device__ __forceinline__ bool bit_is_set(const int* bits, int idx) {
  unsigned w = __ldg((const unsigned*)bits + (idx >> 5));
  return (w >> (idx & 31)) & 1u;
}

// --------------------------------------------------------------------------
// naive: G lanes per row
// --------------------------------------------------------------------------
template <int G, bool GATED>
__global__ void __launch_bounds__(256)
spmv_rowgroup_kernel(int m, int n, const int* __restrict__ rowptr,
                     const int* __restrict__ col, const float* __restrict__ val,
                     const float* __restrict__ x, const int* __restrict__ bits,
                     double alpha, float* __restrict__ y, int* err) {
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int row = (int)(gid / G);
  const int g = (int)(gid % G);
  double sum = 0.0;
  if (row < m) {
    const int a = __ldg(rowptr + row), b = __ldg(rowptr + row + 1);
    int k = a + g;
#pragma unroll 4
    for (; k < b; k += G) {
      int c = __ldg(col + k);
      if ((unsigned)c >= (unsigned)n) { flag_error(err, kDevErrOob); continue; }
      if (GATED && !bit_is_set(bits, c)) continue;
      sum += (double)__ldg(val + k) * (double)__ldg(x + c);
    }
  }
  if (G > 1) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o, G);
  }
  if (row < m && g == 0) y[row] = (float)(alpha * sum);
}

// --------------------------------------------------------------------------
// hola: fixed nnz per CTA
// --------------------------------------------------------------------------

// Splits the chunks into those of short rows (no row has more than kShortRow
// nonzeros in the chunk, the row that continues from the chunk before included;
// list[0 ..)) and the others (from the back of the list): one warp per chunk.
__global__ void chunk_split_kernel(const int* __restrict__ rowptr, int nnz, int K, int nchunks,
                                   const int* __restrict__ chunk_row, int4* __restrict__ list, int* counts) {
  const int lane = threadIdx.x & 31;
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= nchunks) return;
  const int s = c * K, e = (int)min((long long)s + K, (long long)nnz);
  const int lo = __ldg(chunk_row + c), hi = __ldg(chunk_row + c + 1);
  bool is_long = lane == 0 && lo > 0 && min(__ldg(rowptr + lo), e) - s > kShortRow;
  for (int r = lo + lane; r < hi && !is_long; r += 32)
    is_long = min(__ldg(rowptr + r + 1), e) - __ldg(rowptr + r) > kShortRow;
  is_long = __any_sync(0xffffffffu, is_long);
  if (lane == 0) {
    const int at = is_long ? nchunks - 1 - atomicAdd(counts + 1, 1) : atomicAdd(counts, 1);
    list[at] = make_int4(c, lo, hi, 0);
  }
}

// chunk_row[c] = first row r with rowptr[r] >= c*K (lower bound over
// rowptr[0..m)); chunk_row[nchunks] = m.
__global__ void chunk_rows_kernel(int m, const int* __restrict__ rowptr, int K,
                                  int nchunks, int* __restrict__ chunk_row) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > nchunks) return;
  if (c == nchunks) { chunk_row[c] = m; return; }
  long long target = (long long)c * K;
  int lo = 0, hi = m;  // search in [0, m)
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (__ldg(rowptr + mid) < target) lo = mid + 1; else hi = mid;
  }
  chunk_row[c] = lo;
}

// One partial of a row that crosses chunk boundaries.  slot 1: the chunk in
// which the row starts; slot 0: a later chunk the row continues into.
template <int K>
__device__ __forceinline__ void split_row_contribute(
    int R, int c, int slot, double part, const int* __restrict__ rowptr,
    double* carry, unsigned* arrive, double alpha, float* y) {
  const int rs = __ldg(rowptr + R), re = __ldg(rowptr + R + 1);
  const int c_first = rs / K, c_last = (re - 1) / K;
  carry[2 * c + slot] = part;
  __threadfence();
  unsigned old = atomicAdd(&arrive[c_first], 1u);
  if ((int)old == c_last - c_first) {
    __threadfence();
    const volatile double* vc = carry;
    double sum = vc[2 * c_first + 1];
    for (int cc = c_first + 1; cc <= c_last; ++cc) sum += vc[2 * cc];
    y[R] = (float)(alpha * sum);
    arrive[c_first] = 0u;  // ready for the next call
  }
}

// The chunks of short rows: the products go to shared memory in FP64 (exact),
// element by element with coalesced loads, and every row is then summed by one
// thread, in column order; no scan.  Persistent CTAs: the loads of a CTA's next
// chunk are in flight while this one's rows are summed, the descriptor of the
// one after too.  WHOLE (every chunk of the matrix is short): a chunk also reads
// the up to kShortRow nonzeros past its end that its last row may have, so no row
// is split; otherwise split rows meet as in spmv_chunk_kernel.
//
// What bounds it: latency at 32 warps per SM (64 registers); L1/TEX is 68% busy,
// issue slots 53%, DRAM 52%.  5-point Laplacian 2048^2
// (21.0M nonzeros, 218 MB): 43 us (5.1 TB/s) with no check per element where the
// chunk is inside the matrix and its largest column in range, 49 with them (47
// warp instructions per 32 nonzeros), 97 by the segmented scan; one CTA per chunk
// without the loads ahead 78 us, one thread gathering for each row from staged
// columns and values 88 to 94 us.  Row sums in predicated blocks of two, four and
// eight 45 to 47 us, 512 threads per chunk 51 us, conversions to FP64 by integer
// operations 57.
template <int NT, int VT, bool GATED, bool WHOLE>
__global__ void __launch_bounds__(NT, 1024 / NT)
spmv_short_kernel(int n, int nnz, const int* __restrict__ rowptr, const int* __restrict__ col,
                  const float* __restrict__ val, const float* __restrict__ x, const int* __restrict__ bits,
                  double alpha, float* __restrict__ y, const int4* __restrict__ list, int count,
                  double* carry, unsigned* arrive, int* err) {
  constexpr int K = NT * VT;
  extern __shared__ double s_short[];  // two buffers of K + kShortRow products
  int cc[VT + 1], ra[2], rb[2];        // element VT: past the chunk's end, first warp only
  float vv[VT + 1];
  const auto desc = [&](long long i) { return i < count ? __ldg(list + i) : make_int4(-1, 0, 0, 0); };
  const auto load = [&](const int4& d) {
    if (d.x < 0) return;
    const int s = d.x * K, left = nnz - s;
    const int* const cp = col + s + threadIdx.x;
    const float* const vp = val + s + threadIdx.x;
    cc[VT] = 0;
    vv[VT] = 0.f;
    if (left >= K + kShortRow) {
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        cc[j] = __ldcs(cp + j * NT);
        vv[j] = __ldcs(vp + j * NT);
      }
      if (WHOLE && threadIdx.x < kShortRow) {
        cc[VT] = __ldcs(cp + K);
        vv[VT] = __ldcs(vp + K);
      }
    } else {
#pragma unroll
      for (int j = 0; j <= VT; ++j) {
        const int q = j * NT + threadIdx.x;
        const bool in = q < left && (j < VT || (WHOLE && threadIdx.x < kShortRow));
        cc[j] = in ? __ldcs(cp + j * NT) : 0;
        vv[j] = in ? __ldcs(vp + j * NT) : 0.f;
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int r = d.y - 1 + WHOLE + (int)threadIdx.x + q * NT;
      const bool in = r >= 0 && r < d.z;
      ra[q] = in ? __ldg(rowptr + r) : 0;
      rb[q] = in ? __ldg(rowptr + r + 1) : 0;
    }
  };
  int4 d = desc(blockIdx.x), d1 = desc((long long)blockIdx.x + gridDim.x);
  load(d);
  int buf = 0;
  for (long long i = blockIdx.x; i < count; i += gridDim.x) {
    const int4 d2 = desc(i + 2LL * gridDim.x);
    double* const s_p = s_short + buf * (K + kShortRow);
    unsigned top = 0;
#pragma unroll
    for (int j = 0; j <= VT; ++j) top = max(top, (unsigned)cc[j]);
    if (!GATED && top < (unsigned)n) {
      float xv[VT];
#pragma unroll
      for (int j = 0; j < VT; ++j) xv[j] = __ldg(x + cc[j]);
#pragma unroll
      for (int j = 0; j < VT; ++j) s_p[j * NT + threadIdx.x] = (double)vv[j] * (double)xv[j];
      if (WHOLE && threadIdx.x < kShortRow) s_p[K + threadIdx.x] = (double)vv[VT] * (double)__ldg(x + cc[VT]);
    } else {
      bool bad = false;
#pragma unroll
      for (int j = 0; j <= VT; ++j) {
        if (j == VT && threadIdx.x >= kShortRow) break;
        bool use = (unsigned)cc[j] < (unsigned)n;
        bad |= !use;
        if (GATED) use = use && bit_is_set(bits, cc[j]);
        const float xv = use ? __ldg(x + cc[j]) : 0.f;
        s_p[j * NT + threadIdx.x] = use ? (double)vv[j] * (double)xv : 0.0;
      }
      if (bad) flag_error(err, kDevErrOob);
    }
    const int c = d.x, lo = d.y, hi = d.z, s = c * K, e = (int)min((long long)s + K, (long long)nnz);
    const int a0 = ra[0], b0 = rb[0], a1 = ra[1], b1 = rb[1];
    load(d1);
    // the products are there; nobody reads the other buffer (the rows of the
    // chunk before) any more once this barrier is behind everybody
    __syncthreads();
    int q = 0;
    for (int r = lo - 1 + WHOLE + (int)threadIdx.x; r < hi; r += NT, ++q) {
      if (r < 0) continue;
      int a = q == 0 ? a0 : a1, b = q == 0 ? b0 : b1;
      if (q > 1) {
        a = __ldg(rowptr + r);
        b = __ldg(rowptr + r + 1);
      }
      // (a graph that outlives its pattern may find rows longer than the buffer)
      const int p1 = WHOLE ? min(b - s, K + kShortRow) : min(b, e) - s;
      double sum = 0.0;
      for (int p = max(a, s) - s; p < p1; ++p) sum += s_p[p];
      if (r < lo) {
        if (b > s) split_row_contribute<K>(r, c, 0, sum, rowptr, carry, arrive, alpha, y);
      } else if (b == a) {
        y[r] = 0.f;
      } else if (WHOLE || b <= e) {
        y[r] = (float)(alpha * sum);
      } else {
        split_row_contribute<K>(r, c, 1, sum, rowptr, carry, arrive, alpha, y);
      }
    }
    buf ^= 1;
    d = d1;
    d1 = d2;
  }
}

template <int NT, int VT, bool GATED>
__global__ void __launch_bounds__(NT)
spmv_chunk_kernel(int m, int n, int nnz, const int* __restrict__ rowptr,
                  const int* __restrict__ col, const float* __restrict__ val,
                  const float* __restrict__ x, const int* __restrict__ bits,
                  double alpha, float* __restrict__ y,
                  const int* __restrict__ chunk_row, const int4* __restrict__ list, double* carry,
                  unsigned* arrive, int vec_ok, int* err) {
  constexpr int K = NT * VT;
  __shared__ double sP[K];
  __shared__ double s_wtmp[NT / 32 + 1];
  __shared__ int s_tf[NT / 32 + 1];
  __shared__ unsigned s_flag[K / 32];
  const int c = list ? __ldg(list + blockIdx.x).x : (int)blockIdx.x;  // no list: every chunk
  const int s = c * K;
  const int e = min(s + K, nnz);
  const int base = s + (int)threadIdx.x * VT;

  double pr[VT];
#pragma unroll
  for (int j = 0; j < VT; ++j) pr[j] = 0.0;

  if (vec_ok && s + K <= nnz && (VT % 4) == 0) {
#pragma unroll
    for (int q = 0; q < VT / 4; ++q) {
      const int4 c4 = __ldcs(reinterpret_cast<const int4*>(col + base) + q);
      const int cc[4] = {c4.x, c4.y, c4.z, c4.w};
      bool want[4];
      bool any = false;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        bool ok = (unsigned)cc[t] < (unsigned)n;
        if (!ok) flag_error(err, kDevErrOob);
        want[t] = ok && (!GATED || bit_is_set(bits, cc[t]));
        any |= want[t];
      }
      if (!GATED || any) {
        const float4 v4 = __ldcs(reinterpret_cast<const float4*>(val + base) + q);
        const float vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int t = 0; t < 4; ++t)
          if (want[t]) pr[q * 4 + t] = (double)vv[t] * (double)__ldg(x + cc[t]);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < VT; ++j) {
      const int k = base + j;
      if (k < e) {
        const int cj = __ldg(col + k);
        if ((unsigned)cj >= (unsigned)n) { flag_error(err, kDevErrOob); continue; }
        if (GATED && !bit_is_set(bits, cj)) continue;
        pr[j] = (double)__ldg(val + k) * (double)__ldg(x + cj);
      }
    }
  }

  // row-start flags of the rows that begin inside the chunk
  const int lo = __ldg(chunk_row + c), hi = __ldg(chunk_row + c + 1);
  for (int i = threadIdx.x; i < K / 32; i += NT) s_flag[i] = 0u;
  __syncthreads();
  for (int r = lo + (int)threadIdx.x; r < hi; r += NT) {
    const int p = __ldg(rowptr + r) - s;
    if ((unsigned)p < (unsigned)(e - s)) atomicOr(&s_flag[p >> 5], 1u << (p & 31));
  }
  __syncthreads();
  // segmented scan: every row is summed from its own products only (no
  // differences of running sums), so all-zero rows stay exactly zero
  unsigned myf;
  {
    const int bit0 = threadIdx.x * VT;
    const unsigned w = s_flag[bit0 >> 5];
    myf = (w >> (bit0 & 31)) & ((VT >= 32) ? 0xffffffffu : ((1u << VT) - 1u));
  }
  double run = 0.0;
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    run = ((myf >> j) & 1u) ? pr[j] : run + pr[j];
    pr[j] = run;
  }
  const double carry_in = block_exclusive_segscan<NT>(myf != 0u, run, s_tf, s_wtmp);
  const int first = myf ? __ffs(myf) - 1 : VT;
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    if (j < first) pr[j] += carry_in;
    sP[threadIdx.x * VT + j] = pr[j];
  }
  __syncthreads();

  for (int r = lo + (int)threadIdx.x; r < hi; r += NT) {
    const int a = __ldg(rowptr + r), b = __ldg(rowptr + r + 1);
    if (b == a) {
      y[r] = 0.f;
    } else if (b <= e) {
      y[r] = (float)(alpha * sP[max(b - 1 - s, 0)]);
    } else {
      split_row_contribute<K>(r, c, 1, sP[e - 1 - s], rowptr, carry, arrive, alpha, y);
    }
  }
  if (threadIdx.x == 0 && lo > 0) {
    const int R = lo - 1;
    const int endR = __ldg(rowptr + lo);
    if (endR > s) {
      const int stop = min(endR, e);
      split_row_contribute<K>(R, c, 0, sP[stop - 1 - s], rowptr, carry, arrive, alpha, y);
    }
  }
}

// --------------------------------------------------------------------------
// host launchers
// --------------------------------------------------------------------------
int launch_spmv_naive(const SpmvArgs& a, int group, cudaStream_t st) {
  if (a.m <= 0) return 0;
  const int NT = 256;
#define SPMX_NAIVE_CASE(G)                                                        \
  case G: {                                                                      \
    long long threads = (long long)a.m * G;                                      \
    unsigned grid = (unsigned)((threads + NT - 1) / NT);                         \
    if (a.bits)                                                                  \
      spmv_rowgroup_kernel<G, true><<<grid, NT, 0, st>>>(                        \
          a.m, a.n, a.rowptr, a.col, a.val, a.x, a.bits, a.alpha, a.y, a.err);   \
    else                                                                         \
      spmv_rowgroup_kernel<G, false><<<grid, NT, 0, st>>>(                       \
          a.m, a.n, a.rowptr, a.col, a.val, a.x, a.bits, a.alpha, a.y, a.err);   \
    break;                                                                       \
  }
  note_launch();
  switch (group) {
    SPMX_NAIVE_CASE(1)
    SPMX_NAIVE_CASE(2)
    SPMX_NAIVE_CASE(4)
    SPMX_NAIVE_CASE(8)
    SPMX_NAIVE_CASE(16)
    SPMX_NAIVE_CASE(32)
    default: return -1;
  }
#undef SPMX_NAIVE_CASE
  return 0;
}

int hola_chunk_nnz(int vt) { return 256 * vt; }

int launch_chunk_rows(int m, int nnz, const int* rowptr, int K, int nchunks, int* chunk_row,
                      int4* list, int* counts, cudaStream_t st) {
  int threads = nchunks + 1;
  note_launch();
  chunk_rows_kernel<<<(threads + 255) / 256, 256, 0, st>>>(m, rowptr, K, nchunks,
                                                         chunk_row);
  if (nchunks > 0 && list) {
    note_launch();
    chunk_split_kernel<<<(nchunks + 7) / 8, 256, 0, st>>>(rowptr, nnz, K, nchunks, chunk_row, list, counts);
  }
  return 0;
}

int launch_spmv_hola(const SpmvArgs& a, const HolaTables& t, cudaStream_t st) {
  if (a.m <= 0) return 0;
  if (a.nnz == 0 || t.nchunks == 0) {
    cudaMemsetAsync(a.y, 0, sizeof(float) * (size_t)a.m, st);
    return 0;
  }
  const int vec_ok = (((uintptr_t)a.col | (uintptr_t)a.val) & 15u) == 0;
  constexpr int NT = 256;
  // the chunks of short rows by their own kernel, the others by the scan; a
  // matrix with few short chunks goes through the scan whole
  const int nlong = t.nchunks - t.n_short;
  const int4* list = t.n_short > 0 ? t.list + t.n_short : nullptr;
  cudaError_t e = cudaSuccess;
#define SPMX_HOLA_CASE(VT)                                                       \
  case VT: {                                                                     \
    if (t.n_short > 0) {                                                         \
      auto kernel = nlong == 0 ? (a.bits ? spmv_short_kernel<NT, VT, true, true> : spmv_short_kernel<NT, VT, false, true>) \
                               : (a.bits ? spmv_short_kernel<NT, VT, true, false> : spmv_short_kernel<NT, VT, false, false>); \
      constexpr int smem = 16 * (NT * VT + kShortRow);                           \
      e = kernel_smem_limit((const void*)kernel, smem);                          \
      const int cap = 148 * std::min(1024 / NT, (227 << 10) / (smem + 1024));    \
      const int rounds = (t.n_short + cap - 1) / cap;                            \
      if (e == cudaSuccess)                                                      \
        kernel<<<(t.n_short + rounds - 1) / rounds, NT, smem, st>>>(             \
            a.n, a.nnz, a.rowptr, a.col, a.val, a.x, a.bits, a.alpha, a.y, t.list, t.n_short, t.carry, \
            t.arrive, a.err);                                                    \
    }                                                                            \
    if (nlong > 0) {                                         \
      auto kernel = a.bits ? spmv_chunk_kernel<NT, VT, true> : spmv_chunk_kernel<NT, VT, false>; \
      e = launch_l2_window(kernel, dim3(nlong), dim3(NT), 0, st, a.x, 4 * (size_t)a.n, a.m, a.n, a.nnz, \
                           a.rowptr, a.col, a.val, a.x, a.bits, a.alpha, a.y, (const int*)t.chunk_row, list, \
                           t.carry, t.arrive, vec_ok, a.err);                    \
    }                                                                            \
    break;                                                                       \
  }
  note_launch((t.n_short > 0) + (nlong > 0));
  switch (t.vt) {
    SPMX_HOLA_CASE(4)
    SPMX_HOLA_CASE(8)
    SPMX_HOLA_CASE(16)
    default: return -1;
  }
#undef SPMX_HOLA_CASE
  return e == cudaSuccess ? 0 : -2;
}

}  // namespace spmx
