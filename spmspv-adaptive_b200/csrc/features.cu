// Matrix / vector feature extraction on the device and small utility kernels.
//
// Matrix features restate computeMatFeture_serial (H:2275-2335) and the
// parallel stdRow of extractMatFeatureParallel (H:921-976, whose mean is
// truncated to int, H:929): max/min row length, mean, relative range,
// standard deviation, normalised row-length entropy ("edge equality") and the
// Gini coefficient of sorted row lengths.  The Gini sums are formed exactly
// from a row-length histogram (no sort, no float accumulation).
//
// Vector features restate computeVecFeture_serial (H:2338-2361) and
// computeBinlenVer2 (H:2703-2723) without copying colptr to the host.
#include "kernels.h"
#include "feat.h"
#include "common.cuh"

namespace spmx {

// acc layout (doubles): [0] sum (d-avg)^2, [1] sum (d-avg_int)^2, [2] entropy
// ints (separate array): [0] max, [1] min_inv (INT_MAX-min), [2] zero rows
__global__ void mat_features_kernel(int m, const int* __restrict__ rowptr,
                                    double nnz, double avg, double avg_int,
                                    double* acc, int* iacc) {
  double s0 = 0, s1 = 0, s2 = 0;
  int mx = 0, mn = INT_MAX, zeros = 0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += gridDim.x * blockDim.x) {
    const int d = __ldg(rowptr + r + 1) - __ldg(rowptr + r);
    const double dd = (double)d;
    s0 += (dd - avg) * (dd - avg);
    s1 += (dd - avg_int) * (dd - avg_int);
    if (d != 0) { const double p = dd / nnz; s2 += -p * log(p); }
    mx = max(mx, d);
    mn = min(mn, d);
    zeros += (d == 0);
  }
  s0 = warp_sum(s0); s1 = warp_sum(s1); s2 = warp_sum(s2);
  mx = warp_max(mx);
  int mninv = warp_max(INT_MAX - mn);
  zeros = warp_sum(zeros);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(acc + 0, s0);
    atomicAdd(acc + 1, s1);
    atomicAdd(acc + 2, s2);
    atomicMax(iacc + 0, mx);
    atomicMax(iacc + 1, mninv);
    atomicAdd(iacc + 2, zeros);
  }
}

__global__ void degree_hist_kernel(int m, const int* __restrict__ rowptr,
                                   int* __restrict__ hist) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += gridDim.x * blockDim.x) {
    const int d = __ldg(rowptr + r + 1) - __ldg(rowptr + r);
    atomicAdd(hist + d, 1);
  }
}

// sum over degree values v of v * (h_v * P_v + h_v*(h_v-1)/2): the sum of
// j * d_(j) over sorted positions j, with P_v = rows of degree < v.
__global__ void gini_sum_kernel(int maxdeg, const int* __restrict__ hist,
                                const int* __restrict__ pref,
                                unsigned long long* out) {
  unsigned long long s = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= maxdeg;
       v += gridDim.x * blockDim.x) {
    const unsigned long long h = (unsigned)__ldg(hist + v);
    if (h) {
      const unsigned long long P = (unsigned)__ldg(pref + v);
      s += (unsigned long long)v * (h * P + h * (h - 1) / 2);
    }
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// vector features: sum / max / min of the column lengths of x's keys.
// out64[0] = bin_len; out32[0] = max, out32[1] = INT_MAX - min (both max-reduced
// from zero-initialised words).
__global__ void vec_features_kernel(int x_nnz, int n, const int* __restrict__ x_key,
                                    const int* __restrict__ colptr,
                                    unsigned long long* out64, int* out32,
                                    int* err) {
  unsigned long long s = 0;
  int mx = 0, mninv = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < x_nnz;
       i += gridDim.x * blockDim.x) {
    const int k = __ldg(x_key + i);
    if ((unsigned)k >= (unsigned)n) { flag_error(err, kDevErrOob); continue; }
    const int len = __ldg(colptr + k + 1) - __ldg(colptr + k);
    s += (unsigned)len;
    mx = max(mx, len);
    mninv = max(mninv, INT_MAX - len);
  }
  s = warp_sum(s);
  mx = warp_max(mx);
  mninv = warp_max(mninv);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out64, s);
    atomicMax(out32 + 0, mx);
    atomicMax(out32 + 1, mninv);
  }
}

// ---- utility kernels -------------------------------------------------------
// The row of every nonzero of a CSR, and its column as a sort key (n for a
// column out of range).  Each CTA owns K consecutive nonzeros: the rows that
// start among them leave marks in shared memory, and a max-scan of the marks
// gives every position its row, so all traffic is coalesced whatever the row
// lengths.  16.8M nonzeros of Zipf rows: 45 us for 201 MB; one warp
// per row took 107 us for the rows alone.
template <int NT, int VT>
__global__ void __launch_bounds__(NT)
expand_rows_kernel(int m, int n, int nnz, const int* __restrict__ rowptr, const int* __restrict__ col,
                   unsigned* __restrict__ rows, unsigned* __restrict__ keys, int* err) {
  constexpr int K = NT * VT;
  static_assert(VT % 4 == 0, "vector access to the marks");
  __shared__ __align__(16) int s_mark[K];
  __shared__ int s_wtmp[NT / 32 + 1];
  __shared__ int s_lo[2];
  const int tid = threadIdx.x;
  const long long s = (long long)blockIdx.x * K;
  const int cnt = (int)min((long long)K, nnz - s);
  unsigned key[VT];
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int q = j * NT + tid;
    key[j] = q < cnt ? (unsigned)__ldg(col + s + q) : 0u;
  }
  for (int q = tid; q < K / 4; q += NT) reinterpret_cast<int4*>(s_mark)[q] = make_int4(-1, -1, -1, -1);
  // warps 0 and 1: the first row that starts at or after the chunk's first
  // position, and after its last, 32 probes per step
  if (tid < 64) {
    const long long target = s + (tid >= 32 ? cnt : 0);
    int l = 0, r = m;  // the answer is in [l, r]
    while (l < r) {
      const int span = r - l, q = l + (int)(((long long)span * (tid & 31)) >> 5);
      const unsigned below = __ballot_sync(0xffffffffu, __ldg(rowptr + q) < target);
      const int c = __popc(below);  // the probes are sorted: the first c are below
      const int nl = c ? l + (int)(((long long)span * (c - 1)) >> 5) + 1 : l;
      r = c < 32 ? l + (int)(((long long)span * c) >> 5) : r;
      l = nl;
    }
    if ((tid & 31) == 0) s_lo[tid >> 5] = l;
  }
  __syncthreads();
  const int lo = s_lo[0], hi = s_lo[1];
  for (int r = lo + tid; r < hi; r += NT) {
    const long long p = __ldg(rowptr + r) - s;
    if (p >= 0 && p < cnt) atomicMax(&s_mark[p], r);  // empty rows share a position with the row that owns it
  }
  __syncthreads();
  int v[VT];
  int run = tid == 0 ? lo - 1 : -1;  // the row open at the chunk's start
#pragma unroll
  for (int q = 0; q < VT / 4; ++q) {
    const int4 t = reinterpret_cast<const int4*>(s_mark)[tid * (VT / 4) + q];
    run = max(run, t.x); v[4 * q] = run;
    run = max(run, t.y); v[4 * q + 1] = run;
    run = max(run, t.z); v[4 * q + 2] = run;
    run = max(run, t.w); v[4 * q + 3] = run;
  }
  // inclusive max over the threads, then the previous thread's value
  const int inc = block_inclusive_max<NT>(run, s_wtmp);
  int carry = __shfl_up_sync(0xffffffffu, inc, 1);
  if ((tid & 31) == 31) s_wtmp[tid >> 5] = inc;
  __syncthreads();
  if ((tid & 31) == 0) carry = tid ? s_wtmp[(tid >> 5) - 1] : -1;
#pragma unroll
  for (int q = 0; q < VT / 4; ++q)
    reinterpret_cast<int4*>(s_mark)[tid * (VT / 4) + q] =
        make_int4(max(v[4 * q], carry), max(v[4 * q + 1], carry), max(v[4 * q + 2], carry), max(v[4 * q + 3], carry));
  __syncthreads();
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int q = j * NT + tid;
    if (q < cnt) {
      rows[s + q] = (unsigned)s_mark[q];
      if (key[j] >= (unsigned)n) flag_error(err, kDevErrOob);
      keys[s + q] = min(key[j], (unsigned)n);
    }
  }
}

__global__ void set_int_kernel(int* p, int v) { *p = v; }

static int grid_for(long long work, int nt, int cap) {
  long long g = (work + nt - 1) / nt;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

int launch_mat_features(int m, const int* rowptr, int nnz, double avg,
                        double avg_int, double* acc, int* iacc,
                        cudaStream_t st) {
  if (m <= 0) return 0;
  note_launch();
  mat_features_kernel<<<grid_for(m, 256, 148 * 8), 256, 0, st>>>(
      m, rowptr, (double)(nnz > 0 ? nnz : 1), avg, avg_int, acc, iacc);
  return 0;
}

// longest row: one atomic per CTA (mat_features_kernel's six per warp take 70 us
// for 1M rows, this 4)
__global__ void __launch_bounds__(256)
max_degree_kernel(int m, const int* __restrict__ rowptr, int* out) {
  __shared__ int s_w[8];
  int mx = 0;
  for (long long r = (long long)blockIdx.x * 256 + threadIdx.x; r < m; r += (long long)gridDim.x * 256)
    mx = max(mx, __ldg(rowptr + r + 1) - __ldg(rowptr + r));
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < 8; ++q) mx = max(mx, s_w[q]);
    atomicMax(out, mx);
  }
}

int launch_max_degree(int m, const int* rowptr, int* out, cudaStream_t st) {
  cudaMemsetAsync(out, 0, sizeof(int), st);
  if (m <= 0) return 0;
  note_launch();
  max_degree_kernel<<<grid_for(m, 256, 148 * 4), 256, 0, st>>>(m, rowptr, out);
  return 0;
}

int launch_degree_hist(int m, const int* rowptr, int* hist, cudaStream_t st) {
  if (m <= 0) return 0;
  note_launch();
  degree_hist_kernel<<<grid_for(m, 256, 148 * 8), 256, 0, st>>>(m, rowptr, hist);
  return 0;
}

int launch_gini_sum(int maxdeg, const int* hist, const int* pref,
                    unsigned long long* out, cudaStream_t st) {
  note_launch();
  gini_sum_kernel<<<grid_for(maxdeg + 1, 256, 148 * 4), 256, 0, st>>>(maxdeg, hist, pref, out);
  return 0;
}

int launch_vec_features(int x_nnz, int n, const int* x_key, const int* colptr,
                        unsigned long long* out64, int* out32, int* err,
                        cudaStream_t st) {
  if (x_nnz <= 0) return 0;
  note_launch();
  vec_features_kernel<<<grid_for(x_nnz, 256, 148 * 8), 256, 0, st>>>(
      x_nnz, n, x_key, colptr, out64, out32, err);
  return 0;
}

int launch_expand_rows(int m, int n, int nnz, const int* rowptr, const int* col, unsigned* rows, unsigned* keys,
                       int* err, cudaStream_t st) {
  if (m <= 0 || nnz <= 0) return 0;
  constexpr int NT = 256, VT = 8;
  note_launch();
  expand_rows_kernel<NT, VT><<<(unsigned)(((long long)nnz + NT * VT - 1) / (NT * VT)), NT, 0, st>>>(
      m, n, nnz, rowptr, col, rows, keys, err);
  return 0;
}

int launch_set_int(int* p, int v, cudaStream_t st) {
  note_launch();
  set_int_kernel<<<1, 1, 0, st>>>(p, v);
  return 0;
}

}  // namespace spmx
