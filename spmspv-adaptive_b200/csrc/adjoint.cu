// Adjoint of y = A x for the FP32 semiring (no reference counterpart: the
// reference has no differentiation).  For a loss L(y):
//   dx    = A^T dy                  (the transpose product)
//   dvals = dy[row_k] * x[col_k]    (the gradient on the nonzero pattern)
//
// dense dy, handle with a CSC: dx is the row-ordered SpMV of the transpose
//   (the CSC read as the CSR of A^T, dy as its x: a gather, no atomics) and
//   dvals a streaming pass over the CSR.  Both are deterministic.
// dense dy, CSR only: ONE pass over the CSR, fixed 2048 nonzeros per CTA
//   (the Hola chunks): every nonzero writes its dvals entry and adds
//   val*dy[row] into dx[col] with an FP32 atomic, so the matrix is streamed
//   once for both gradients.  The row of each nonzero comes from a max-scan
//   of row-start marks in shared memory (no per-element search).
// sparse dy (dy_key, dy_val): only the rows in dy's support contribute, so a
//   group of lanes per dy entry walks that row (the CSR of A is the CSC of
//   A^T: this is the CSC SpMSpV of the transpose) after dx and dvals are
//   zeroed.
#include <algorithm>

#include "common.cuh"
#include "engine.h"
#include "kernels.h"

namespace spmx {

__device__ __forceinline__ bool gate_shut(const DevGate& g) {
  return g.count && (__ldg(g.count) < g.limit) != g.below;
}

template <int NT, int VT>
__global__ void __launch_bounds__(NT)
spmv_backward_kernel(int m, int n, int nnz, const int* __restrict__ rowptr,
                     const int* __restrict__ col, const float* __restrict__ val,
                     const float* __restrict__ x, const float* __restrict__ dy,
                     const int* __restrict__ chunk_row, const int4* __restrict__ list, float* __restrict__ dx,
                     float* __restrict__ dvals, DevGate gate, int* err) {
  if (gate_shut(gate)) return;
  constexpr int K = NT * VT;
  __shared__ int s_mark[K];
  __shared__ int s_incl[NT];
  __shared__ int s_wtmp[NT / 32 + 1];
  const int c = list ? __ldg(list + blockIdx.x).x : (int)blockIdx.x;  // no list: every chunk
  const int s = c * K;
  const int e = min(s + K, nnz);
  const int lo = __ldg(chunk_row + c), hi = __ldg(chunk_row + c + 1);
  for (int q = threadIdx.x; q < K; q += NT) s_mark[q] = -1;
  __syncthreads();
  // rows that start inside the chunk mark their first element; several empty
  // rows at one position leave the largest index, the non-empty one
  for (int r = lo + (int)threadIdx.x; r < hi; r += NT) {
    const int p = __ldg(rowptr + r) - s;
    if ((unsigned)p < (unsigned)(e - s)) atomicMax(&s_mark[p], r);
  }
  __syncthreads();
  int loc[VT];
  int run = INT_MIN;
  const int head = lo - 1;  // the row open at the chunk start (if any)
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int q = threadIdx.x * VT + j;
    int v = s_mark[q];
    if (q == 0) v = max(v, head);
    run = max(run, v);
    loc[j] = run;
  }
  const int inc = block_inclusive_max<NT>(run, s_wtmp);
  s_incl[threadIdx.x] = inc;
  __syncthreads();
  const int carry = threadIdx.x ? s_incl[threadIdx.x - 1] : INT_MIN;
#pragma unroll
  for (int j = 0; j < VT; ++j) s_mark[threadIdx.x * VT + j] = max(loc[j], carry);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int q = j * NT + threadIdx.x;  // coalesced over the chunk
    const int k = s + q;
    if (k < e) {
      const int r = s_mark[q];
      const int cc = __ldg(col + k);
      if ((unsigned)r >= (unsigned)m || (unsigned)cc >= (unsigned)n) {
        flag_error(err, kDevErrOob);
        continue;
      }
      const float g = __ldg(dy + r);
      if (dvals) dvals[k] = g * __ldg(x + cc);
      if (dx && g != 0.0f) atomicAdd(dx + cc, __ldg(val + k) * g);
    }
  }
}

// The same for the chunks of short rows: one thread per row leaves dy of its row
// beside every nonzero, no scan.  Persistent CTAs: while a chunk is worked, the
// columns and values of the next are copied into the other shared buffer
// (cp.async), and the bounds and dy of its rows are on their way into registers.
//
// What bounds it: the latency of the x gathers beside the 21M reductions into dx
// (long-scoreboard stalls 10.9 cycles per instruction; L1/TEX 68%, DRAM 56%, L2 44%).  5-point
// Laplacian 2048^2 (21.0M nonzeros): 80 us against 136 with the rows found by a
// scan of marks; one thread walking each row, so that the reductions of
// neighbouring lanes fall on neighbouring entries, took 89 (chunk by chunk) and
// 92 us (persistent).  512 threads per chunk in three CTAs 80 us, in four 83, 256 in
// four 84 (86 with a range check per element); dvals alone 57, 48 and 53 us, so
// four there.
template <int NT, int VT>
struct BackwardChunk {
  static constexpr int K = NT * VT;
  int col[K];
  float val[K];
  float g[K];
};

// every nonzero of a staged chunk: its dvals entry and its share of dx
template <int NT, int VT, bool FULL, bool DX, bool DV>
__device__ __forceinline__ void backward_elements(const BackwardChunk<NT, VT>& t, int n, int cnt,
                                                  const float* __restrict__ x, float* __restrict__ dx,
                                                  float* __restrict__ dvals, int* err) {
  const int e0 = threadIdx.x;
  int c[VT];
  float xv[VT];
  if (FULL) {  // every column in range: no check per element
    unsigned top = 0;
#pragma unroll
    for (int j = 0; j < VT; ++j) {
      c[j] = t.col[e0 + j * NT];
      top = max(top, (unsigned)c[j]);
    }
    if (top < (unsigned)n) {
      if (DV) {
#pragma unroll
        for (int j = 0; j < VT; ++j) xv[j] = __ldg(x + c[j]);
      }
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        const float g = t.g[e0 + j * NT];
        if (DX && g != 0.0f) atomicAdd(dx + c[j], t.val[e0 + j * NT] * g);
        if (DV) __stcs(dvals + e0 + j * NT, g * xv[j]);
      }
      return;
    }
  }
  bool bad = false;
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const bool in = FULL || e0 + j * NT < cnt;
    c[j] = in ? t.col[e0 + j * NT] : 0;
    const bool ok = (unsigned)c[j] < (unsigned)n;
    bad |= !ok;
    if (!ok || !in) c[j] = -1;
    xv[j] = DV && c[j] >= 0 ? __ldg(x + c[j]) : 0.f;
  }
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    if (c[j] < 0) continue;
    const float g = t.g[e0 + j * NT];
    if (DX && g != 0.0f) atomicAdd(dx + c[j], t.val[e0 + j * NT] * g);
    if (DV) __stcs(dvals + e0 + j * NT, g * xv[j]);
  }
  if (bad) flag_error(err, kDevErrOob);
}

template <int NT, int VT, int CTAS, bool DX, bool DV>
__global__ void __launch_bounds__(NT, CTAS)
spmv_backward_short_kernel(int n, int nnz, const int* __restrict__ rowptr, const int* __restrict__ col,
                           const float* __restrict__ val, const float* __restrict__ x,
                           const float* __restrict__ dy, const int4* __restrict__ list, int count,
                           float* __restrict__ dx, float* __restrict__ dvals, int vec_ok, DevGate gate,
                           int* err) {
  if (gate_shut(gate)) return;
  constexpr int K = NT * VT;
  extern __shared__ __align__(16) unsigned char s_raw[];
  BackwardChunk<NT, VT>* const sh = reinterpret_cast<BackwardChunk<NT, VT>*>(s_raw);  // two of them
  int ra[2], rb[2];
  float rg[2];
  const auto desc = [&](long long i) { return i < count ? __ldg(list + i) : make_int4(-1, 0, 0, 0); };
  const auto load = [&](const int4& d, int into) {
    if (d.x >= 0) {
      const int s = d.x * K, cnt = (int)min((long long)K, (long long)nnz - s);
      if (vec_ok && cnt == K) {
        for (int q = threadIdx.x; q < K / 4; q += NT) {
          cp_async16(sh[into].col + 4 * q, col + s + 4 * q);
          if (DX) cp_async16(sh[into].val + 4 * q, val + s + 4 * q);
        }
      } else {
        for (int q = threadIdx.x; q < cnt; q += NT) {
          cp_async4(sh[into].col + q, col + s + q);
          if (DX) cp_async4(sh[into].val + q, val + s + q);
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int r = d.y - 1 + (int)threadIdx.x + q * NT;
        const bool in = r >= 0 && r < d.z;
        ra[q] = in ? __ldg(rowptr + r) : 0;
        rb[q] = in ? __ldg(rowptr + r + 1) : 0;
        rg[q] = in ? __ldg(dy + r) : 0.f;
      }
    }
    cp_async_commit();
  };
  int4 d = desc(blockIdx.x), d1 = desc((long long)blockIdx.x + gridDim.x);
  load(d, 0);
  int buf = 0;
  for (long long i = blockIdx.x; i < count; i += gridDim.x) {
    const int4 d2 = desc(i + 2LL * gridDim.x);
    BackwardChunk<NT, VT>& t = sh[buf];
    const int s = d.x * K, cnt = (int)min((long long)K, (long long)nnz - s);
    int q = 0;
    for (int r = d.y - 1 + (int)threadIdx.x; r < d.z; r += NT, ++q) {
      if (r < 0) continue;
      int a = q == 0 ? ra[0] : ra[1], b = q == 0 ? rb[0] : rb[1];
      float g = q == 0 ? rg[0] : rg[1];
      if (q > 1) {
        a = __ldg(rowptr + r);
        b = __ldg(rowptr + r + 1);
        g = __ldg(dy + r);
      }
      const int p1 = min(b - s, cnt);
      for (int p = max(a - s, 0); p < p1; ++p) t.g[p] = g;
    }
    cp_async_wait<0>();
    __syncthreads();  // the chunk is complete, and nobody reads the other one any more
    load(d1, buf ^ 1);
    if (cnt == K) backward_elements<NT, VT, true, DX, DV>(t, n, K, x, dx, DV ? dvals + s : nullptr, err);
    else backward_elements<NT, VT, false, DX, DV>(t, n, cnt, x, dx, DV ? dvals + s : nullptr, err);
    buf ^= 1;
    d = d1;
    d1 = d2;
  }
}

// Dense-dy adjoint on a handle with a CSC, one launch: even CTAs compute dx
// (G1 lanes per column of the CSC, a gather of dy with FP64 sums, every dx
// entry written once), odd CTAs write dvals (G2 lanes per row of the CSR).
// The two halves stream different arrays side by side; neither uses atomics.
template <int G1, int G2>
__global__ void __launch_bounds__(256)
adjoint_csc_kernel(int m, int n, const int* __restrict__ rowptr, const int* __restrict__ col,
                   const int* __restrict__ colptr, const int* __restrict__ crow,
                   const float* __restrict__ cval, const float* __restrict__ x,
                   const float* __restrict__ dy, float* __restrict__ dx,
                   float* __restrict__ dvals, DevGate gate, int* err) {
  if (gate_shut(gate)) return;
  const long long gid = (long long)(blockIdx.x >> 1) * blockDim.x + threadIdx.x;
  if ((blockIdx.x & 1) == 0) {
    if (!dx || gid / G1 >= ((long long)n + 31) / 32 * 32) return;  // whole warps past the end
    const long long j = gid / G1;
    const int g = (int)(gid % G1);
    double sum = 0.0;
    if (j < n) {
      const int a = __ldg(colptr + j), b = __ldg(colptr + j + 1);
      for (int k = a + g; k < b; k += G1) {
        const int r = __ldg(crow + k);
        if ((unsigned)r >= (unsigned)m) {
          flag_error(err, kDevErrOob);
          continue;
        }
        sum += (double)__ldg(cval + k) * (double)__ldg(dy + r);
      }
    }
    if (G1 > 1) {
#pragma unroll
      for (int o = G1 / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o, G1);
    }
    if (j < n && g == 0) dx[j] = (float)sum;
  } else {
    const long long row = gid / G2;
    if (!dvals || row >= m) return;
    const int g = (int)(gid % G2);
    const float d = __ldg(dy + row);
    const int a = __ldg(rowptr + row), b = __ldg(rowptr + row + 1);
    for (int k = a + g; k < b; k += G2) {
      const int c = __ldg(col + k);
      if ((unsigned)c >= (unsigned)n) {
        flag_error(err, kDevErrOob);
        dvals[k] = 0.f;
        continue;
      }
      dvals[k] = d * __ldg(x + c);
    }
  }
}

// G lanes per dy entry; with a gate the entry count is on the device
template <int G>
__global__ void __launch_bounds__(256)
spmv_backward_sparse_kernel(int m, int n, const int* __restrict__ rowptr,
                            const int* __restrict__ col, const float* __restrict__ val,
                            const float* __restrict__ x, int dy_nnz,
                            const int* __restrict__ dy_key, const float* __restrict__ dy_val,
                            float* __restrict__ dx, float* __restrict__ dvals, DevGate gate, int* err) {
  if (gate.count) {
    dy_nnz = __ldg(gate.count);
    if ((dy_nnz < gate.limit) != gate.below) return;
  }
  const long long step = (long long)gridDim.x * blockDim.x / G;
  const int g = (int)(threadIdx.x % G);
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G; i < dy_nnz; i += step) {
    const int r = __ldg(dy_key + i);
    if ((unsigned)r >= (unsigned)m) {
      if (g == 0) flag_error(err, kDevErrOob);
      continue;
    }
    const float d = __ldg(dy_val + i);
    const int a = __ldg(rowptr + r), b = __ldg(rowptr + r + 1);
    for (int k = a + g; k < b; k += G) {
      const int cc = __ldg(col + k);
      if ((unsigned)cc >= (unsigned)n) { flag_error(err, kDevErrOob); continue; }
      if (dvals) dvals[k] = d * __ldg(x + cc);
      if (dx) atomicAdd(dx + cc, __ldg(val + k) * d);
    }
  }
}

__device__ __forceinline__ void clear_floats(float* p, long long len) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
  const long long head = min(len, (long long)((16 - ((uintptr_t)p & 15)) & 15) / 4);  // up to the 16-byte boundary
  const long long quads = (len - head) >> 2;
  float4* p4 = reinterpret_cast<float4*>(p + head);
  for (long long i = tid; i < quads; i += nt) p4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long long i = tid; i < head; i += nt) p[i] = 0.f;
  for (long long i = head + 4 * quads + tid; i < len; i += nt) p[i] = 0.f;
}

__global__ void __launch_bounds__(256)
backward_clear_kernel(int n, int nnz, float* dx, float* dvals, int dx_always, DevGate gate) {
  const bool shut = gate_shut(gate);
  if (dx && (dx_always || !shut)) clear_floats(dx, n);
  if (dvals && !shut) clear_floats(dvals, nnz);
}

int launch_backward_clear(int n, int nnz, float* dx, float* dvals, bool dx_always, int num_sms, DevGate gate,
                          cudaStream_t st) {
  if (!dx && !dvals) return 0;
  note_launch();
  backward_clear_kernel<<<num_sms * 8, 256, 0, st>>>(n, nnz, dx, dvals, dx_always, gate);
  return 0;
}

int launch_spmv_backward(int m, int n, int nnz, const int* rowptr, const int* col,
                         const float* val, const float* x, const float* dy,
                         const HolaTables& t, float* dx, float* dvals, int* err,
                         DevGate gate, cudaStream_t st) {
  // the kernels of short rows have a form for dx, for dvals and for both
  if (nnz <= 0 || t.nchunks == 0 || (!dx && !dvals)) return 0;
  if (t.K != 2048) return -1;  // the backward pass uses 256 x 8 chunks
  const int nlong = t.nchunks - t.n_short;
  note_launch((t.n_short > 0) + (nlong > 0));
  if (t.n_short > 0) {
    constexpr int NT = 512, VT = 4;
    constexpr int smem = 2 * sizeof(BackwardChunk<NT, VT>);
    const auto kernel = !dvals ? spmv_backward_short_kernel<NT, VT, 3, true, false>
                        : dx   ? spmv_backward_short_kernel<NT, VT, 3, true, true>
                               : spmv_backward_short_kernel<NT, VT, 4, false, true>;
    if (kernel_smem_limit((const void*)kernel, smem) != cudaSuccess) return -2;
    const int cap = 148 * (dx ? 3 : 4);
    const int rounds = (t.n_short + cap - 1) / cap;
    kernel<<<(t.n_short + rounds - 1) / rounds, NT, smem, st>>>(
        n, nnz, rowptr, col, val, x, dy, t.list, t.n_short, dx, dvals,
        (((uintptr_t)col | (uintptr_t)val) & 15u) == 0, gate, err);
  }
  if (nlong > 0)
    spmv_backward_kernel<256, 8><<<nlong, 256, 0, st>>>(m, n, nnz, rowptr, col, val, x, dy, t.chunk_row,
                                                        t.n_short > 0 ? t.list + t.n_short : nullptr, dx, dvals, gate,
                                                 err);
  return 0;
}

template <int G1>
static void adjoint_csc_g2(int g2, unsigned grid, cudaStream_t st, int m, int n, const int* rowptr,
                           const int* col, const int* colptr, const int* crow, const float* cval,
                           const float* x, const float* dy, float* dx, float* dvals, DevGate gate, int* err) {
  switch (g2) {
    case 1: adjoint_csc_kernel<G1, 1><<<grid, 256, 0, st>>>(m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
    case 2: adjoint_csc_kernel<G1, 2><<<grid, 256, 0, st>>>(m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
    case 4: adjoint_csc_kernel<G1, 4><<<grid, 256, 0, st>>>(m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
    default: adjoint_csc_kernel<G1, 8><<<grid, 256, 0, st>>>(m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
  }
}

int launch_spmv_backward_csc(int m, int n, const int* rowptr, const int* col, const int* colptr,
                             const int* crow, const float* cval, const float* x, const float* dy,
                             int g1, int g2, float* dx, float* dvals, int* err, DevGate gate,
                             cudaStream_t st) {
  if ((!dx || n <= 0) && (!dvals || m <= 0)) return 0;
  const long long t1 = dx ? ((long long)n + 31) / 32 * 32 * g1 : 0;
  const long long t2 = dvals ? (long long)m * g2 : 0;
  const long long half = (std::max(t1, t2) + 255) / 256;
  const unsigned grid = (unsigned)(2 * half);
  note_launch();
  switch (g1) {
    case 1: adjoint_csc_g2<1>(g2, grid, st, m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
    case 2: adjoint_csc_g2<2>(g2, grid, st, m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
    case 4: adjoint_csc_g2<4>(g2, grid, st, m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
    case 8: adjoint_csc_g2<8>(g2, grid, st, m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
    case 16: adjoint_csc_g2<16>(g2, grid, st, m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
    default: adjoint_csc_g2<32>(g2, grid, st, m, n, rowptr, col, colptr, crow, cval, x, dy, dx, dvals, gate, err); break;
  }
  return 0;
}

static void sparse_backward(int group, unsigned grid, cudaStream_t st, int m, int n, const int* rowptr,
                            const int* col, const float* val, const float* x, int dy_nnz, const int* dy_key,
                            const float* dy_val, float* dx, float* dvals, DevGate gate, int* err) {
#define SPMX_SPARSE_BACKWARD(G) \
  spmv_backward_sparse_kernel<G><<<grid, 256, 0, st>>>(m, n, rowptr, col, val, x, dy_nnz, dy_key, dy_val, dx, dvals, gate, err)
  note_launch();
  switch (group) {
    case 1: SPMX_SPARSE_BACKWARD(1); break;
    case 2: SPMX_SPARSE_BACKWARD(2); break;
    case 4: SPMX_SPARSE_BACKWARD(4); break;
    case 8: SPMX_SPARSE_BACKWARD(8); break;
    case 16: SPMX_SPARSE_BACKWARD(16); break;
    default: SPMX_SPARSE_BACKWARD(32); break;
  }
#undef SPMX_SPARSE_BACKWARD
}

int launch_spmv_backward_sparse(int m, int n, const int* rowptr, const int* col,
                                const float* val, const float* x, int dy_nnz,
                                const int* dy_key, const float* dy_val, int group,
                                float* dx, float* dvals, int* err, cudaStream_t st) {
  if (dy_nnz <= 0) return 0;
  const unsigned grid = (unsigned)(((long long)dy_nnz * group + 255) / 256);
  sparse_backward(group, grid, st, m, n, rowptr, col, val, x, dy_nnz, dy_key, dy_val, dx, dvals, DevGate{}, err);
  return 0;
}

int launch_spmv_backward_gated(int m, int n, const int* rowptr, const int* col, const float* val, const float* x,
                               const int* dy_key, const float* dy_val, int group, float* dx, float* dvals,
                               int num_sms, int* err, DevGate gate, cudaStream_t st) {
  const long long want = ((long long)gate.limit * group + 255) / 256;
  const unsigned grid = (unsigned)std::max(1LL, std::min<long long>(want, (long long)num_sms * 8));
  sparse_backward(group, grid, st, m, n, rowptr, col, val, x, 0, dy_key, dy_val, dx, dvals, gate, err);
  return 0;
}

}  // namespace spmx
