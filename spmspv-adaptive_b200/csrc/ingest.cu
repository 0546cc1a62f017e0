// Device COO -> CSR for a handle: the GPU side of matrix ingestion.  It
// replaces the host std::sort by (row, col) after ReadMTX
// (hice-spmspv/hice/la/include/spmspv/mtx.hpp:335-360) and the cuSPARSE
// coo2csr of the reference's drivers.
//
// 1. coo_check_kernel: range check of every index, and whether the entries
//    are already in (row, col) order, or at least in non-decreasing column
//    order (a column-major file such as a SuiteSparse export).
// 2. one stable LSD radix sort (sort.cu) by (row, col), over the row bits alone
//    when the columns are already non-decreasing, none when the input is
//    already in (row, col) order.  Stability keeps duplicates in input order.
// 3. sorted_bounds_kernel (sort.cu): the row pointers from the sorted rows;
//    every entry is written once, empty rows included, with no atomics and no
//    search.
#include <algorithm>

#include "common.cuh"
#include "engine.h"
#include "sort.h"

namespace spmx {
namespace {

constexpr int kIngestNT = 256;

__global__ void __launch_bounds__(kIngestNT)
coo_check_kernel(int nnz, int m, int n, const int* __restrict__ row,
                 const int* __restrict__ col, int* __restrict__ flags) {
  int oob = 0, unsorted = 0, col_desc = 0;
  constexpr int U = 4;  // entries in flight per thread
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < nnz; b += U * step) {
    int r[U], c[U], rp[U], cp[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = min(b + u * step, (long long)nnz - 1), p = max(i - 1, 0LL);
      r[u] = __ldg(row + i);
      c[u] = __ldg(col + i);
      rp[u] = __ldg(row + p);
      cp[u] = __ldg(col + p);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      oob |= (unsigned)r[u] >= (unsigned)m || (unsigned)c[u] >= (unsigned)n;
      unsorted |= rp[u] > r[u] || (rp[u] == r[u] && cp[u] > c[u]);
      col_desc |= cp[u] > c[u];
    }
  }
  oob = __syncthreads_or(oob);
  unsorted = __syncthreads_or(unsorted);
  col_desc = __syncthreads_or(col_desc);
  if (threadIdx.x == 0) {
    if (oob) atomicOr(flags + 0, 1);
    if (unsorted) atomicOr(flags + 1, 1);
    if (col_desc) atomicOr(flags + 2, 1);
  }
}

int ingest_grid(long long work) {
  const long long g = (work + kIngestNT - 1) / kIngestNT;
  return (int)std::max<long long>(1, std::min<long long>(g, 148LL * 16));
}

int key_bits(int extent) {
  int b = 1;
  while (b < 31 && (1LL << b) < extent) ++b;
  return b;
}

}  // namespace
}  // namespace spmx

using namespace spmx;

// What the handle keeps of the matrix in its own CSR arrays, about to be written
// or just written, is not that matrix's any more: features, chunk and hub tables,
// and a CSC that spmx_to_csc derived from it.
static void forget_csr(spmx_handle_t h) {
  h->has_csr = false;
  h->mat_feat_ready = false;
  h->std_row_ready = false;
  h->batch_chunk_ready = false;
  h->ms_hubs_ready = false;
  h->hola_rowptr = nullptr;
  if (h->has_csc && h->csc_colptr == h->own_colptr) h->has_csc = false;
}

extern "C" int spmx_input_coo(spmx_handle_t h, int nnz, const int* row, const int* col,
                              const float* val) {
  SPMX_CHECK_HANDLE(h);
  if (nnz != h->nnz) return set_error(SPMX_ERR_INVALID_VALUE, "nnz differs from the handle's nnz");
  if (nnz > 0 && (!row || !col)) return set_error(SPMX_ERR_INVALID_VALUE, "NULL COO array");
  const int m = h->m, n = h->n;
  cudaStream_t st = h->stream;
  const size_t b = 4 * (size_t)std::max(nnz, 1);

  // 1. range and order check (synchronous: the result picks the sort passes);
  // the feature accumulators hold the three flags
  SPMX_CUDA(cudaMemsetAsync(h->d_iacc, 0, 4 * sizeof(int), st));
  if (nnz > 0) {
    note_launch();
    coo_check_kernel<<<ingest_grid(nnz), kIngestNT, 0, st>>>(nnz, m, n, row, col, h->d_iacc);
    SPMX_TRY(launch_ok("coo check"));
  }
  SPMX_CUDA(cudaMemcpyAsync(h->h_pinned, h->d_iacc, 3 * sizeof(int), cudaMemcpyDeviceToHost, st));
  SPMX_CUDA(cudaStreamSynchronize(st));
  const int unsorted = h->h_pinned[1], col_desc = h->h_pinned[2];
  if (h->h_pinned[0]) return set_error(SPMX_ERR_INVALID_VALUE, "COO index out of range");

  // 2. the new CSR, in the handle's own arrays (its sizes never change); all
  // memory is there before the first of them is written.  The radix passes
  // alternate between two buffer sets; the pass count is known here, so the
  // set the last pass writes is the column / value arrays themselves.
  char* scratch = nullptr;
  const size_t al = (b + 255) & ~(size_t)255;
  if (unsorted)
    SPMX_TRY(scratch_alloc((void**)&scratch, al * (val ? 4 : 3) + radix_scratch_bytes(nnz), st, "coo sort"));
  int *nrp = h->own_csr_rowptr, *ncol = h->own_csr_col;
  float* nval = val ? h->own_csr_val : nullptr;
  int rc = SPMX_SUCCESS;
  // a caller's work on another stream may still read the previous CSR
  if (nrp && cudaDeviceSynchronize() != cudaSuccess) rc = set_error(SPMX_ERR_CUDA, "coo to csr");
  if (!nrp) rc = rc ? rc : dalloc((void**)&nrp, 4 * ((size_t)m + 1), "csr rowptr");
  if (!ncol) rc = rc ? rc : dalloc((void**)&ncol, b, "csr col");
  if (val && !nval) rc = rc ? rc : dalloc((void**)&nval, b, "csr val");
  const unsigned* rows_sorted = (const unsigned*)row;
  // a failure from here on leaves the handle without a matrix, unless the one it
  // has is the caller's
  if (!rc && h->own_csr_rowptr && h->rowptr == h->own_csr_rowptr) forget_csr(h);
  if (!rc && unsorted) {
    const int bits_c = key_bits(n), bits_r = key_bits(m);
    const int first = col_desc ? 0 : bits_c;
    const int fin = radix_sort_passes(first, bits_c + bits_r) & 1;  // set holding the result after the last pass
    unsigned *k[2], *r[2], *v[2] = {nullptr, nullptr};
    char* q = scratch;
    k[fin] = (unsigned*)ncol;
    k[1 - fin] = (unsigned*)q; q += al;
    r[0] = (unsigned*)q; q += al;
    r[1] = (unsigned*)q; q += al;
    if (val) {
      v[fin] = (unsigned*)nval;
      v[1 - fin] = (unsigned*)q; q += al;
    }
    RadixBuffers rb{k[0], k[1], r[0], r[1], v[0], v[1], q, false, (const unsigned*)col, (const unsigned*)row,
                    (const unsigned*)val, first, bits_c};
    if (radix_sort_pairs(rb, nnz, bits_c + bits_r, h->d_err, st)) rc = set_error(SPMX_ERR_CUDA, "coo sort launch");
    rows_sorted = r[fin];
  }
  // 3. row pointers from the sorted rows; columns and values into place
  if (!rc) {
    launch_sorted_bounds(nnz, rows_sorted, m, nrp, st);
    if (nnz > 0 && !unsorted) {
      cudaMemcpyAsync(ncol, col, 4 * (size_t)nnz, cudaMemcpyDeviceToDevice, st);
      if (val) cudaMemcpyAsync(nval, val, 4 * (size_t)nnz, cudaMemcpyDeviceToDevice, st);
    }
    rc = launch_ok("coo to csr");
  }
  scratch_free(scratch, st);
  const cudaError_t ce = cudaStreamSynchronize(st);
  if (!rc && ce != cudaSuccess) rc = set_error(SPMX_ERR_CUDA, std::string("coo to csr: ") + cudaGetErrorString(ce));
  if (rc) {
    if (nrp != h->own_csr_rowptr) dfree(nrp);
    if (ncol != h->own_csr_col) dfree(ncol);
    if (nval && nval != h->own_csr_val) dfree(nval);
    return rc;
  }
  if (!val) dfree(h->own_csr_val);
  h->own_csr_rowptr = nrp;
  h->own_csr_col = ncol;
  h->own_csr_val = nval;
  h->rowptr = nrp;
  h->col = ncol;
  h->val = nval;
  forget_csr(h);
  h->has_csr = true;
  return SPMX_SUCCESS;
}

extern "C" int spmx_copy_csr(spmx_handle_t h, int* rowptr, int* col, float* val) {
  SPMX_CHECK_HANDLE(h);
  if (!h->has_csr) return set_error(SPMX_ERR_NOT_READY, "no CSR (call spmx_input_csr or spmx_input_coo)");
  cudaStream_t st = h->stream;
  if (rowptr)
    SPMX_CUDA(cudaMemcpyAsync(rowptr, h->rowptr, 4 * ((size_t)h->m + 1), cudaMemcpyDeviceToDevice, st));
  if (col && h->nnz)
    SPMX_CUDA(cudaMemcpyAsync(col, h->col, 4 * (size_t)h->nnz, cudaMemcpyDeviceToDevice, st));
  if (val && h->val && h->nnz)
    SPMX_CUDA(cudaMemcpyAsync(val, h->val, 4 * (size_t)h->nnz, cudaMemcpyDeviceToDevice, st));
  return SPMX_SUCCESS;
}
