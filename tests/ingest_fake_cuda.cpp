// spmx_input_coo against a stand-in for the CUDA runtime and for the library's
// own allocations and sort: "device" memory is host memory, kernels do nothing,
// and one step of a call can be made to fail.  Prints nothing and returns 0 where
// every handle is left as it has to be.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "engine.h"

static int g_sort_rc = 0;         // what the sort returns
static int g_alloc_fail = 0;      // allocations refused
static int g_sync_fail_at = 0;    // the stream synchronisation that fails, counted from 1
static int g_syncs = 0;

static int* g_flags = nullptr;    // the handle's flag words

extern "C" {
struct dim3_ { unsigned x, y, z; };
void** __cudaRegisterFatBinary(void*) { static void* p; return &p; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
unsigned __cudaPushCallConfiguration(dim3_, dim3_, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3_*, dim3_*, size_t*, void*) { return cudaSuccess; }
}

cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
  g_flags[1] = 1;  // the only kernel is the check: not in order
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return ++g_syncs == g_sync_fail_at ? cudaErrorUnknown : cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }

namespace spmx {
void note_launch(int) {}
int set_error(int code, const std::string&) { return code; }
int dalloc(void** p, size_t n, const char*) { *p = g_alloc_fail ? nullptr : malloc(n + 16); return *p ? SPMX_SUCCESS : SPMX_ERR_ALLOC; }
void dfree(void* p) { free(p); }
int scratch_alloc(void** p, size_t n, cudaStream_t, const char* what) { return dalloc(p, n, what); }
void scratch_free(void* p, cudaStream_t) { free(p); }
size_t radix_scratch_bytes(int) { return 64; }
int radix_sort_passes(int, int) { return 1; }
int radix_sort_pairs(RadixBuffers&, int, int, int*, cudaStream_t) { return g_sort_rc; }
int launch_sorted_bounds(int, const unsigned*, int, int*, cudaStream_t) { return 0; }
}  // namespace spmx

#define CHECK(c) do { if (!(c)) { printf("%s:%d %s\n", __FILE__, __LINE__, #c); return 1; } } while (0)

enum Fault { kNone, kSort, kLastSync, kLaunch, kAlloc };

static int input(spmx_handle_t h, Fault f) {
  static const int row[4] = {2, 0, 1, 0}, col[4] = {0, 1, 2, 0};
  static const float val[4] = {1, 2, 3, 4};
  g_sort_rc = f == kSort ? -1 : 0;
  g_alloc_fail = f == kAlloc;
  g_syncs = 0;
  g_sync_fail_at = f == kLastSync ? 2 : 0;  // the first is that of the check
  const int rc = spmx_input_coo(h, 4, row, col, val);
  g_sort_rc = g_alloc_fail = g_sync_fail_at = 0;
  return rc;
}

int main() {
  for (Fault f : {kSort, kLastSync, kAlloc}) {
    for (bool borrowed : {false, true}) {
      spmx_handle_s hs;
      spmx_handle_t h = &hs;
      h->m = h->n = 3;
      h->nnz = 4;
      std::vector<int> iacc(4), pinned(16), colptr(4), rp(4), cl(4);
      h->d_iacc = g_flags = iacc.data();
      h->h_pinned = pinned.data();
      h->own_colptr = colptr.data();
      CHECK(input(h, kNone) == SPMX_SUCCESS && h->has_csr);
      if (borrowed) {  // as spmx_input_csr leaves it
        h->rowptr = rp.data();
        h->col = cl.data();
      }
      h->has_csc = true;  // as spmx_to_csc leaves it
      h->csc_colptr = h->own_colptr;
      h->mat_feat_ready = h->std_row_ready = h->batch_chunk_ready = h->ms_hubs_ready = true;
      h->hola_rowptr = h->rowptr;
      CHECK(input(h, f) != SPMX_SUCCESS);
      const bool kept = borrowed || f == kAlloc;  // nothing of the matrix was written
      CHECK(h->has_csr == kept && h->has_csc == kept);
      CHECK(h->mat_feat_ready == kept && h->std_row_ready == kept);
      CHECK(h->batch_chunk_ready == kept && h->ms_hubs_ready == kept && (h->hola_rowptr == h->rowptr) == kept);
      if (borrowed) CHECK(h->rowptr == rp.data() && h->col == cl.data());
      CHECK(input(h, kNone) == SPMX_SUCCESS && h->has_csr && !h->has_csc && h->rowptr == h->own_csr_rowptr);
    }
  }
  return 0;
}
