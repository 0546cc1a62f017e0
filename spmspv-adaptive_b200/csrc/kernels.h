// Host-side launchers of the spmx kernels (implemented in the .cu files of
// this directory).  All launches are asynchronous on the given stream.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace spmx {

// number of kernels this library has launched (all handles, all threads)
void note_launch(int k = 1);

struct SpmvArgs {
  int m, n, nnz;
  const int* rowptr;
  const int* col;
  const float* val;
  const float* x;
  const int* bits;  // non-NULL selects the bitmap-gated SpMSpV form
  double alpha;
  float* y;
  int* err;
};

struct HolaTables {
  int vt;        // nonzeros per thread (4, 8 or 16); 256 threads per CTA
  int K;         // nonzeros per CTA = 256 * vt
  int nchunks;   // ceil(nnz / K)
  int* chunk_row;  // [nchunks + 1]
  int4* list;      // [nchunks] chunk descriptors: n_short chunks of short rows, then the others
  int n_short;     // 0: not worth their own kernel
  double* carry;   // [2 * nchunks]
  unsigned* arrive;  // [nchunks], zero between calls
};

// a chunk none of whose rows has more nonzeros in it is worked row by row
constexpr int kShortRow = 32;

// ---- spmv.cu
int launch_spmv_naive(const SpmvArgs& a, int group, cudaStream_t st);
int launch_spmv_hola(const SpmvArgs& a, const HolaTables& t, cudaStream_t st);
// the first row of every chunk; with a list also which chunks have only short rows
int launch_chunk_rows(int m, int nnz, const int* rowptr, int K, int nchunks, int* chunk_row,
                      int4* list, int* counts, cudaStream_t st);
int hola_chunk_nnz(int vt);

// A kernel that runs or returns at once by a count on the device: with `count`
// set it runs where (*count < limit) == below.
struct DevGate {
  const int* count;
  int limit;
  bool below;
};

// ---- adjoint.cu
int launch_spmv_backward(int m, int n, int nnz, const int* rowptr, const int* col,
                         const float* val, const float* x, const float* dy,
                         const HolaTables& t, float* dx, float* dvals, int* err,
                         DevGate gate, cudaStream_t st);
int launch_spmv_backward_csc(int m, int n, const int* rowptr, const int* col, const int* colptr,
                             const int* crow, const float* cval, const float* x, const float* dy,
                             int g1, int g2, float* dx, float* dvals, int* err, DevGate gate,
                             cudaStream_t st);
int launch_spmv_backward_sparse(int m, int n, const int* rowptr, const int* col,
                                const float* val, const float* x, int dy_nnz,
                                const int* dy_key, const float* dy_val, int group,
                                float* dx, float* dvals, int* err, cudaStream_t st);
// the same for a compacted dy of *gate.count entries
int launch_spmv_backward_gated(int m, int n, const int* rowptr, const int* col, const float* val, const float* x,
                               const int* dy_key, const float* dy_val, int group, float* dx, float* dvals,
                               int num_sms, int* err, DevGate gate, cudaStream_t st);
// dx = 0 and dvals = 0 behind the gate; dx behind no gate where dx_always
int launch_backward_clear(int n, int nnz, float* dx, float* dvals, bool dx_always, int num_sms, DevGate gate,
                          cudaStream_t st);

// ---- lookback scratch shared by the single-pass scans
struct ScanScratch {
  unsigned long long* status;  // tile status words
  int status_len;              // capacity in tiles
  unsigned* ticket;            // 4 words, zeroed once: ticket, epoch, publish count
  unsigned* counts;            // kCompactMaxRanges per-range counts (the compaction's first pass)
};

// ranges of a compaction, each counted by a CTA before any is written
constexpr int kCompactMaxRanges = 1024;

// indices into the handle's device counter block
enum CounterSlot : int {
  kCntYnnz = 0,
  kCntBinlen = 1,
  kCntXnnz = 2,
  kCntBlocksTL = 3,
  kCntBlocksMG = 4,
  kCntDy = 5,          // nonzeros of the adjoint's dy
  kCntLong = 6,        // chunks of long columns, 64-bit (slots 6..7): repeated x keys count past 2^31
  kCntFeatSum = 8,   // 64-bit (slots 8..9)
  kCntFeatMax = 10,
  kCntFeatMinInv = 11,
  kCntTotal = 16
};

// ---- csc.cu
struct CscArgs {
  int m, n;
  const int* colptr;   // [n+1]
  const int* row;      // [nnz]
  const float* val;    // [nnz]
  int x_nnz;
  const int* x_key;
  const float* x_val;
  double alpha;
  int* err;
  int* counts;         // device counter block
};

struct CscScratch {
  int* off;        // [x_nnz + 1] exclusive scan of column lengths
  int* colstart;   // [x_nnz]     colptr[x_key[i]]
  int* bstart_tl;  // block -> first x entry (fixed nnz per block)
  int* bstart_mg;  // block -> first x entry (merge-path items)
  int tl_cap, mg_cap;  // capacities of the two tables
  struct CscLong* longq;  // chunks of long columns (csc_flat_kernel)
  int long_cap;
};

// kFlatChunk nonzeros of one column and its x value
struct CscLong {
  int k0, k1;
  float x;
};
constexpr int kFlatCut = 128;    // columns above this are cut into chunks of
constexpr int kFlatChunk = 128;  // this many nonzeros

constexpr int kCscScanNT = 256, kCscScanVT = 8;   // 2048 x entries per tile
constexpr int kCscLbNT = 256, kCscLbVT = 8;       // 2048 items per LB block

int launch_csc_scan(const CscArgs& a, const CscScratch& s, ScanScratch& ls, cudaStream_t st);
// variant: 1 merge, 2 twolayer.  pairs_row/pairs_val non-NULL: write (row,
// alpha*val*x) pairs at their scanned position instead of atomics into y.
int launch_csc_lb(const CscArgs& a, const CscScratch& s, int variant, float* y,
                  int* pairs_row, float* pairs_val, int grid, cudaStream_t st);
int launch_csc_naive(const CscArgs& a, int group, float* y, cudaStream_t st);
// y = 0, then the load-balanced SpMSpV with atomic write-back; col_max: the
// longest column of the matrix, -1 where it is not known.  bin_len goes to
// counts[kCntBinlen].
int launch_csc_flat(const CscArgs& a, const CscScratch& s, float* y, long long col_max, int num_sms,
                    cudaStream_t st);
// the same into acc, whose rows that no nonzero reaches stay -0.0 (no other is);
// row_max: the longest row, -1 where it is not known
int launch_csc_flat_rows(const CscArgs& a, const CscScratch& s, double* acc, long long col_max, long long row_max,
                         int num_sms, cudaStream_t st);
// the naive CSC SpMSpV of a handful of x entries in one launch, and whether it
// applies (col_max: the longest column, -1 where it is not known)
bool csc_slice_fits(const CscArgs& a, long long col_max, cudaStream_t st);
int launch_csc_slice(const CscArgs& a, float* y, cudaStream_t st);
// y = 0 then the naive CSC SpMSpV, as a programmatic dependent launch pair
int launch_csc_naive_zeroed(const CscArgs& a, int group, float* y, int num_sms, cudaStream_t st);
int launch_csc_naive_pairs(const CscArgs& a, const CscScratch& s, int group,
                           int* pairs_row, float* pairs_val, cudaStream_t st);

// ---- vecconv.cu
// y[0..m) = 0 with a kernel that lets the next grid launch early
int launch_zero_fill(float* y, long long m, int num_sms, cudaStream_t st, int* c0 = nullptr,
                     unsigned long long* c1 = nullptr);
// dense[0..len) from (key, val): a zero fill, then the scatter as a
// programmatic dependent launch that reads its keys and values while the
// fill runs; the scatter in turn lets the next grid start early
int launch_dense_from_sparse(int nvals, int len, const int* key, const float* val, float* dense,
                             int* err, int num_sms, cudaStream_t st);
int launch_scatter(int nvals, int len, const int* key, const float* val,
                   float* dense, int* bits, int* err, cudaStream_t st);
int launch_dense2bits(int len, const float* dense, int* bits, cudaStream_t st);
// keys/vals of the entries != 0 of dense[0..len), in order; count -> *d_count.
// limit > 0: nothing but the count is written where it reaches the limit.
// h_counts (optional, two ints of page-locked host memory; without a limit): the
// count once the grid is done
// range_counts: kCompactMaxRanges words that no compaction beside this one uses
int launch_compact_nonzero(int len, const float* dense, int* key, float* val,
                           int* d_count, unsigned* range_counts, cudaStream_t st, int limit = 0,
                           int* h_counts = nullptr);
// keys/vals (each optional) of the entries of acc[0..len) other than -0.0, in
// order; dense (optional): all of them, rounded, the others 0; count -> *d_count.
// *total above cap >= 0: kDevErrCapacity.  h_counts (optional, page-locked host
// memory): the count and *total once the grid is done
int launch_compact_rows(int len, const double* acc, float* dense, int* key, float* val, int* d_count,
                        const int* total, int cap, int* err, int* h_counts, unsigned* range_counts,
                        cudaStream_t st);

}  // namespace spmx
