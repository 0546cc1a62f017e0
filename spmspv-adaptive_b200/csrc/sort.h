// Radix sort / scan / reduce_by_key launchers (sort.cu).
#pragma once
#include "kernels.h"

namespace spmx {

// A stable sort by the key bits [first_bit, key_bits) of radix_sort_pairs.
// With src_keys the first pass reads the source arrays and leaves them as they
// are; `keys` and the payloads are then only the second buffer set.
struct RadixBuffers {
  unsigned* keys;      // input keys; result here unless result_in_alt
  unsigned* keys_alt;
  unsigned* p1;        // optional payloads (NULL when absent)
  unsigned* p1_alt;
  unsigned* p2;
  unsigned* p2_alt;
  void* scratch;       // radix_scratch_bytes(n), 8-byte aligned
  bool result_in_alt;  // set by radix_sort_pairs: an odd number of passes
  const unsigned* src_keys;
  const unsigned* src_p1;
  const unsigned* src_p2;
  int first_bit;
  int lo_bits;         // > 0: sorts by (p1 << lo_bits) | key; p1 is needed
};

size_t radix_scratch_bytes(int n);
int radix_sort_passes(int first_bit, int end_bit);
int radix_sort_pairs(RadixBuffers& b, int n, int key_bits, int* err, cudaStream_t st);
int launch_sorted_bounds(int cnt, const unsigned* key, int extent, int* ptr, cudaStream_t st);
int launch_scan_exclusive(const int* in, int* out, int n, int* total_out,
                          ScanScratch& ls, int* err, cudaStream_t st);
int reduce_by_key_sorted(const unsigned* keys, const float* vals, int n,
                         int* slot_scratch, int* out_key, float* out_val,
                         int* d_count, ScanScratch& ls, int* err,
                         cudaStream_t st);

}  // namespace spmx
