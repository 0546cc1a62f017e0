// Stable LSD radix sort of 32-bit keys with up to two 32-bit payloads, a
// generic single-pass exclusive scan, and reduce_by_key over sorted keys.
//
// They replace the Thrust / CUB calls of the reference's sort write-back
// (thrust::sort_by_key + thrust::reduce_by_key, DEV/csc_sort_spmspv.cuh:341,
// :412) and cuSPARSE csr2csc inside ToCSC (H:409): a transpose is a stable
// sort of the row-major COO by column.
//
// A sort is one histogram kernel, which reads the keys once and counts the
// digits of every pass, and one kernel per pass of at most 8 bits (the bits
// are spread evenly over the passes: fewer digits, longer runs of equal digits
// in the output).  A pass reads and writes every array once.  Its tiles chain
// through per-digit decoupled look-back words, so the digit counts of a tile
// never make a round trip through memory; the tile is put in digit order in
// shared memory first, so a warp's stores cover runs of consecutive addresses.
//
// What bounds a pass: the shared-memory pipe (86% busy; issue slots 49%, DRAM
// 33%) with the ranking and the exchange, about 140 warp instructions per 32
// items with two payloads; 32 warps per SM at 64 registers.  16.8M items with two
// payloads: 119 us per pass (3.4 TB/s; 140 with two keys) and 34 us for the
// histogram (105 for the five digits of two keys: issue slots, 71%); the form before (per-tile histogram,
// scan of the histograms, scatter straight from registers, each 4-byte store in
// a sector of its own) took 430 + 37 + 13 us per pass.  Measured beside it:
// peers by __match_any_sync 210 us, by one ballot per digit bit 143 us, by the
// shared match word 128 us (512 threads, 6,144 items); 256 threads and 4,096
// items 119 us, 5,120 items 128 us, 384 threads and 4,608 items 126 us.
#include <algorithm>

#include "kernels.h"
#include "sort.h"
#include "common.cuh"

namespace spmx {

constexpr int kRadixNT = 256;
constexpr int kRadixWarps = kRadixNT / 32;
constexpr int kRadixDigits = 256;
constexpr int kRadixMaxPasses = 8;  // two 31-bit keys

// look-back words: [63:34] pass + 1, [33:32] 1 = tile count, 2 = inclusive
// prefix, [31:0] value; cleared once per sort, the pass number tells the
// passes apart
struct RadixPass {
  const unsigned *k_in, *p1_in, *p2_in;
  unsigned *k_out, *p1_out, *p2_out;
  int n, shift, bits, lo_bits, pass, ntiles;
  unsigned long long* status;  // [ntiles][256]
  unsigned* ticket;
  const unsigned* ghist;       // [256] digit counts of this pass
  int* err;
};

// digit of an item; with two keys the sort key is (p1 << lo_bits) | key
template <bool TWO>
__device__ __forceinline__ unsigned radix_digit(unsigned lo, unsigned hi, int lo_bits, int shift, unsigned mask) {
  if (TWO) {
    const unsigned long long k = ((unsigned long long)hi << lo_bits) | lo;
    return (unsigned)(k >> shift) & mask;
  }
  return (lo >> shift) & mask;
}

// digit counts of all passes: pass p has the bits [first + p * bits, first +
// (p + 1) * bits)
template <bool TWO>
__global__ void __launch_bounds__(kRadixNT)
radix_hist_kernel(const unsigned* keys, const unsigned* hi, int n, int first, int bits, int lo_bits, int passes,
                  unsigned* ghist) {
  __shared__ unsigned s_h[kRadixMaxPasses * kRadixDigits];
  constexpr int U = 8;
  for (int i = threadIdx.x; i < passes * kRadixDigits; i += kRadixNT) s_h[i] = 0u;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  __syncthreads();
  const unsigned mask = (1u << bits) - 1u;
  const int lane = threadIdx.x & 31;
  for (long long b = (long long)blockIdx.x * kRadixNT * U; b < n; b += (long long)gridDim.x * kRadixNT * U) {
    unsigned k[U], h[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = b + u * kRadixNT + threadIdx.x;
      k[u] = i < n ? keys[i] : 0u;
      h[u] = TWO && i < n ? hi[i] : 0u;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool valid = b + u * kRadixNT + threadIdx.x < n;
      const unsigned act = __ballot_sync(0xffffffffu, valid);
      for (int p = 0; p < passes; ++p) {
        const unsigned d = radix_digit<TWO>(k[u], h[u], lo_bits, first + p * bits, mask);
        // a warp of one digit (sorted or constant keys) adds once
        const unsigned d0 = __shfl_sync(0xffffffffu, d, 0);
        if (__all_sync(0xffffffffu, !valid || d == d0)) {
          if (lane == 0 && act) atomicAdd(&s_h[p * kRadixDigits + d0], (unsigned)__popc(act));
        } else if (valid) {
          atomicAdd(&s_h[p * kRadixDigits + d], 1u);
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kRadixDigits; i += kRadixNT)
    if (s_h[i]) atomicAdd(ghist + i, s_h[i]);
}

// One pass over one tile of kRadixNT * IPT items.  Each warp owns 32 * IPT
// consecutive items and ranks them round by round: each lane sets its bit in
// its digit's match word, the word then names the lanes of equal digit, and
// warp-private digit counters carry the rank from round to round, so equal
// digits keep their input order.
template <int IPT, int NPAY, bool TWO, int BITS>
__global__ void __launch_bounds__(kRadixNT, 4) radix_pass_kernel(RadixPass a) {
  constexpr int TILE = kRadixNT * IPT;
  __shared__ unsigned s_stage[TILE > (kRadixWarps << BITS) ? TILE : kRadixWarps << BITS];
  __shared__ unsigned short s_wc[kRadixWarps][1 << BITS];
  __shared__ unsigned char s_dig[TWO ? TILE : 4];
  __shared__ int s_gb[1 << BITS];  // output position of local position 0 of the digit's run
  __shared__ unsigned long long s_wtmp[kRadixWarps + 1];
  __shared__ int s_tile;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const unsigned mask = (1u << a.bits) - 1u;
  constexpr int ND = 1 << BITS;
  for (int i = tid; i < kRadixWarps * ND / 2; i += kRadixNT) reinterpret_cast<unsigned*>(s_wc)[i] = 0u;
  // the lanes that hold each digit, one word per digit and warp (in the stage,
  // which is not in use yet)
  unsigned* const s_match = s_stage + w * ND;
  for (int i = tid; i < kRadixWarps * ND; i += kRadixNT) s_stage[i] = 0u;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  if (tid == 0) s_tile = (int)atomicAdd(a.ticket, 1u);
  __syncthreads();
  const int tile = s_tile;
  const size_t tbase = (size_t)tile * TILE;
  const int valid = (int)min((long long)TILE, a.n - (long long)tbase);
  const int li = w * 32 * IPT + lane;  // the thread's items: li + 32 j of the tile
  const unsigned* kin = a.k_in + tbase;
  unsigned k[IPT];
  unsigned pos[IPT];  // digit << 16 | rank, then the local position
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    // items past the end take the largest digit: they are the tile's last
    // items, so they end up behind every valid one
    const bool in = li + j * 32 < valid;
    k[j] = in ? kin[li + j * 32] : 0xffffffffu;
    if (TWO) pos[j] = in ? a.p1_in[tbase + li + j * 32] : 0xffffffffu;
  }
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    const unsigned d = radix_digit<TWO>(k[j], TWO ? pos[j] : 0u, a.lo_bits, a.shift, mask);
    atomicOr(&s_match[d], 1u << lane);
    __syncwarp();
    const unsigned peers = s_match[d];
    const int base = s_wc[w][d];
    __syncwarp();
    if ((peers & lanemask_lt()) == 0u) {
      s_wc[w][d] = (unsigned short)(base + __popc(peers));
      s_match[d] = 0u;
    }
    pos[j] = (d << 16) | (unsigned)(base + __popc(peers & lanemask_lt()));
    __syncwarp();
  }
  __syncthreads();
  // thread d: the tile's count of digit d, published at once; then the digit
  // offsets inside the tile (low word) and in the output (high word)
  unsigned cnt = 0;
  if (tid < ND) {
#pragma unroll
    for (int q = 0; q < kRadixWarps; ++q) cnt += s_wc[q][tid];
    st_volatile_u64(a.status + (size_t)tile * ND + tid,
                    lb_pack((unsigned)a.pass + 1u, tile == 0 ? 2u : 1u, cnt));
  }
  unsigned long long both = 0;
  if (tid < ND) both = ((unsigned long long)a.ghist[tid] << 32) | cnt;
  unsigned long long total;
  const unsigned long long ex = block_exclusive_sum<kRadixNT>(both, s_wtmp, &total);
  const unsigned off = (unsigned)ex;
  if (tid < ND) {
    unsigned run = off;
#pragma unroll
    for (int q = 0; q < kRadixWarps; ++q) {
      const unsigned t = s_wc[q][tid];
      s_wc[q][tid] = (unsigned short)run;
      run += t;
    }
  }
  __syncthreads();
  // local positions; keys into digit order; the first payload's loads in
  // flight during the look-back
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    const unsigned d = pos[j] >> 16;
    pos[j] = s_wc[w][d] + (pos[j] & 0xffffu);
    s_stage[pos[j]] = k[j];
    if (TWO) s_dig[pos[j]] = (unsigned char)d;
  }
  if (NPAY > 0) {
#pragma unroll
    for (int j = 0; j < IPT; ++j) k[j] = li + j * 32 < valid ? a.p1_in[tbase + li + j * 32] : 0u;
  }
  int fail = 0;
  if (tid < ND) {
    // look-back, four predecessors per round trip
    constexpr int LW = 4;
    unsigned before = 0;
    int j = tile - 1;
    long long spins = 0;
    bool done = tile == 0;
    while (!done) {
      unsigned long long word[LW];
#pragma unroll
      for (int q = 0; q < LW; ++q)
        word[q] = j - q >= 0 ? ld_volatile_u64(a.status + (size_t)(j - q) * ND + tid)
                             : lb_pack((unsigned)a.pass + 1u, 2u, 0u);
      int used = 0;
#pragma unroll
      for (int q = 0; q < LW; ++q) {
        if (done || used < q) continue;  // behind a prefix, or behind a tile not yet published
        if ((unsigned)(word[q] >> 34) != (unsigned)a.pass + 1u) continue;
        before += (unsigned)word[q];
        ++used;
        done = ((word[q] >> 32) & 3u) == 2u;
      }
      j -= used;
      if (!done && used == 0) {
        if (++spins > kSpinLimit) {
          flag_error(a.err, kDevErrTimeout);
          fail = 1;
          break;
        }
        __nanosleep(20);
      }
    }
    if (tile > 0 && !fail)
      st_volatile_u64(a.status + (size_t)tile * ND + tid, lb_pack((unsigned)a.pass + 1u, 2u, before + cnt));
    s_gb[tid] = (int)((unsigned)(ex >> 32) + before - off);
  }
  if (__syncthreads_or(fail)) return;  // nothing is written after a wait that gave up
  int dst[IPT];
#pragma unroll
  for (int r = 0; r < IPT; ++r) {
    const int i = r * kRadixNT + tid;
    const unsigned key = s_stage[i];
    const unsigned d = TWO ? s_dig[i] : radix_digit<false>(key, 0u, 0, a.shift, mask);
    dst[r] = s_gb[d] + i;
    if (i < valid) a.k_out[dst[r]] = key;
  }
#pragma unroll
  for (int p = 0; p < NPAY; ++p) {
    unsigned* out = p == 0 ? a.p1_out : a.p2_out;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < IPT; ++j) s_stage[pos[j]] = k[j];
    __syncthreads();
    if (p + 1 < NPAY) {
#pragma unroll
      for (int j = 0; j < IPT; ++j) k[j] = li + j * 32 < valid ? a.p2_in[tbase + li + j * 32] : 0u;
    }
#pragma unroll
    for (int r = 0; r < IPT; ++r)
      if (r * kRadixNT + tid < valid) out[dst[r]] = s_stage[r * kRadixNT + tid];
  }
}

// generic exclusive scan of ints (single pass, decoupled look-back)
template <int NT, int VT>
__global__ void __launch_bounds__(NT)
scan_exclusive_kernel(const int* __restrict__ in, int* __restrict__ out, int n,
                      LookbackState st, int ntiles, int* total_out, int* err) {
  __shared__ int s_v[NT * VT];
  __shared__ unsigned s_wtmp[NT / 32 + 1];
  __shared__ int s_tile;
  __shared__ unsigned s_prefix;
  const int tile = lb_acquire_tile(st, ntiles, &s_tile);
  const int base = tile * NT * VT;
  const int tid = threadIdx.x;
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int i = base + j * NT + tid;
    s_v[j * NT + tid] = (i < n) ? __ldg(in + i) : 0;
  }
  __syncthreads();
  unsigned loc[VT];
  unsigned sum = 0;
#pragma unroll
  for (int j = 0; j < VT; ++j) { loc[j] = (unsigned)s_v[tid * VT + j]; sum += loc[j]; }
  unsigned total;
  const unsigned ex = block_exclusive_sum<NT>(sum, s_wtmp, &total);
  if (tid < 32) {
    const unsigned p = lb_warp_lookback(st, tile, ntiles, total, err);
    if (tid == 0) s_prefix = p;
  }
  __syncthreads();
  unsigned run = s_prefix + ex;
#pragma unroll
  for (int j = 0; j < VT; ++j) { s_v[tid * VT + j] = (int)run; run += loc[j]; }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int i = base + j * NT + tid;
    if (i < n) out[i] = s_v[j * NT + tid];
  }
  if (tile == ntiles - 1 && tid == 0 && total_out) *total_out = (int)(s_prefix + total);
}

int launch_scan_exclusive(const int* in, int* out, int n, int* total_out,
                          ScanScratch& ls, int* err, cudaStream_t st) {
  constexpr int NT = 256, VT = 8;
  if (n <= 0) return 0;
  const int ntiles = (n + NT * VT - 1) / (NT * VT);
  if (ntiles > ls.status_len) return -1;
  LookbackState lbs{ls.status, ls.ticket};
  note_launch();
  scan_exclusive_kernel<NT, VT><<<ntiles, NT, 0, st>>>(in, out, n, lbs, ntiles,
                                                      total_out, err);
  return 0;
}

// items per thread: tiles of 4,096 items while they fill the 592 resident CTAs
// (4 per SM), of 2,048 or 1,024 below.  A run of equal digits is 32 items long
// in a tile of 4,096 and 7-bit digits, and a short input needs the tiles more
// (0.56M items, three passes: 31 us in tiles of 2,048, 36 us in tiles of 6,144)
constexpr int kRadixFrom16 = 148 * 4 * 4096, kRadixFrom8 = 148 * 2048;
static int radix_ipt(int n) { return n >= kRadixFrom16 ? 16 : n >= kRadixFrom8 ? 8 : 4; }

static int radix_tiles(int n) {
  const int tile = kRadixNT * radix_ipt(n);
  return (int)(((long long)n + tile - 1) / tile);
}

// scratch of a sort: look-back words, digit counts, tickets
static size_t radix_status_bytes(int ntiles) { return (size_t)ntiles * kRadixDigits * 8; }

// enough for every sort of at most n items: the tile count is not monotonic
// where the tile grows
size_t radix_scratch_bytes(int n) {
  int t = radix_tiles(n);
  if (n >= kRadixFrom8) t = std::max(t, radix_tiles(kRadixFrom8 - 1));
  if (n >= kRadixFrom16) t = std::max(t, radix_tiles(kRadixFrom16 - 1));
  return radix_status_bytes(t) + 4 * (size_t)kRadixMaxPasses * (kRadixDigits + 1);
}

template <int IPT, int BITS>
static cudaError_t launch_radix_pass(const RadixPass& a, int npay, bool two, cudaStream_t st) {
  const dim3 grid((unsigned)a.ntiles), block(kRadixNT);
  if (two && npay == 2) return launch_pdl(radix_pass_kernel<IPT, 2, true, BITS>, grid, block, 0, st, a);
  if (two) return launch_pdl(radix_pass_kernel<IPT, 1, true, BITS>, grid, block, 0, st, a);
  if (npay == 2) return launch_pdl(radix_pass_kernel<IPT, 2, false, BITS>, grid, block, 0, st, a);
  if (npay == 1) return launch_pdl(radix_pass_kernel<IPT, 1, false, BITS>, grid, block, 0, st, a);
  return launch_pdl(radix_pass_kernel<IPT, 0, false, BITS>, grid, block, 0, st, a);
}

template <int IPT>
static cudaError_t launch_radix_pass(const RadixPass& a, int npay, bool two, cudaStream_t st) {
  return a.bits <= 7 ? launch_radix_pass<IPT, 7>(a, npay, two, st) : launch_radix_pass<IPT, 8>(a, npay, two, st);
}

int radix_sort_passes(int first_bit, int end_bit) {
  return std::max(1, (end_bit - first_bit + 7) / 8);
}

int radix_sort_pairs(RadixBuffers& b, int n, int key_bits, int* err, cudaStream_t st) {
  b.result_in_alt = false;
  const bool two = b.lo_bits > 0;
  const int passes = radix_sort_passes(b.first_bit, key_bits);
  if (passes > kRadixMaxPasses || (two && !b.p1)) return -1;
  if (n <= 0 || (n == 1 && !b.src_keys)) return 0;
  const int bits = std::max(1, (key_bits - b.first_bit + passes - 1) / passes);
  const int npay = b.p2 ? 2 : b.p1 ? 1 : 0;
  const int ipt = radix_ipt(n), ntiles = radix_tiles(n);
  unsigned long long* status = reinterpret_cast<unsigned long long*>(b.scratch);
  unsigned* ghist = reinterpret_cast<unsigned*>(reinterpret_cast<char*>(b.scratch) + radix_status_bytes(ntiles));
  unsigned* ticket = ghist + kRadixMaxPasses * kRadixDigits;
  if (cudaMemsetAsync(b.scratch, 0, radix_status_bytes(ntiles) + 4 * (size_t)kRadixMaxPasses * (kRadixDigits + 1),
                      st) != cudaSuccess)
    return -1;
  const unsigned *kin = b.src_keys ? b.src_keys : b.keys, *p1in = b.src_keys ? b.src_p1 : b.p1,
                 *p2in = b.src_keys ? b.src_p2 : b.p2;
  unsigned *kout = b.keys_alt, *p1out = b.p1_alt, *p2out = b.p2_alt;
  note_launch(1 + passes);
  const int hgrid = (int)std::min<long long>(((long long)n + kRadixNT * 8 - 1) / (kRadixNT * 8), 148 * 4);
  cudaError_t e = two ? launch_pdl(radix_hist_kernel<true>, dim3(hgrid), dim3(kRadixNT), 0, st, kin, p1in, n,
                                   b.first_bit, bits, b.lo_bits, passes, ghist)
                      : launch_pdl(radix_hist_kernel<false>, dim3(hgrid), dim3(kRadixNT), 0, st, kin,
                                   (const unsigned*)nullptr, n, b.first_bit, bits, 0, passes, ghist);
  for (int p = 0; p < passes && e == cudaSuccess; ++p) {
    const RadixPass a{kin, p1in, p2in, kout, p1out, p2out, n, b.first_bit + p * bits, bits, b.lo_bits, p, ntiles,
                      status, ticket + p, ghist + p * kRadixDigits, err};
    e = ipt == 16 ? launch_radix_pass<16>(a, npay, two, st)
        : ipt == 8 ? launch_radix_pass<8>(a, npay, two, st)
                   : launch_radix_pass<4>(a, npay, two, st);
    const bool alt = (p & 1) == 0;  // this pass wrote the alternate set
    kin = alt ? b.keys_alt : b.keys;
    p1in = alt ? b.p1_alt : b.p1;
    p2in = alt ? b.p2_alt : b.p2;
    kout = alt ? b.keys : b.keys_alt;
    p1out = alt ? b.p1 : b.p1_alt;
    p2out = alt ? b.p2 : b.p2_alt;
    b.result_in_alt = alt;
  }
  return e == cudaSuccess ? 0 : -1;
}

// ptr[j] = first position whose key is >= j, j in [0, extent], of `cnt` sorted
// keys (keys past the extent end the last range): position i owns the entries
// after its predecessor's key up to its own key (extent at i = cnt), so every
// entry is written once, empty ranges included.  A thread owns four consecutive
// positions, a warp reads 512 bytes per load, and the key before a thread's
// first comes from its neighbour lane.
//
// A thread writes up to kBoundsNarrow entries by itself, a warp together a longer
// gap; of that the whole tiles of kBoundsTile entries (counted from entry 0) are
// left to the last `tiles` CTAs, each of which looks up the value of its tile's
// first entry and fills the tile if the last has the same.  ToCSC of 8M columns
// with all 2M nonzeros in 64 of them takes 0.14 ms so, 29.5 ms with one thread
// alone on each gap (0.18 with the nonzeros spread out, either way); 16.8M keys
// without a gap 39.5 us against 37.  Eight CTAs per SM: at 40 registers, six,
// these took 44.
constexpr int kBoundsNarrow = 32, kBoundsTile = 4096;

// ptr[l..h] = p without the whole tiles in between (whole warp)
__device__ __forceinline__ void bounds_fill(int* __restrict__ ptr, unsigned l, unsigned h, int p) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned c0 = (l + kBoundsTile - 1) / kBoundsTile * kBoundsTile, c1 = (h + 1) / kBoundsTile * kBoundsTile;
  const unsigned end = c1 > c0 ? c0 : h + 1;
  for (unsigned j = l + lane; j < end; j += 32) ptr[j] = p;
  if (c1 > c0)
    for (unsigned j = c1 + lane; j <= h; j += 32) ptr[j] = p;
}

__global__ void __launch_bounds__(256, 8)
sorted_bounds_kernel(int cnt, const unsigned* __restrict__ key, int extent, int* __restrict__ ptr, int vec_ok,
                     int tiles) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if ((int)(gridDim.x - blockIdx.x) <= tiles) {
    __shared__ int s_p;
    const unsigned j0 = (unsigned)(blockIdx.x + tiles - gridDim.x) * kBoundsTile, last = j0 + kBoundsTile - 1;
    if (threadIdx.x < 32) {
      int l = 0, r = cnt;  // the first position whose key is >= j0 is in [l, r]; 32 probes per step
      while (l < r) {
        const int span = r - l, q = l + (int)(((long long)span * lane) >> 5);
        const int c = __popc(__ballot_sync(FULL, __ldg(key + q) < j0));  // sorted: the first c are below
        const int nl = c ? l + (int)(((long long)span * (c - 1)) >> 5) + 1 : l;
        r = c < 32 ? l + (int)(((long long)span * c) >> 5) : r;
        l = nl;
      }
      if (lane == 0) s_p = l == cnt || __ldg(key + l) >= last ? l : -1;
    }
    __syncthreads();
    const int p = s_p;
    if (p < 0) return;
    for (int j = threadIdx.x; j < kBoundsTile; j += 256) ptr[j0 + j] = p;
    return;
  }
  constexpr int U = 2;
  const long long step = (long long)(gridDim.x - tiles) * blockDim.x * 4;
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  // whole warps stay in the loop: the condition is that of the warp's first lane
  for (long long b = first; b - 4 * lane <= cnt; b += U * step) {
    unsigned k[U][5];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = b + u * step;
      if (vec_ok && i + 4 <= cnt) {
        const uint4 t = __ldg(reinterpret_cast<const uint4*>(key + i));
        k[u][1] = t.x; k[u][2] = t.y; k[u][3] = t.z; k[u][4] = t.w;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) k[u][q + 1] = i + q < cnt ? __ldg(key + i + q) : (unsigned)extent;
      }
      k[u][0] = __shfl_up_sync(FULL, k[u][4], 1);
      if (lane == 0 && i > 0 && i <= cnt) k[u][0] = __ldg(key + i - 1);
    }
    // sorted: no gap of the thread is wider than all of its keys are apart
    bool wide = false;
#pragma unroll
    for (int u = 0; u < U; ++u)
      wide |= min(k[u][4], (unsigned)extent) - (b + u * step == 0 ? 0u : min(k[u][0], (unsigned)extent)) > kBoundsNarrow;
    if (!__any_sync(FULL, wide)) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const long long i = b + u * step + q;
          if (i > cnt) continue;
          const int lo = i == 0 ? 0 : (int)min(k[u][q], (unsigned)extent) + 1;
          const int hi = i == cnt ? extent : (int)min(k[u][q + 1], (unsigned)extent);
          for (int j = lo; j <= hi; ++j) ptr[j] = (int)i;
        }
      }
      continue;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long i = b + u * step + q;
        const int lo = i == 0 ? 0 : (int)min(k[u][q], (unsigned)extent) + 1;
        const int hi = i > cnt ? lo - 1 : i == cnt ? extent : (int)min(k[u][q + 1], (unsigned)extent);
        for (unsigned w = __ballot_sync(FULL, hi - lo >= kBoundsNarrow); w; w &= w - 1) {
          const int src = __ffs(w) - 1;
          bounds_fill(ptr, (unsigned)__shfl_sync(FULL, lo, src), (unsigned)__shfl_sync(FULL, hi, src),
                      (int)(i + 4 * (src - lane)));
        }
        if (hi - lo >= kBoundsNarrow) continue;
        for (int j = lo; j <= hi; ++j) ptr[j] = (int)i;
      }
    }
  }
}

int launch_sorted_bounds(int cnt, const unsigned* key, int extent, int* ptr, cudaStream_t st) {
  if (cnt <= 0) return cudaMemsetAsync(ptr, 0, 4 * ((size_t)extent + 1), st) == cudaSuccess ? 0 : -1;
  note_launch();
  const int tiles = (int)(((long long)extent + 1) / kBoundsTile);
  const int grid = (int)std::min<long long>(((long long)cnt + 1 + 2047) / 2048, 148LL * 8);
  sorted_bounds_kernel<<<tiles + grid, 256, 0, st>>>(cnt, key, extent, ptr, ((uintptr_t)key & 15u) == 0, tiles);
  return 0;
}

// ---------------------------------------------------------------------------
// reduce_by_key over sorted keys: unique keys in order and the sum of the
// values of each run.  Pass 1 finds run heads (single-pass scan of head flags)
// and writes the unique keys, zeroes the sums and records each item's output
// slot; pass 2 adds every warp-run of equal slots with one atomic.
// ---------------------------------------------------------------------------
template <int NT, int VT>
__global__ void __launch_bounds__(NT)
rbk_heads_kernel(const unsigned* __restrict__ keys, int n, int* __restrict__ slot,
                 int* __restrict__ out_key, float* __restrict__ out_val,
                 int* d_count, LookbackState st, int ntiles, int* err) {
  constexpr int NW = NT / 32;
  __shared__ unsigned s_cnt[VT * NW];
  __shared__ unsigned s_wtmp[NT / 32 + 1];
  __shared__ int s_tile;
  __shared__ unsigned s_prefix, s_total;
  const int tile = lb_acquire_tile(st, ntiles, &s_tile);
  const int base = tile * NT * VT;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  bool head[VT];
  unsigned mask[VT];
  unsigned kk[VT];
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int i = base + j * NT + tid;
    head[j] = false;
    kk[j] = 0;
    if (i < n) {
      kk[j] = __ldg(keys + i);
      head[j] = (i == 0) || (__ldg(keys + i - 1) != kk[j]);
    }
    mask[j] = __ballot_sync(0xffffffffu, head[j]);
    if (lane == 0) s_cnt[j * NW + w] = __popc(mask[j]);
  }
  __syncthreads();
  unsigned c = (tid < VT * NW) ? s_cnt[tid] : 0u;
  unsigned total;
  const unsigned ex = block_exclusive_sum<NT>(c, s_wtmp, &total);
  if (tid < VT * NW) s_cnt[tid] = ex;
  if (tid < 32) {
    const unsigned p = lb_warp_lookback(st, tile, ntiles, total, err);
    if (tid == 0) { s_prefix = p; s_total = total; }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < VT; ++j) {
    const int i = base + j * NT + tid;
    if (i < n) {
      // slot = number of heads at or before i, minus one
      const int pos = (int)(s_prefix + s_cnt[j * NW + w] +
                            __popc(mask[j] & lanemask_lt())) + (head[j] ? 0 : -1);
      slot[i] = pos;
      if (head[j]) { out_key[pos] = (int)kk[j]; out_val[pos] = 0.0f; }
    }
  }
  if (tile == ntiles - 1 && tid == 0) *d_count = (int)(s_prefix + s_total);
}

__global__ void rbk_add_kernel(const int* __restrict__ slot,
                               const float* __restrict__ vals, int n,
                               float* __restrict__ out_val) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool valid = i < n;
  const int s = valid ? __ldg(slot + i) : -1;
  float v = valid ? __ldg(vals + i) : 0.0f;
  // runs of equal slots are contiguous lanes (slots are non-decreasing);
  // a segmented suffix sum leaves each run's total in its first lane
  const unsigned same = __match_any_sync(0xffffffffu, s);
  const int first = __ffs(same) - 1;
  const int run_end = 31 - __clz(same);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float t = __shfl_down_sync(0xffffffffu, v, o);
    if (lane + o <= run_end) v += t;
  }
  if (valid && lane == first) atomicAdd(out_val + s, v);
}

int reduce_by_key_sorted(const unsigned* keys, const float* vals, int n,
                         int* slot_scratch, int* out_key, float* out_val,
                         int* d_count, ScanScratch& ls, int* err,
                         cudaStream_t st) {
  constexpr int NT = 256, VT = 8;
  if (n <= 0) { cudaMemsetAsync(d_count, 0, sizeof(int), st); return 0; }
  const int ntiles = (n + NT * VT - 1) / (NT * VT);
  if (ntiles > ls.status_len) return -1;
  LookbackState lbs{ls.status, ls.ticket};
  note_launch(2);
  rbk_heads_kernel<NT, VT><<<ntiles, NT, 0, st>>>(keys, n, slot_scratch, out_key, out_val,
                                                 d_count, lbs, ntiles, err);
  rbk_add_kernel<<<(n + 255) / 256, 256, 0, st>>>(slot_scratch, vals, n, out_val);
  return 0;
}

}  // namespace spmx
