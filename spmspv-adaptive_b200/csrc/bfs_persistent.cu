// Persistent BFS kernels: every level of a traversal inside ONE cooperative
// launch (all CTAs co-resident), levels separated by bounded grid barriers, the
// push/pull choice made on the device from frontier counters.  No host round
// trip per level.
//
// bfs_persistent_kernel: one source; levels as in the level-stepped kernels
//   of bfs.cu (push = Boolean CSC SpMSpV masked by the visited set, pull =
//   bitmap-gated CSR SpMSpV).
// msbfs_persistent_kernel: up to 64 sources at once, one bit per source in a
//   64-bit word per vertex (visited / frontier / next).  A frontier vertex
//   pushes its whole word to every neighbour (one 64-bit atomicOr), or an
//   unvisited vertex pulls the OR of its neighbours' frontier words and stops
//   once every source has reached it.  While the level fits 4 bits the levels
//   are kept bit-sliced, four 64-bit planes (one 32-byte sector) per vertex;
//   msbfs_expand_kernel turns them into the caller's layout with coalesced
//   stores.  A deeper traversal expands them at level 16 and writes the later
//   levels directly.
#include <algorithm>

#include "bfs.h"
#include "common.cuh"
#include "kernels.h"

namespace spmx {

__device__ __forceinline__ bool tbit(const unsigned* bits, int v) {
  return (bits[v >> 5] >> (v & 31)) & 1u;
}

// A warp's way into the next queue: entries collect in shared memory and are
// appended about a hundred at a time, because every append adds to one counter
// (queue length in the high word, sum of the degrees, at most nnz, in the low
// word) and atomics on one address take about 2 ns each.
constexpr int kOutFlush = 96, kOutCap = kOutFlush + 32;
template <class T>
struct WarpOut {
  T* buf;         // kOutCap entries of this warp
  int cnt;        // warp-uniform
  unsigned deg;   // the lane's share of their degrees
  T* q;
  unsigned long long* counter;

  __device__ __forceinline__ void flush() {
    if (!cnt) return;
    const int lane = threadIdx.x & 31;
    const unsigned d = __reduce_add_sync(0xffffffffu, deg);
    unsigned base = 0;
    if (lane == 0) base = (unsigned)(atomicAdd(counter, ((unsigned long long)cnt << 32) | d) >> 32);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int i = lane; i < cnt; i += 32) q[base + i] = buf[i];
    __syncwarp();
    cnt = 0;
    deg = 0;
  }
  __device__ __forceinline__ void add(bool want, T e, int d) {
    const unsigned mask = __ballot_sync(0xffffffffu, want);
    if (!mask) return;
    if (want) {
      buf[cnt + __popc(mask & lanemask_lt())] = e;
      deg += (unsigned)d;
    }
    cnt += __popc(mask);
    __syncwarp();
    if (cnt >= kOutFlush) flush();
  }
};

// Every CTA leaves through here; the last one puts the barrier back for the next
// launch (also after a barrier that gave up), so no launch clears it first.
__device__ __forceinline__ void bfs_leave(BfsCtrl* ctrl) {
  __syncthreads();
  if (threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd(&ctrl->left, 1u) != gridDim.x - 1) return;
  ctrl->bar_count = 0u;
  ctrl->abort_flag = 0;
  ctrl->left = 0u;
}

// What bounds it: L2 round trips and the grid barrier of every level.  A queue
// entry is a vertex's range of columns, looked up when it is found, beside the
// atomic that finds it, so a push level is queue -> columns -> visited bit ->
// append.  R-MAT 14 (16,384 vertices, 0.43M edges, 6 levels) 38 us, 16 43, 18 61,
// 20 (31M edges) 116, against 42, 50, 133 and 242 us with vertices in the queue
// (row bounds a round trip later on both sides), an append of two atomics per 32
// edges, and the barrier's two words on one line (which alone took 95 and 188 at
// 18 and 20).  Two edges in flight per lane instead of one, with the early exits
// after both: 41, 46, 63 and 128 us; four: 47, 52, 70 and 178.
__global__ void __launch_bounds__(256)
bfs_persistent_kernel(int n, long long total_edges, const int* __restrict__ rowptr,
                      const int* __restrict__ col, int* __restrict__ levels,
                      unsigned* visited, unsigned* fb0, unsigned* fb1, unsigned* fb2, int2* q0, int2* q1,
                      BfsCtrl* ctrl, double alpha_b, double beta_b, int src, int* err) {
  __shared__ int2 s_out[8][kOutCap];
  const GridBarrier bar{&ctrl->bar_count, &ctrl->bar_gen, &ctrl->abort_flag};
  const int lane = threadIdx.x & 31;
  const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  const long long gwarp = gtid >> 5, nwarps = nthreads >> 5;
  const long long words = (n + 31) >> 5;
  // initial state: every write goes to a distinct place, so one barrier suffices
  for (long long i = gtid; i < n; i += nthreads) levels[i] = i == src ? 0 : -1;
  for (long long w = gtid; w < words; w += nthreads) {
    const unsigned sb = w == (src >> 5) ? 1u << (src & 31) : 0u;
    visited[w] = sb;
    fb0[w] = sb;
    fb1[w] = 0u;
    fb2[w] = 0u;
  }
  if (gtid == 0) {
    q0[0] = make_int2(__ldg(rowptr + src), __ldg(rowptr + src + 1));
    for (int k = 0; k < 3; ++k) ctrl->edges[k] = 0ull;
  }
  if (!grid_sync(bar, err)) {
      bfs_leave(ctrl);
      return;
    }
  const int src_deg = __ldg(rowptr + src + 1) - __ldg(rowptr + src);
  long long nf = 1, mf = src_deg, mu = total_edges - src_deg;
  bool pull = false;
  int L = 0, cur = 0;
  unsigned* fbs[3] = {fb0, fb1, fb2};
  while (true) {
    if (!pull && (double)mf > (double)mu / alpha_b) pull = true;
    else if (pull && (double)nf < (double)n / beta_b) pull = false;
    const int nxt = cur ^ 1;
    const int slot = (L + 1) % 3;
    const int2* qc = cur ? q1 : q0;
    WarpOut<int2> out{s_out[threadIdx.x >> 5], 0, 0u, nxt ? q1 : q0, &ctrl->edges[slot]};
    // frontier bitmaps rotate over three buffers: this level reads fbs[L % 3],
    // writes fbs[(L + 1) % 3], and clears fbs[(L + 2) % 3] (the frontier of
    // the previous level, read by nobody now) for the next level; the counter
    // slot of the next level is cleared the same way.  One barrier per level.
    const unsigned* fbc = fbs[L % 3];
    unsigned* fbn = fbs[(L + 1) % 3];
    unsigned* fbr = fbs[(L + 2) % 3];
    if (L > 0)
      for (long long w = gtid; w < words; w += nthreads) fbr[w] = 0u;
    if (gtid == 0) ctrl->edges[(L + 2) % 3] = 0ull;
    if (pull) {
      for (long long vb = gwarp * 32; vb < n; vb += nwarps * 32) {
        const int v = (int)(vb + lane);
        bool found = false;
        int deg = 0, a = 0, b = 0;
        const bool open = v < n && !tbit(visited, v);
        if (open) {
          a = __ldg(rowptr + v);
          b = __ldg(rowptr + v + 1);
          deg = b - a;
        }
        const bool heavy = open && deg > 32;
        if (open && !heavy) {
          for (int k = a; k < b && !found; ++k) {
            const int u = __ldg(col + k);
            if ((unsigned)u >= (unsigned)n) flag_error(err, kDevErrOob);
            else found = tbit(fbc, u);
          }
        }
        // vertices of degree > 32: the whole warp looks for a frontier neighbour
        unsigned hm = __ballot_sync(0xffffffffu, heavy);
        while (hm) {
          const int sl = __ffs(hm) - 1;
          hm &= hm - 1;
          const int ha = __shfl_sync(0xffffffffu, a, sl), hb = __shfl_sync(0xffffffffu, b, sl);
          bool any = false;
          for (int kb = ha; kb < hb && !any; kb += 32) {
            const int k = kb + lane;
            bool hit = false;
            if (k < hb) {
              const int u = __ldg(col + k);
              if ((unsigned)u >= (unsigned)n) flag_error(err, kDevErrOob);
              else hit = tbit(fbc, u);
            }
            any = __any_sync(0xffffffffu, hit);
          }
          if (lane == sl) found = any;
        }
        if (found) {
          levels[v] = L + 1;
          atomicOr(visited + (v >> 5), 1u << (v & 31));
          atomicOr(fbn + (v >> 5), 1u << (v & 31));
        }
        out.add(found, make_int2(a, b), deg);
      }
    } else {
      // a small frontier gets several warps per vertex (equal slices of its
      // adjacency), so a hub vertex does not serialise on one warp
      const long long g = nf < nwarps ? nwarps / nf : 1;
      for (long long wi = gwarp; wi < nf * g; wi += nwarps) {
        const long long f = wi / g;
        const long long part = wi - f * g;
        const int2 e = qc[f];
        const int a = e.x + (int)(((long long)(e.y - e.x) * part) / g);
        const int b = e.x + (int)(((long long)(e.y - e.x) * (part + 1)) / g);
        for (int kb = a; kb < b; kb += 32) {
          const int k = kb + lane;
          bool win = false;
          int v = 0, va = 0, vb = 0;
          if (k < b) {
            v = __ldg(col + k);
            if ((unsigned)v >= (unsigned)n) {
              flag_error(err, kDevErrOob);
            } else if (!tbit(visited, v)) {
              const unsigned bit = 1u << (v & 31);
              win = !(atomicOr(visited + (v >> 5), bit) & bit);
              va = __ldg(rowptr + v);  // beside the atomic, whether it wins or not
              vb = __ldg(rowptr + v + 1);
              if (win) {
                levels[v] = L + 1;
                atomicOr(fbn + (v >> 5), bit);
              }
            }
          }
          out.add(win, make_int2(va, vb), vb - va);
        }
      }
    }
    out.flush();
    if (!grid_sync(bar, err)) {
      bfs_leave(ctrl);
      return;
    }
    const unsigned long long packed = *(volatile unsigned long long*)&ctrl->edges[slot];
    nf = (long long)(packed >> 32);
    mf = (long long)(packed & 0xffffffffull);
    mu -= mf;
    if (nf == 0) break;
    cur = nxt;
    ++L;
  }
  if (gtid == 0) ctrl->depth = L + 1;
  bfs_leave(ctrl);
}


// ---------------------------------------------------------------------------
// multi-source BFS, up to 64 sources
// ---------------------------------------------------------------------------
constexpr int kMsPlanes = 4;
constexpr int kMsPlaneLevels = 1 << kMsPlanes;  // levels the planes can hold

struct MsBfsState {
  int n, ns, layout;
  int* levels;
  unsigned long long *visit, *front0, *front1, *next;
  ulonglong4* planes;  // [n] level bits 0..3 of every source; valid where visit is set
};

__device__ __forceinline__ long long ms_at(const MsBfsState& t, int v, int s) {
  return t.layout ? (long long)s * t.n + v : (long long)v * t.ns + s;
}

// vertex v is reached at level `lev` by the sources nv, none of which had
// reached it before (vis: those that had)
__device__ __forceinline__ void ms_reach(const MsBfsState& t, int v, unsigned long long vis, unsigned long long nv,
                                         int lev, bool direct) {
  t.visit[v] = vis | nv;
  if (direct) {
    for (unsigned long long w = nv; w; w &= w - 1) t.levels[ms_at(t, v, __ffsll((long long)w) - 1)] = lev;
    return;
  }
  ulonglong2* p = reinterpret_cast<ulonglong2*>(t.planes + v);
  ulonglong2 a = make_ulonglong2(0ull, 0ull), b = a;
  if (vis) {  // the planes of a vertex are first written here: they need no clearing
    a = p[0];
    b = p[1];
  }
  if (lev & 1) a.x |= nv;
  if (lev & 2) a.y |= nv;
  if (lev & 4) b.x |= nv;
  if (lev & 8) b.y |= nv;
  p[0] = a;
  p[1] = b;
}

// planes -> levels (-1 where a source never came), 32 vertices per warp
__device__ __forceinline__ void ms_expand(const MsBfsState& t, long long gwarp, long long nwarps) {
  const int lane = threadIdx.x & 31;
  for (long long vb = gwarp * 32; vb < t.n; vb += nwarps * 32) {
    const int v = (int)vb + lane;
    unsigned long long vis = 0ull;
    ulonglong2 a = make_ulonglong2(0ull, 0ull), b = a;
    if (v < t.n) {
      vis = t.visit[v];
      if (vis) {
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(t.planes + v);
        a = p[0];
        b = p[1];
      }
    }
    if (t.layout) {  // lane = vertex: a warp's store covers 32 vertices of one source
      if (v >= t.n) continue;
      for (int h = 0; h < t.ns; h += 32) {
        const unsigned w = (unsigned)(vis >> h), b0 = (unsigned)(a.x >> h), b1 = (unsigned)(a.y >> h),
                       b2 = (unsigned)(b.x >> h), b3 = (unsigned)(b.y >> h);
        const int e = min(32, t.ns - h);
        int* out = t.levels + (long long)h * t.n + v;
#pragma unroll 8
        for (int s = 0; s < e; ++s, out += t.n) {
          const int lev = (int)(((b0 >> s) & 1u) | (((b1 >> s) & 1u) << 1) | (((b2 >> s) & 1u) << 2) |
                                (((b3 >> s) & 1u) << 3));
          __stcs(out, (w >> s) & 1u ? lev : -1);
        }
      }
    } else {  // lane = source: a warp's store covers one vertex
      const int cnt = (int)min(32LL, t.n - vb);
      for (int q = 0; q < cnt; ++q) {
        const unsigned long long w = __shfl_sync(0xffffffffu, vis, q), b0 = __shfl_sync(0xffffffffu, a.x, q),
                                 b1 = __shfl_sync(0xffffffffu, a.y, q), b2 = __shfl_sync(0xffffffffu, b.x, q),
                                 b3 = __shfl_sync(0xffffffffu, b.y, q);
        for (int s = lane; s < t.ns; s += 32) {
          const int lev = (int)(((b0 >> s) & 1u) | (((b1 >> s) & 1u) << 1) | (((b2 >> s) & 1u) << 2) |
                                (((b3 >> s) & 1u) << 3));
          __stcs(t.levels + (vb + q) * t.ns + s, (w >> s) & 1u ? lev : -1);
        }
      }
    }
  }
}

// edges in flight per lane: pushes and mid-degree vertices, then light vertices
// and hub chunks; a single lane pushes at most kMsLane.  Early exits are tested
// after each group, so more is not better: R-MAT 22 / 20 (20 sources), us: 2 and
// 4 1688 / 503, 2 and 2 1697 / 503, 4 and 8 1875 / 607, 1 and 1 1981 / 605
constexpr int kMsU = 2, kMsHubU = 4, kMsLane = 8;

// pushes the word fu over the edges [a, b) (whole warp)
__device__ __forceinline__ void ms_push(const MsBfsState& t, const int* __restrict__ rowptr,
                                        const int* __restrict__ col, int a, int b, unsigned long long fu,
                                        WarpOut<int>& out, int* err) {
  const int lane = threadIdx.x & 31;
  for (int kb = a; kb < b; kb += 32 * kMsU) {
    int v[kMsU];
    unsigned long long nv[kMsU];
#pragma unroll
    for (int j = 0; j < kMsU; ++j) {
      const int k = kb + 32 * j + lane;
      v[j] = k < b ? __ldg(col + k) : -1;
      if (k < b && (unsigned)v[j] >= (unsigned)t.n) {
        flag_error(err, kDevErrOob);
        v[j] = -1;
      }
    }
#pragma unroll
    for (int j = 0; j < kMsU; ++j) {
      nv[j] = 0ull;
      if (v[j] >= 0) {
        // a plain read of next first: most edges into a hub add nothing, and
        // atomics on one address serialise
        nv[j] = fu & ~t.visit[v[j]];
        if (!(nv[j] & ~*(volatile unsigned long long*)(t.next + v[j]))) nv[j] = 0ull;
      }
    }
#pragma unroll
    for (int j = 0; j < kMsU; ++j) {
      bool add = false;
      int deg = 0;
      if (nv[j]) {
        add = atomicOr(t.next + v[j], nv[j]) == 0ull;
        if (add) deg = __ldg(rowptr + v[j] + 1) - __ldg(rowptr + v[j]);
      }
      out.add(add, v[j], deg);
    }
  }
}

// OR of the frontier words over the edges [a, b), until it has every bit
// missing from vis (whole warp)
template <int U>
__device__ __forceinline__ unsigned long long ms_pull(const unsigned long long* fc, const int* __restrict__ col,
                                                      int n, int a, int b, unsigned long long vis,
                                                      unsigned long long full, int* err) {
  const int lane = threadIdx.x & 31;
  unsigned long long acc = 0ull;
  for (int kb = a; kb < b; kb += 32 * U) {
    int u[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int k = kb + 32 * j + lane;
      u[j] = k < b ? __ldg(col + k) : -1;
      if (k < b && (unsigned)u[j] >= (unsigned)n) {
        flag_error(err, kDevErrOob);
        u[j] = -1;
      }
    }
#pragma unroll
    for (int j = 0; j < U; ++j)
      if (u[j] >= 0) acc |= fc[u[j]];
    const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)acc),
                   hi = __reduce_or_sync(0xffffffffu, (unsigned)(acc >> 32));
    acc = ((unsigned long long)hi << 32) | lo;
    if ((acc | vis) == full) break;
  }
  return acc;
}

// What bounds it: the gathers of the frontier words in the two heavy pull levels
// (one 32-byte L2 sector per edge) and their latency.  64 sources on R-MAT 22
// (4.2M vertices, 128M edges), expansion included: 1.7 ms (the two pull levels
// 1.2, the first push 0.18, expansion 0.23), against 15.7 ms with level
// stores per vertex and a strided transposition (1.7 + 5.0 ms), hubs of up to
// 10^5 edges on four warps each (one push level 8.8 ms) and one dependent
// chain per 32 edges (first pull level 3.2 ms).
__global__ void __launch_bounds__(256)
msbfs_persistent_kernel(MsBfsState t, long long total_edges, double alpha_ms, const int* __restrict__ rowptr,
                        const int* __restrict__ col, int* q0, int* q1, BfsCtrl* ctrl, HubChunks hub, int* err) {
  const GridBarrier bar{&ctrl->bar_count, &ctrl->bar_gen, &ctrl->abort_flag};
  __shared__ int s_out[8][kOutCap];
  const unsigned long long FULL = t.ns >= 64 ? ~0ull : ((1ull << t.ns) - 1ull);
  const int n = t.n;
  const int lane = threadIdx.x & 31;
  const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  const long long gwarp = gtid >> 5, nwarps = nthreads >> 5;
  // the first frontier (written by msbfs_init_kernel into slot 0)
  unsigned long long packed = *(volatile unsigned long long*)&ctrl->edges[0];
  long long nq = (long long)(packed >> 32), mf = (long long)(packed & 0xffffffffull);
  int L = 0, cur = 0;
  bool direct = false;
  while (true) {
    if (L + 1 == kMsPlaneLevels) {  // the next level does not fit the planes
      ms_expand(t, gwarp, nwarps);
      if (gtid == 0) ctrl->pad = 1;
      if (!grid_sync(bar, err)) {
      bfs_leave(ctrl);
      return;
    }
      direct = true;
    }
    const bool pull = (double)mf > (double)total_edges / alpha_ms;
    const int nxt = cur ^ 1;
    unsigned long long* counter = &ctrl->edges[(L + 1) % 3];
    int* qn = nxt ? q1 : q0;
    const int* qc = cur ? q1 : q0;
    WarpOut<int> out{s_out[threadIdx.x >> 5], 0, 0u, qn, counter};
    const unsigned long long* fc = cur ? t.front1 : t.front0;
    unsigned long long* fn = nxt ? t.front1 : t.front0;
    if (pull) {
      // only v's own words are written, so a vertex is finished on the spot
      for (long long vb = gwarp * 32; vb < n; vb += nwarps * 32) {
        const int v = (int)(vb + lane);
        int a = 0, b = 0;
        unsigned long long vis = FULL;
        if (v < n) {
          vis = t.visit[v];
          a = __ldg(rowptr + v);
          b = __ldg(rowptr + v + 1);
        }
        // hubs (degree > hub.deg) are pulled chunk by chunk below
        const bool open = vis != FULL && b - a <= hub.deg;
        const bool heavy = open && b - a > 32;
        unsigned long long nv = 0ull;
        if (open && !heavy) {
          unsigned long long acc = 0ull;
          for (int k = a; k < b && (acc | vis) != FULL; k += kMsHubU) {
            int u[kMsHubU];
#pragma unroll
            for (int j = 0; j < kMsHubU; ++j) {
              u[j] = k + j < b ? __ldg(col + k + j) : -1;
              if (k + j < b && (unsigned)u[j] >= (unsigned)n) {
                flag_error(err, kDevErrOob);
                u[j] = -1;
              }
            }
#pragma unroll
            for (int j = 0; j < kMsHubU; ++j)
              if (u[j] >= 0) acc |= fc[u[j]];
          }
          nv = acc & ~vis;
        }
        // vertices of degree > 32: the whole warp pulls, one vertex at a time
        unsigned hm = __ballot_sync(0xffffffffu, heavy);
        while (hm) {
          const int sl = __ffs(hm) - 1;
          hm &= hm - 1;
          const unsigned long long acc =
              ms_pull<kMsU>(fc, col, n, __shfl_sync(0xffffffffu, a, sl), __shfl_sync(0xffffffffu, b, sl),
                      __shfl_sync(0xffffffffu, vis, sl), FULL, err);
          if (lane == sl) nv = acc & ~vis;
        }
        if (nv) {
          fn[v] = nv;
          ms_reach(t, v, vis, nv, L + 1, direct);
        }
        out.add(nv != 0ull, v, b - a);
      }
      // hub chunks, spread over all warps: each ORs its slice of a hub's
      // neighbours into the hub's accumulator, unless that has every missing
      // bit already; the hubs are finished after the barrier.  The next
      // chunk's descriptor and words are in flight meanwhile.
      int4 ch = make_int4(0, 0, 0, 0);  // {vertex, first edge, end edge, hub index}
      unsigned long long have = 0ull;
      if (gwarp < hub.nchunks) {
        ch = hub.chunk[gwarp];
        have = t.visit[ch.x];
      }
      for (long long c = gwarp; c < hub.nchunks; c += nwarps) {
        int4 nch = ch;
        if (c + nwarps < hub.nchunks) nch = hub.chunk[c + nwarps];
        // other warps add to the accumulator meanwhile: one lane's reading of it
        // decides for the warp, which goes through full-mask reductions below
        unsigned long long got = 0ull;
        if (lane == 0) got = have | *(volatile unsigned long long*)(hub.acc + ch.w);
        got = __shfl_sync(0xffffffffu, got, 0);
        if (got != FULL) {
          const unsigned long long acc = ms_pull<kMsHubU>(fc, col, n, ch.y, ch.z, have, FULL, err);
          if (lane == 0 && (acc & ~got)) atomicOr(hub.acc + ch.w, acc);
        }
        ch = nch;
        have = t.visit[ch.x];
      }
    } else {
      // frontier vertices up to hub.deg edges, several warps each while the
      // frontier is small; hubs of the frontier chunk by chunk
      if (nq > nwarps * 4) {
        // a lane per vertex: those of at most kMsLane edges push them by themselves
        for (long long fb = gwarp * 32; fb < nq; fb += nwarps * 32) {
          int a = 0, b = 0;
          unsigned long long fu = 0ull;
          if (fb + lane < nq) {
            const int u = qc[fb + lane];
            a = __ldg(rowptr + u);
            b = __ldg(rowptr + u + 1);
            fu = fc[u];
          }
          const bool small = b - a <= kMsLane;
          for (int j = 0; __any_sync(0xffffffffu, small && a + j < b); ++j) {
            bool add = false;
            int v = 0, deg = 0;
            if (small && a + j < b) {
              v = __ldg(col + a + j);
              if ((unsigned)v >= (unsigned)n) {
                flag_error(err, kDevErrOob);
              } else {
                const unsigned long long nv = fu & ~t.visit[v];
                if (nv & ~*(volatile unsigned long long*)(t.next + v)) add = atomicOr(t.next + v, nv) == 0ull;
                if (add) deg = __ldg(rowptr + v + 1) - __ldg(rowptr + v);
              }
            }
            out.add(add, v, deg);
          }
          for (unsigned hm = __ballot_sync(0xffffffffu, !small && b - a <= hub.deg); hm; hm &= hm - 1) {
            const int sl = __ffs(hm) - 1;
            ms_push(t, rowptr, col, __shfl_sync(0xffffffffu, a, sl), __shfl_sync(0xffffffffu, b, sl),
                    __shfl_sync(0xffffffffu, fu, sl), out, err);
          }
        }
      } else {
        const long long g = min(8LL, nq < nwarps ? nwarps / nq : 1LL);
        for (long long wi = gwarp; wi < nq * g; wi += nwarps) {
          const long long f = wi / g;
          const long long part = wi - f * g;
          const int u = qc[f];
          const int a0 = __ldg(rowptr + u), b0 = __ldg(rowptr + u + 1);
          if (b0 - a0 > hub.deg) continue;
          ms_push(t, rowptr, col, a0 + (int)(((long long)(b0 - a0) * part) / g),
                  a0 + (int)(((long long)(b0 - a0) * (part + 1)) / g), fc[u], out, err);
        }
      }
      // a lane per chunk to find the frontier's; a hub's chunks go to as many warps
      for (long long cb = 0; cb < hub.nchunks; cb += nwarps * 32) {
        const long long c = cb + (long long)lane * nwarps + gwarp;
        int4 ch = make_int4(0, 0, 0, 0);
        unsigned long long fu = 0ull;
        if (c < hub.nchunks) {
          ch = hub.chunk[c];
          fu = fc[ch.x];
        }
        for (unsigned hm = __ballot_sync(0xffffffffu, fu != 0ull); hm; hm &= hm - 1) {
          const int sl = __ffs(hm) - 1;
          ms_push(t, rowptr, col, __shfl_sync(0xffffffffu, ch.y, sl), __shfl_sync(0xffffffffu, ch.z, sl),
                  __shfl_sync(0xffffffffu, fu, sl), out, err);
        }
      }
    }
    out.flush();
    if (!grid_sync(bar, err)) {
      bfs_leave(ctrl);
      return;
    }
    // retire the current frontier
    for (long long f = gtid; f < nq; f += nthreads) ((unsigned long long*)fc)[qc[f]] = 0ull;
    const long long nn = (long long)(*(volatile unsigned long long*)counter >> 32);  // before the pulled hubs
    if (pull) {
      // finish the hubs, and clear their accumulators for the next pull level
      for (long long ib = gwarp * 32; ib < hub.nhubs; ib += nwarps * 32) {
        const int i = (int)ib + lane;
        int v = 0, deg = 0;
        unsigned long long nv = 0ull;
        if (i < hub.nhubs) {
          v = hub.vertex[i];
          const unsigned long long vis = t.visit[v];
          nv = hub.acc[i] & ~vis;
          hub.acc[i] = 0ull;
          if (nv) {
            fn[v] = nv;
            ms_reach(t, v, vis, nv, L + 1, direct);
            deg = __ldg(rowptr + v + 1) - __ldg(rowptr + v);
          }
        }
        out.add(nv != 0ull, v, deg);
      }
      out.flush();
    } else if (nn * 8 > n) {
      // finish the pushed vertices; many: in index order, coalesced
      for (long long v = gtid; v < n; v += nthreads) {
        const unsigned long long w = t.next[v];
        if (!w) continue;
        const unsigned long long vis = t.visit[v], nv = w & ~vis;
        t.next[v] = 0ull;
        fn[v] = nv;
        ms_reach(t, (int)v, vis, nv, L + 1, direct);
      }
    } else {
      for (long long f = gtid; f < nn; f += nthreads) {
        const int v = qn[f];
        const unsigned long long vis = t.visit[v], nv = t.next[v] & ~vis;
        t.next[v] = 0ull;
        fn[v] = nv;
        ms_reach(t, v, vis, nv, L + 1, direct);
      }
    }
    if (gtid == 0) ctrl->edges[(L + 2) % 3] = 0ull;
    if (!grid_sync(bar, err)) {
      bfs_leave(ctrl);
      return;
    }
    packed = *(volatile unsigned long long*)counter;
    nq = (long long)(packed >> 32);
    mf = (long long)(packed & 0xffffffffull);
    if (nq == 0) break;
    cur = nxt;
    ++L;
  }
  if (gtid == 0) ctrl->depth = L + 1;
  bfs_leave(ctrl);
}

__global__ void __launch_bounds__(256) msbfs_expand_kernel(MsBfsState t, const BfsCtrl* ctrl) {
  if (ctrl->pad) return;  // a deep traversal has written its levels
  ms_expand(t, ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, ((long long)gridDim.x * blockDim.x) >> 5);
}

// sources: distinct vertices enter the first frontier once, a vertex shared by
// several sources carries all their bits.  One thread per source.
__global__ void __launch_bounds__(64)
msbfs_init_kernel(MsBfsState t, MsSources srcs, const int* __restrict__ rowptr, int* q0, BfsCtrl* ctrl) {
  __shared__ int s_v[64];
  const int s = threadIdx.x;
  const int v = s < t.ns ? srcs.v[s] : -1;
  const bool ok = (unsigned)v < (unsigned)t.n;
  s_v[s] = ok ? v : -1;
  if (s < 3) ctrl->edges[s] = 0ull;
  if (s == 3) ctrl->pad = 0;
  __syncthreads();
  unsigned long long bits = 0ull;
  bool first = ok;
  if (ok) {
    for (int q = 0; q < t.ns; ++q) {
      if (s_v[q] != v) continue;
      bits |= 1ull << q;
      first = first && q >= s;
    }
  }
  if (first) {
    t.front0[v] = bits;
    ms_reach(t, v, 0ull, bits, 0, false);
  }
  if (first) {
    const unsigned d = (unsigned)(__ldg(rowptr + v + 1) - __ldg(rowptr + v));
    q0[(unsigned)(atomicAdd(&ctrl->edges[0], (1ull << 32) | d) >> 32)] = v;
  }
}

// --------------------------------------------------------------------------
// Co-resident grid for a cooperative launch, scaled to the work: every CTA
// joins every grid barrier, so a small graph gets few CTAs (one per SM down
// to 1024 vertices per CTA) and a large one the whole resident capacity.
template <class K>
static int coop_grid(K kernel, int num_sms, int min_ctas, long long work_items) {
  // the occupancy query costs host time on every launch otherwise; one value
  // per kernel (the same on every GPU of a node)
  static int per = -1;
  if (per < 0) {
    int p = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, kernel, 256, 0) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    per = p;
  }
  const long long cap = (long long)per * num_sms;
  long long want = (work_items + 255) / 256;
  if (want < min_ctas) want = min_ctas;
  if (want > cap) want = cap;
  return (int)want;
}

int launch_bfs_persistent(const BfsPersistentArgs& a, cudaStream_t st) {
  // small graphs get few CTAs: the level barriers then cost less
  const int grid = coop_grid(bfs_persistent_kernel, a.num_sms, 16, a.n);
  if (grid <= 0) return -1;
  note_launch();
  int n = a.n;
  long long te = a.total_edges;
  const int* rp = a.rowptr;
  const int* cl = a.col;
  int* lv = a.levels;
  unsigned* vis = a.visited;
  unsigned* f0 = a.fb0;
  unsigned* f1 = a.fb1;
  unsigned* f2 = a.fb2;
  int2* q0 = a.q0;
  int2* q1 = a.q1;
  BfsCtrl* ctrl = a.ctrl;
  double al = a.alpha, be = a.beta;
  int src = a.src;
  int* err = a.err;
  void* args[] = {&n, &te, &rp, &cl, &lv, &vis, &f0, &f1, &f2, &q0, &q1, &ctrl, &al, &be, &src, &err};
  cudaError_t e = cudaLaunchCooperativeKernel((void*)bfs_persistent_kernel, grid, 256, args, 0, st);
  return e == cudaSuccess ? 0 : -2;
}

// chunks of hub.deg edges of every vertex of degree > hub.deg
__global__ void hub_chunks_kernel(int n, const int* __restrict__ rowptr, int deg_cut, int4* chunk,
                                  int* vertex, int* counters, int max_hubs, int max_chunks) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int a = __ldg(rowptr + v), b = __ldg(rowptr + v + 1);
    if (b - a <= deg_cut) continue;
    const int nch = (b - a + deg_cut - 1) / deg_cut;
    const int hi = atomicAdd(counters, 1);
    const int base = atomicAdd(counters + 1, nch);
    if (hi >= max_hubs || base + nch > max_chunks) continue;  // cannot happen by the bounds
    vertex[hi] = v;
    for (int j = 0; j < nch; ++j)
      chunk[base + j] = make_int4(v, a + j * deg_cut, min(b, a + (j + 1) * deg_cut), hi);
  }
}

int launch_hub_chunks(int n, const int* rowptr, int deg_cut, int4* chunk, int* vertex,
                      int* counters, int max_hubs, int max_chunks, cudaStream_t st) {
  if (n <= 0) return 0;
  note_launch();
  hub_chunks_kernel<<<std::min((n + 255) / 256, 148 * 8), 256, 0, st>>>(n, rowptr, deg_cut, chunk, vertex,
                                                                       counters, max_hubs, max_chunks);
  return 0;
}

int launch_msbfs(const MsBfsArgs& a, cudaStream_t st) {
  const int grid = coop_grid(msbfs_persistent_kernel, a.num_sms, a.num_sms, a.n);
  if (grid <= 0) return -1;
  MsBfsState t{a.n, a.ns, a.layout, a.levels, a.visit, a.front0, a.front1, a.next, a.planes};
  note_launch(3);
  msbfs_init_kernel<<<1, 64, 0, st>>>(t, a.srcs, a.rowptr, a.q0, a.ctrl);
  long long te = a.total_edges;
  double al = a.alpha;
  const int* rp = a.rowptr;
  const int* cl = a.col;
  int* q0 = a.q0;
  int* q1 = a.q1;
  BfsCtrl* ctrl = a.ctrl;
  HubChunks hub = a.hub;
  int* err = a.err;
  void* args[] = {&t, &te, &al, &rp, &cl, &q0, &q1, &ctrl, &hub, &err};
  if (cudaLaunchCooperativeKernel((void*)msbfs_persistent_kernel, grid, 256, args, 0, st) != cudaSuccess) return -2;
  const int egrid = (int)std::min<long long>(((long long)a.n + 255) / 256, (long long)a.num_sms * 32);
  msbfs_expand_kernel<<<egrid, 256, 0, st>>>(t, a.ctrl);
  return 0;
}

}  // namespace spmx
