// BFS launchers (bfs.cu).
#pragma once
#include <cuda_runtime.h>

namespace spmx {

// device control block of the persistent BFS kernels (zeroed once)
struct BfsCtrl {
  unsigned long long edges[3];   // next frontier by level % 3: size << 32 | sum of the degrees
  // grid barrier: arrivals on one line, what the waiting CTAs poll on another
  unsigned bar_count, gap0[31];
  unsigned bar_gen, gap1[31];
  int abort_flag;
  unsigned left;                 // CTAs that have left the kernel
  int depth;                     // number of levels, written at the end
  int pad;                       // multi-source: levels already expanded
};

struct BfsPersistentArgs {
  int n, src, num_sms;
  long long total_edges;
  const int* rowptr;
  const int* col;
  int* levels;
  unsigned* visited;
  unsigned* fb0;
  unsigned* fb1;
  unsigned* fb2;
  int2* q0;  // [n] ranges of columns
  int2* q1;
  BfsCtrl* ctrl;
  double alpha, beta;  // direction switch: push->pull when m_f > m_u/alpha,
                       // pull->push when n_f < n/beta
  int* err;
};

// Hubs of the multi-source BFS: every vertex of degree > deg is cut into
// chunks of deg edges that all warps share; acc holds per-hub OR accumulators
// of a pull level, zero between levels.
struct HubChunks {
  const int4* chunk;     // {vertex, first edge, end edge, hub index}
  long long nchunks;
  const int* vertex;     // [nhubs]
  unsigned long long* acc;
  int nhubs;
  int deg;
};

struct MsSources {
  int v[64];
};

struct MsBfsArgs {
  int n, ns, layout, num_sms;
  long long total_edges;
  double alpha;        // pull when the frontier's edges exceed total/alpha
  MsSources srcs;      // by value: no copy to the device
  const int* rowptr;
  const int* col;
  int* levels;         // device [n * ns], layout 1: [s][v], 0: [v][s]
  unsigned long long* visit;   // the four arrays start zeroed
  unsigned long long* front0;
  unsigned long long* front1;
  unsigned long long* next;
  ulonglong4* planes;  // [n]
  int* q0;
  int* q1;
  BfsCtrl* ctrl;
  HubChunks hub;
  int* err;
};

int launch_hub_chunks(int n, const int* rowptr, int deg_cut, int4* chunk, int* vertex,
                      int* counters, int max_hubs, int max_chunks, cudaStream_t st);
int launch_bfs_persistent(const BfsPersistentArgs& a, cudaStream_t st);
int launch_msbfs(const MsBfsArgs& a, cudaStream_t st);

int launch_bfs_init(int src, int* levels, unsigned* visited, int* q,
                    int* q_count, cudaStream_t st);
int launch_bfs_push(int nf, const int* queue, int n, const int* rowptr,
                    const int* col, unsigned* visited, int* levels,
                    int next_level, int* q_next, int* q_next_count,
                    unsigned long long* next_edges, int* err, int max_grid,
                    cudaStream_t st);
int launch_bfs_pull(int n, const int* rowptr, const int* col, unsigned* visited,
                    const unsigned* front, int* levels, int next_level,
                    int* q_next, int* q_next_count,
                    unsigned long long* next_edges, int* err, int max_grid,
                    cudaStream_t st);

}  // namespace spmx
