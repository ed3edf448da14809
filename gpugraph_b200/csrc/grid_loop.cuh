// Whole traversals in one cooperative launch: a grid barrier with a bounded
// wait, the per-level totals that travel with it, and the result block the host
// reads. Used where a level's work is short beside the launches of a
// level-by-level loop (12-25 us a level on a B200, against 4 us here on a path graph
// and 7 on a road grid).
//
// The launch is cooperative (cudaLaunchCooperativeKernel), so every CTA is
// resident and a barrier only waits for CTAs that run. A wait still ends after
// mg_options.spin_limit polls: the run then stops with MG_ERR_TIMEOUT.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "common.cuh"
#include "graph.cuh"

namespace mg {

constexpr int kLoopNT = 1024;  // one CTA per SM: the fewest arrivals a barrier can have
constexpr int kRange = 256;    // edges per entry of a queue of edge ranges
// In-edges of a vertex up to which k_bfs_loop may pull it: one lane walks the list, four
// edges a step, while every other CTA polls at the barrier, 2^22 times (2 to 3 s) by
// default. A list of 2^20 edges walked to its end takes 49 ms (58 in the level loop), so
// one of 2^22 a tenth of the limit. Longer ones are left to the level loop, whose kernels
// have no time limit.
constexpr int32_t kLoopPullList = 1 << 22;

// Device state of a loop. `arrived` grows for the life of the graph (a run
// starts from the value the host passes in); the totals rotate over three
// slots, so slot L+1 can be cleared while level L runs.
struct LoopCtl {
  unsigned long long count[3];  // vertices found in a level
  unsigned long long edges[3];  // sum of their out-degrees
  uint32_t items[3];            // items appended to the next queue
  uint32_t ranges[3];           // batched BFS: edge ranges, beside the vertices counted by items
  unsigned long long mask[3];   // batched BFS: OR of the level's source masks
  int32_t low[3];               // SSSP: smallest waiting distance
  double residual[3], dangling[3];  // PageRank: L1 change and dangling mass
  uint32_t arrived;
  int32_t error;
};

// What the host reads after the launch (pinned memory, written by the kernel).
struct LoopOut {
  uint32_t level, push_levels, pull_levels, frontier_size;
  unsigned long long visited_count, visited_edges;
  double residual, norm;
  uint32_t barriers;
  int32_t error;
  int32_t timed_out;  // set by every CTA whose wait ran out
};

struct LoopShared {
  unsigned long long my_count, my_edges, my_mask;  // this CTA's totals of the level
  unsigned long long count, edges, mask;           // the grid's, after the level's barrier
  uint32_t items, ranges;
  int32_t low;
  double residual, dangling;
  int fail;
};

struct GridLoop {
  LoopCtl *c;
  uint32_t base;       // value of c->arrived when the run began
  unsigned long long spin_limit;
  LoopOut *out;
};

// End of a level: adds this CTA's totals (my_count, my_edges, my_mask, summed by its
// threads since the last call; cleared here) to slot `slot`, waits for the whole
// grid and leaves the grid's totals in sh. `n` counts the barriers of the run. False when the wait ran out.
// Data written before the barrier by any CTA is visible after it to ordinary
// loads.
MG_DEVINL bool grid_level_end(const GridLoop &g, LoopShared *sh, uint32_t slot, uint32_t &n) {
  __syncthreads();
  ++n;
  if (threadIdx.x == 0) {
    if (sh->my_count) atomicAdd(&g.c->count[slot], sh->my_count);
    if (sh->my_edges) atomicAdd(&g.c->edges[slot], sh->my_edges);
    if (sh->my_mask) atomicOr(&g.c->mask[slot], sh->my_mask);
    sh->my_count = sh->my_edges = sh->my_mask = 0;
    __threadfence();
    atomicAdd(&g.c->arrived, 1u);
    const uint32_t target = g.base + n * gridDim.x;
    unsigned long long spins = 0;
    while ((int32_t)(ld_acquire(&g.c->arrived) - target) < 0) {
      if (++spins >= g.spin_limit) {
        // reported by the CTA itself: at the last barrier CTA 0 may still get
        // through, and `error` say that all is well
        sh->fail = 1;
        *(volatile int32_t *)&g.out->timed_out = 1;
        break;
      }
    }
    // (the acquire above orders the reads below, and with the barrier at the end
    // the CTA's; a second fence here cost 0.5 us a level: R-MAT 21 BFS 111 / 97 us)
    sh->count = *(volatile unsigned long long *)&g.c->count[slot];
    sh->edges = *(volatile unsigned long long *)&g.c->edges[slot];
    sh->mask = *(volatile unsigned long long *)&g.c->mask[slot];
    sh->items = *(volatile uint32_t *)&g.c->items[slot];
    sh->ranges = *(volatile uint32_t *)&g.c->ranges[slot];
    sh->low = *(volatile int32_t *)&g.c->low[slot];
    sh->residual = *(volatile double *)&g.c->residual[slot];
    sh->dangling = *(volatile double *)&g.c->dangling[slot];
  }
  __syncthreads();
  return !sh->fail;
}

// The launch's status where the process or the stream has fewer SMs than the GPU (an
// MPS share, a green context): nothing was launched, the caller takes its
// level-by-level loop, which needs no CTA beside another.
constexpr int kLoopRefused = -1;

// One run of a loop kernel: the GPU's turn is held from here until the run's stream
// was synchronised (two loops launched by different threads would each wait for SMs
// the other one holds), by finish() or, when a call leaves in between with an error,
// by the destructor: the arrivals of every run are accounted for. What the caller's
// stream still has to do is waited for first: the turn is held for the run alone, not
// for work that may take long or depend on another thread's call.
class LoopRun {
 public:
  LoopRun(mg_graph *g, cudaStream_t s);
  ~LoopRun();
  LoopRun(const LoopRun &) = delete;
  LoopRun &operator=(const LoopRun &) = delete;
  // The kernel's GridLoop.
  GridLoop args(const mg_options *o);
  // One cooperative launch of `kernel` (one CTA per SM), between the graph's events
  // when the caller wants its time. MG_OK, an error, or kLoopRefused.
  int launch(const void *kernel, void **args, bool timed, const char *what);
  // Waits for the stream and returns the run's status; `e` is that of the work
  // queued behind the kernel.
  int finish(cudaError_t e, const char *what);

 private:
  cudaError_t settle(int *error);
  mg_graph *g_;
  cudaStream_t s_;
  std::unique_lock<std::mutex> turn_;
  bool launched_ = false;
};

// The runs below return what LoopRun::launch does.
// bfs_loop.cu: a BFS in one launch, depths to `labels` (device).
int bfs_loop_run(LoopRun &run, mg_graph *g, cudaStream_t s, const std::vector<int32_t> &roots, uint32_t max_iter,
                 const mg_options *o, int32_t *labels, bool timed);
// sssp_loop.cu: an SSSP in one launch, distances to `dist` (device).
int sssp_loop_run(LoopRun &run, mg_graph *g, int32_t src, const mg_options *o, int32_t *dist, bool timed);

}  // namespace mg
