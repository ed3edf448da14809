// Single-source SSSP in one cooperative launch (grid_loop.cuh), by distance
// windows. done[v] is the distance at which v's edges were last relaxed; v waits
// while its distance is smaller. A step selects the waiting vertices below the
// window's end (the smallest waiting distance plus `delta`), turns them into edge
// ranges, and relaxes the ranges: an improving candidate lowers the head's
// distance without waiting for the result, and that is all an edge writes (on large
// graphs a flag as well, kSpWide). With
// non-negative weights the smallest waiting distance is final, so every step
// settles a vertex and V steps suffice; the fixpoint is the one of the
// level-by-level loop (sssp.cu), the unique shortest distances.
//
// Why windows: on a power-law graph relaxing every pending vertex per level
// expands 3.0 times the edges (R-MAT 17, weights 1..64, simulated), a window of
// a few weights 1.3 to 1.9 times. It takes two to four times as many steps,
// which only pays with steps as cheap as here (two grid barriers and no scan;
// the level loop lost by it: 4.7 against 3.3 ms at R-MAT 22). R-MAT 21: 1.8 ms a
// run level by level, 1.2 here. 0.8 ms of it are three steps that relax 1.9 times
// the edges at 150 G/s, bound by the gathers and reductions in L2.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "algo_util.cuh"
#include "gas/driver.cuh"
#include "gas/programs.cuh"
#include "grid_loop.cuh"

namespace mg {

constexpr int kSpU = 8;        // edges per lane in flight (R-MAT 21: 1.30 ms a run against 1.38 with 4)
constexpr int kSpVerts = 8;    // vertices per lane and step of the selection (R-MAT 21: 1.21 ms, 1.40 with 4)
// Window: this many times the largest weight over the mean degree (with uniform
// weights a vertex has about that many edges inside it). R-MAT 21, weights
// 1..64: 1.21 ms a run at 4, 1.33 at 8; with a pending bitmap, before done[], 1.39
// at 2, 1.38 at 4, 1.44 at 8, 1.52 at 32 (no window in effect).
constexpr double kSsspWindow = 4.0;

constexpr uint32_t kSpBlock = 32 * kSpVerts;  // vertices a warp step selects from
// Vertices from which the selection looks only into blocks in which one may wait, by a
// flag per block that an improving edge sets (WIDE): the two arrays it reads (8 bytes a
// vertex) are larger than L2 then, and every step read them whole. With the flags /
// without / level by level: R-MAT 24 with a path of 2000 vertices attached 20.8 / 58.3 /
// 35.4 ms, 6000x6000 lattice, weights 1..1000, 162 / 716 / 1131, with shortcuts and
// weights 1 7.6 / 8.9 / 7.5, R-MAT 24, weights 1..64, 7.1 / 7.3 / 11.7. With 9 M vertices
// (3000x3000, weights 1) the flags still lose, 2.4 / 2.1 ms.
constexpr int64_t kSpWide = 3ll << 22;

struct SsspLoopArgs {
  DevCsr g;
  int32_t *dist;
  int32_t *done;
  uint8_t *open;  // per block of kSpBlock vertices: one of them may wait (WIDE)
  int4 *q;       // (first edge, length, distance of the tail, unused)
  uint32_t cap;  // entries of q
  int32_t src, delta;
  uint32_t max_iter;
  GridLoop loop;
};

template <bool WIDE>
__global__ void __launch_bounds__(kLoopNT, 1) k_sssp_loop(SsspLoopArgs a) {
  constexpr int32_t INF = programs::sssp::INIT_VALUE;
  __shared__ LoopShared sh;
  __shared__ int s_min;
  const int lane = lane_id();
  const uint32_t V = (uint32_t)a.g.V;
  const uint32_t tid = blockIdx.x * kLoopNT + threadIdx.x, nt = gridDim.x * kLoopNT;
  const uint32_t nw = nt / 32, gw = warp_id() * gridDim.x + blockIdx.x;
  const int32_t *ro = a.g.row_offsets, *col = a.g.col, *wgt = a.g.wgt;
  LoopCtl *c = a.loop.c;
  if (threadIdx.x == 0) {
    sh.my_count = sh.my_edges = sh.my_mask = 0;
    sh.fail = 0;
    s_min = INT_MAX;
  }
  __syncthreads();
  for (uint32_t i = tid; i < V; i += nt) {
    a.dist[i] = i == (uint32_t)a.src ? 0 : INF;
    a.done[i] = INF;
  }
  if (WIDE)
    for (uint32_t i = tid; i < (V + kSpBlock - 1) / kSpBlock; i += nt) a.open[i] = i == (uint32_t)a.src / kSpBlock;
  if (blockIdx.x == 0 && threadIdx.x < 3) {
    c->count[threadIdx.x] = c->edges[threadIdx.x] = 0;
    c->items[threadIdx.x] = 0;
    c->low[threadIdx.x] = INT_MAX;
    if (threadIdx.x == 0) c->error = 0;
  }
  uint32_t nbar = 0, step = 0;
  bool ok = grid_level_end(a.loop, &sh, 2, nbar);
  int low = 0;  // smallest waiting distance
  while (ok && low != INT_MAX && step < a.max_iter) {
    const uint32_t slot = step % 3;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      c->items[(step + 1) % 3] = 0;
      c->low[(step + 1) % 3] = INT_MAX;
    }
    const int end = (int)min((long long)INT_MAX - 1, (long long)low + a.delta);
    int rest = INT_MAX;  // smallest waiting distance past the window
    // selection from the block at v0: 32 * kSpVerts vertices (two coalesced streams);
    // whether one is left waiting
    auto select = [&](uint32_t v0) {
      int d[kSpVerts], n[kSpVerts], b[kSpVerts];
      uint32_t sel = 0;  // bit k: the lane's k-th vertex is selected
      bool left = false;
#pragma unroll
      for (int k = 0; k < kSpVerts; ++k) {
        const uint32_t v = v0 + 32 * k + lane;
        d[k] = v < V ? __ldcg(&a.dist[v]) : INT_MAX;
        n[k] = v < V ? a.done[v] : 0;
      }
#pragma unroll
      for (int k = 0; k < kSpVerts; ++k)
        if (d[k] < n[k]) {
          if (d[k] < end) sel |= 1u << k;
          else rest = min(rest, d[k]), left = true;
        }
      if (!__any_sync(0xffffffffu, sel != 0u)) return left;
#pragma unroll
      for (int k = 0; k < kSpVerts; ++k) {
        const uint32_t v = v0 + 32 * k + lane;
        b[k] = n[k] = 0;
        if ((sel >> k) & 1u) {
          a.done[v] = d[k];
          b[k] = ro[v];
          n[k] = ro[v + 1];
        }
      }
      uint32_t need = 0;
#pragma unroll
      for (int k = 0; k < kSpVerts; ++k) {
        n[k] -= b[k];
        need += (uint32_t)(n[k] + kRange - 1) / kRange;
      }
      const uint32_t inc = warp_inclusive_sum(need);
      uint32_t at = 0;
      if (lane == 31 && inc) at = atomicAdd(&c->items[slot], inc);
      at = __shfl_sync(0xffffffffu, at, 31) + inc - need;
      if (at + need > a.cap) {
        atomicCAS(&c->error, 0, (int)MG_ERR_OVERFLOW);
      } else {
#pragma unroll
        for (int k = 0; k < kSpVerts; ++k)
          for (int i = 0; i < n[k]; i += kRange)
            a.q[at++] = make_int4(b[k] + i, min(kRange, n[k] - i), d[k], 0);
      }
      return left;
    };
    if (!WIDE) {
      for (uint32_t v0 = gw * kSpBlock; v0 < V; v0 += nw * kSpBlock) select(v0);
    } else {
      // the flags of 32 of the warp's blocks at a time
      const uint32_t blocks = (V + kSpBlock - 1) / kSpBlock;
      for (uint32_t b0 = gw; b0 < blocks; b0 += nw * 32) {
        const uint32_t mine = b0 + lane * nw;
        const bool waits = mine < blocks && __ldcg(&a.open[mine]);
        for (uint32_t todo = __ballot_sync(0xffffffffu, waits); todo; todo &= todo - 1) {
          const uint32_t blk = b0 + (__ffs(todo) - 1) * nw;
          const bool left = __any_sync(0xffffffffu, select(blk * kSpBlock));
          if (lane == 0 && !left) a.open[blk] = 0;
        }
      }
    }
    rest = __reduce_min_sync(0xffffffffu, rest);
    if (lane == 0 && rest != INT_MAX) atomicMin(&s_min, rest);
    if (!(ok = grid_level_end(a.loop, &sh, slot, nbar))) break;
    // relaxation of the selected ranges
    const uint32_t n = sh.items;
    // ranges are dealt one by one over the warps (a hub's full ranges are
    // neighbours in the queue: in blocks of 32 they would land on a few warps)
    const uint32_t per = min(32u, (n + nw - 1) / nw);
    int best = INT_MAX;  // smallest distance written
    for (uint32_t base = gw; base < n; base += nw * per) {
      int4 r = make_int4(0, 0, 0, 0);
      if (lane < (int)per && base + lane * nw < n) r = __ldcg(&a.q[base + lane * nw]);
      const int inc = warp_inclusive_sum(r.y);
      const int total = __shfl_sync(0xffffffffu, inc, 31);
      const int off = r.x - (inc - r.y);
      for (int t = 0; t < total; t += 32 * kSpU) {
        int u[kSpU], cand[kSpU], dv[kSpU];
#pragma unroll
        for (int k = 0; k < kSpU; ++k) {
          const int p = t + 32 * k + lane;
          int own = 0;  // the first range that ends past p
          if (per > 1) {
#pragma unroll
            for (int s = 16; s > 0; s >>= 1)
              if (__shfl_sync(0xffffffffu, inc, own + s - 1) <= p) own += s;
            own = min(own, 31);
          }
          const int e = __shfl_sync(0xffffffffu, off, own) + p;
          const int du = __shfl_sync(0xffffffffu, r.z, own);
          const bool in = p < total && (unsigned)e < (unsigned)a.g.E;
          u[k] = in ? __ldcs(col + e) : -1;
          cand[k] = in ? du + __ldcs(wgt + e) : 0;
        }
#pragma unroll
        for (int k = 0; k < kSpU; ++k) dv[k] = (unsigned)u[k] < V ? __ldcg(&a.dist[u[k]]) : INT_MIN;
#pragma unroll
        for (int k = 0; k < kSpU; ++k)
          if (cand[k] < dv[k]) {
            atomicMin(&a.dist[u[k]], cand[k]);
            if (WIDE) a.open[(uint32_t)u[k] / kSpBlock] = 1;
            best = min(best, cand[k]);
          }
      }
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if (lane == 0 && best != INT_MAX) atomicMin(&s_min, best);
    __syncthreads();
    if (threadIdx.x == 0) {
      if (s_min != INT_MAX) atomicMin(&c->low[slot], s_min);
      s_min = INT_MAX;
    }
    if (!(ok = grid_level_end(a.loop, &sh, slot, nbar))) break;
    low = sh.low;
    ++step;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    LoopOut *o = a.loop.out;
    o->level = o->push_levels = step;
    o->pull_levels = 0;
    o->frontier_size = low != INT_MAX ? 1u : 0u;
    o->visited_count = o->visited_edges = 0;
    o->barriers = nbar;
    o->error = ok ? *(volatile int32_t *)&c->error : (int32_t)MG_ERR_TIMEOUT;
  }
}

int sssp_loop_run(LoopRun &run, mg_graph *g, int32_t src, const mg_options *o, int32_t *dist, bool timed) {
  SsspLoopArgs a;
  a.g = g->csr;
  a.dist = dist;
  a.done = g->ws.vbuf[1];
  a.open = reinterpret_cast<uint8_t *>(g->ws.queue[0]);  // (a level loop's queue, free here)
  // the room of the two BFS queues: a step selects every vertex at most once
  static_assert(sizeof(int4) == 2 * sizeof(int2), "one queue of the same number of entries");
  a.q = reinterpret_cast<int4 *>(g->loop_queue);
  a.cap = (uint32_t)g->loop_cap;
  a.src = src;
  const double mean = std::max(1.0, (double)g->edges / (double)g->nodes);
  a.delta = (int32_t)std::min(1e9, std::max(1.0, kSsspWindow * (double)std::max(g->weight_max, 0) / mean));
  a.max_iter = (uint32_t)(g->nodes + 2);
  a.loop = run.args(o);
  void *args[] = {&a};
  const void *kernel = g->nodes >= kSpWide ? (const void *)k_sssp_loop<true> : (const void *)k_sssp_loop<false>;
  return run.launch(kernel, args, timed, "sssp loop launch");
}

}  // namespace mg
