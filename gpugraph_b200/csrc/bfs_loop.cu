// Direction-optimising BFS in one cooperative launch (grid_loop.cuh): the start,
// every level and its direction decision, with one grid barrier per level (two
// where the frontier changes its form). The rules are those of the
// level-by-level loop (bfs.cu), so are the depths.
//
// The push frontier is a queue of edge ranges (first edge, length <= kRange):
// the thread that finds a vertex reads its row offsets anyway (the direction
// rule needs its degree) and appends its ranges, so a level needs no degree
// scan, and a hub's adjacency is spread over many warps. A warp takes up to 32
// ranges (fewer when the queue is short, so that all warps share it), its lanes
// the concatenated edges. The pull frontier is a bitmap; it is built from the
// depths when a push level hands over, and turned into ranges when a pull level
// does, so push levels keep no bitmap.
//
// Bound by the round trips of a level (ranges, columns, test-and-sets, the
// reservation, the barrier: 4 us a level on a path, 7 on a road grid) on small
// frontiers, by the bottom-up sweeps' loads on large ones. Against the
// level-by-level loop, per call: R-MAT 16 with host output 210 -> 91 us, R-MAT 21
// 230 -> 103 us, 1200x1200 road grid (67 levels) 1513 -> 460 us, 256 small graphs
// 295 -> 150 us.
#include <cuda_runtime.h>

#include <vector>

#include "gas/driver.cuh"
#include "grid_loop.cuh"
#include "host_util.h"

namespace mg {

constexpr int kLoopU = 4;     // edges per lane in flight
constexpr int kLoopWords = 4; // 32-vertex words per warp and step of a pull level
constexpr int kConvWords = 8; // and of a change of direction (256 small graphs: 160 us a run, 228 one word at a time)

struct BfsLoopArgs {
  DevCsr g;
  int32_t *labels;
  uint32_t *visited, *bm0, *bm1;
  int2 *q0, *q1;
  uint32_t cap;  // entries of a queue
  const int32_t *roots;  // device list of distinct roots, or null: the single root `root`
  int32_t root, nroots;
  uint32_t max_iter;
  int32_t dir;
  float alpha, beta;
  GridLoop loop;
};

// Appends the ranges of the N vertices of every lane (deg 0: none; first edge at
// beg) to queue q, one reservation per warp; called by the whole warp.
template <int N>
MG_DEVINL void append_ranges(int2 *q, uint32_t *tail, uint32_t cap, int32_t *error, const int (&beg)[N],
                             const int (&deg)[N]) {
  uint32_t k = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) k += (uint32_t)(deg[j] + kRange - 1) / kRange;
  if (!__any_sync(0xffffffffu, k != 0u)) return;
  const uint32_t inc = warp_inclusive_sum(k);
  uint32_t at = 0;
  if (lane_id() == 31) at = atomicAdd(tail, inc);
  at = __shfl_sync(0xffffffffu, at, 31) + inc - k;
  if (at + k > cap) {
    atomicCAS(error, 0, (int)MG_ERR_OVERFLOW);
    return;
  }
#pragma unroll
  for (int j = 0; j < N; ++j)
    for (int i = 0; i < deg[j]; i += kRange) q[at++] = make_int2(beg[j] + i, min(kRange, deg[j] - i));
}

// Top-down level: the ranges q[0, n) of level L's frontier. `probe`: look at a
// vertex's visited bit before setting it (a short level sets it at once, one
// round trip less).
MG_DEVINL void loop_push(const BfsLoopArgs &a, const int2 *q, uint32_t n, int2 *qn, uint32_t *tail, uint32_t L,
                         bool probe, LoopShared *sh) {
  const int lane = lane_id();
  const uint32_t nw = gridDim.x * (kLoopNT / 32), gw = warp_id() * gridDim.x + blockIdx.x;
  // ranges are dealt one by one over the warps (a hub's full ranges are
  // neighbours in the queue: in blocks of 32 they would land on a few warps)
  const uint32_t per = min(32u, (n + nw - 1) / nw);
  const int32_t *ro = a.g.row_offsets, *col = a.g.col;
  const uint32_t V = (uint32_t)a.g.V;
  uint32_t cnt = 0;
  unsigned long long edges = 0;
  for (uint32_t base = gw; base < n; base += nw * per) {
    int2 r = make_int2(0, 0);
    if (lane < (int)per && base + lane * nw < n) r = __ldcg(&q[base + lane * nw]);
    const int inc = warp_inclusive_sum(r.y);
    const int total = __shfl_sync(0xffffffffu, inc, 31);
    const int off = r.x - (inc - r.y);  // edge id of concatenated position p in this lane's range: off + p
    for (int t = 0; t < total; t += 32 * kLoopU) {
      int u[kLoopU];
#pragma unroll
      for (int k = 0; k < kLoopU; ++k) {
        const int p = t + 32 * k + lane;
        int own = 0;  // the first range that ends past p
        if (per > 1) {
#pragma unroll
          for (int s = 16; s > 0; s >>= 1)
            if (__shfl_sync(0xffffffffu, inc, own + s - 1) <= p) own += s;
          own = min(own, 31);
        }
        const int e = __shfl_sync(0xffffffffu, off, own) + p;
        u[k] = p < total && (unsigned)e < (unsigned)a.g.E ? __ldcs(col + e) : -1;
      }
      // heads not seen yet; their row offsets travel with the test-and-sets (a
      // level's time is its chain of round trips, so one less counts)
      uint32_t seen[kLoopU];
#pragma unroll
      for (int k = 0; k < kLoopU; ++k)
        seen[k] = (unsigned)u[k] >= V ? ~0u : probe ? __ldcg(&a.visited[u[k] >> 5]) : 0u;
      int b[kLoopU], d[kLoopU];
#pragma unroll
      for (int k = 0; k < kLoopU; ++k) {
        const uint32_t bit = 1u << (u[k] & 31);
        b[k] = d[k] = 0;
        if (!(seen[k] & bit)) {
          b[k] = ro[u[k]];
          d[k] = ro[u[k] + 1];
          seen[k] = atomicOr(&a.visited[u[k] >> 5], bit);
        }
      }
#pragma unroll
      for (int k = 0; k < kLoopU; ++k) {
        const bool won = !((seen[k] >> (u[k] & 31)) & 1u);
        d[k] = won ? d[k] - b[k] : 0;
        if (won) {
          a.labels[u[k]] = (int)L + 1;
          ++cnt;
          edges += (unsigned long long)d[k];
        }
      }
      append_ranges(qn, tail, a.cap, &a.loop.c->error, b, d);
    }
  }
  cnt = warp_sum(cnt);
  edges = warp_sum(edges);
  if (lane == 0 && cnt) atomicAdd(&sh->my_count, (unsigned long long)cnt);
  if (lane == 0 && edges) atomicAdd(&sh->my_edges, edges);
}

// Bottom-up level: every unvisited vertex looks for an in-neighbour in the
// frontier bitmap `cur` (hub-first lists, four in-edges per step, stop at the
// first parent); `nxt` is written for every word.
MG_DEVINL void loop_pull(const BfsLoopArgs &a, const uint32_t *cur, uint32_t *nxt, uint32_t L, LoopShared *sh) {
  const int lane = lane_id();
  const int32_t V = a.g.V;
  const int32_t *coff = a.g.csc_offsets, *crow = a.g.pull_rows, *ro = a.g.row_offsets;
  const uint32_t words = ((uint32_t)V + 31) / 32, steps = (words + kLoopWords - 1) / kLoopWords;
  const uint32_t nw = gridDim.x * (kLoopNT / 32), gw = warp_id() * gridDim.x + blockIdx.x;
  uint32_t cnt = 0;
  unsigned long long edges = 0;
  for (uint32_t t = gw; t < steps; t += nw) {
    uint32_t vis[kLoopWords];
    int beg[kLoopWords], end[kLoopWords];
#pragma unroll
    for (int q = 0; q < kLoopWords; ++q) {
      const uint32_t w = t * kLoopWords + q;
      const int v = (int)(w * 32 + lane);
      vis[q] = w < words ? __ldcg(&a.visited[w]) : ~0u;
      beg[q] = v < V ? coff[v] : 0;
      end[q] = v < V ? coff[v + 1] : 0;
    }
    int u[kLoopWords][4];
#pragma unroll
    for (int q = 0; q < kLoopWords; ++q) {
      const int v = (int)((t * kLoopWords + q) * 32 + lane);
      if (v >= V || ((vis[q] >> lane) & 1u)) end[q] = beg[q];  // nothing to scan
#pragma unroll
      for (int k = 0; k < 4; ++k) u[q][k] = beg[q] + k < end[q] ? __ldcs(crow + beg[q] + k) : -1;
    }
    bool found[kLoopWords];
#pragma unroll
    for (int q = 0; q < kLoopWords; ++q) {
      uint32_t hit = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (u[q][k] >= 0) hit |= cur[u[q][k] >> 5] >> (u[q][k] & 31);
      found[q] = hit & 1u;
    }
#pragma unroll
    for (int q = 0; q < kLoopWords; ++q) {
      const uint32_t w = t * kLoopWords + q;
      const int v = (int)(w * 32 + lane);
      if (!found[q]) {
        for (int e = beg[q] + 4; e < end[q]; e += 4) {
          const int c = min(4, end[q] - e);
          const int u0 = __ldcs(crow + e);
          const int u1 = c > 1 ? __ldcs(crow + e + 1) : u0;
          const int u2 = c > 2 ? __ldcs(crow + e + 2) : u0;
          const int u3 = c > 3 ? __ldcs(crow + e + 3) : u0;
          if (((cur[u0 >> 5] >> (u0 & 31)) | (cur[u1 >> 5] >> (u1 & 31)) | (cur[u2 >> 5] >> (u2 & 31)) |
               (cur[u3 >> 5] >> (u3 & 31))) &
              1u) {
            found[q] = true;
            break;
          }
        }
      }
      const uint32_t bal = __ballot_sync(0xffffffffu, found[q]);
      if (lane == 0 && w < words) {
        nxt[w] = bal;
        if (bal) a.visited[w] = vis[q] | bal;
      }
      if (found[q]) {
        a.labels[v] = (int)L + 1;
        edges += (unsigned long long)(ro[v + 1] - ro[v]);
      }
      cnt += found[q];
    }
  }
  cnt = warp_sum(cnt);
  edges = warp_sum(edges);
  if (lane == 0 && cnt) atomicAdd(&sh->my_count, (unsigned long long)cnt);
  if (lane == 0 && edges) atomicAdd(&sh->my_edges, edges);
}

__global__ void __launch_bounds__(kLoopNT, 1) k_bfs_loop(BfsLoopArgs a) {
  __shared__ LoopShared sh;
  const int lane = lane_id();
  const int32_t V = a.g.V;
  const int32_t *ro = a.g.row_offsets;
  const uint32_t words = ((uint32_t)V + 31) / 32;
  const uint32_t tid = blockIdx.x * kLoopNT + threadIdx.x, nt = gridDim.x * kLoopNT;
  const uint32_t nw = nt / 32, gw = warp_id() * gridDim.x + blockIdx.x;
  LoopCtl *c = a.loop.c;
  if (threadIdx.x == 0) {
    sh.my_count = sh.my_edges = sh.my_mask = 0;
    sh.fail = 0;
  }
  __syncthreads();
  // start: every depth and bitmap word; several roots are set after a barrier
  const bool one = a.roots == nullptr;
  for (uint32_t i = tid; i < (uint32_t)V; i += nt) a.labels[i] = one && (int32_t)i == a.root ? 0 : -1;
  for (uint32_t i = tid; i < words; i += nt) {
    const uint32_t x = one && i == (uint32_t)a.root >> 5 ? 1u << (a.root & 31) : 0u;
    a.visited[i] = x;
    a.bm0[i] = x;
  }
  if (blockIdx.x == 0 && threadIdx.x < 3) {
    c->count[threadIdx.x] = c->edges[threadIdx.x] = 0;
    c->items[threadIdx.x] = 0;
    if (threadIdx.x == 0) c->error = 0;
  }
  uint32_t nbar = 0, items = 0;
  unsigned long long vcount = (unsigned long long)a.nroots, vedges = 0, m = 0;
  if (one) {
    // the root's ranges: CTA 0 writes them, every thread knows their number
    const int b = ro[a.root], d = ro[a.root + 1] - b;
    items = (uint32_t)(d + kRange - 1) / kRange;
    m = (unsigned long long)d;
    if (blockIdx.x == 0)
      for (uint32_t i = threadIdx.x; i < items; i += kLoopNT)
        a.q0[i] = make_int2(b + (int)i * kRange, min(kRange, d - (int)i * kRange));
  }
  bool ok = grid_level_end(a.loop, &sh, 2, nbar);
  if (ok && !one) {
    unsigned long long e = 0;
    for (uint32_t base = gw * 32; base < (uint32_t)a.nroots; base += nw * 32) {
      int b[1] = {0}, d[1] = {0};
      if (base + lane < (uint32_t)a.nroots) {
        const int v = a.roots[base + lane];
        b[0] = ro[v];
        d[0] = ro[v + 1] - b[0];
        a.labels[v] = 0;
        atomicOr(&a.visited[v >> 5], 1u << (v & 31));
        atomicOr(&a.bm0[v >> 5], 1u << (v & 31));
      }
      e += (unsigned long long)d[0];
      append_ranges(a.q0, &c->items[2], a.cap, &c->error, b, d);
    }
    e = warp_sum(e);
    if (lane == 0 && e) atomicAdd(&sh.my_edges, e);
    ok = grid_level_end(a.loop, &sh, 2, nbar);
    m = sh.edges;
    items = sh.items;
  }
  vedges = m;
  // state of the level about to run, the same in every thread
  uint32_t L = 0, push = 0, pull = 0;
  unsigned long long n = (unsigned long long)a.nroots;
  bool bitmap = a.dir == MG_DIR_PULL;  // the level's form; level 0 has both
  bool ready = true;                   // the frontier exists in that form
  while (ok && n > 0 && L < a.max_iter) {
    const uint32_t slot = L % 3;
    // slot of the next level: last read after the barrier of level L-2
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      c->count[(L + 1) % 3] = c->edges[(L + 1) % 3] = 0;
      c->items[(L + 1) % 3] = 0;
    }
    uint32_t *cur = (L & 1) ? a.bm1 : a.bm0, *nxt = (L & 1) ? a.bm0 : a.bm1;
    int2 *q = (L & 1) ? a.q1 : a.q0, *qn = (L & 1) ? a.q0 : a.q1;
    if (bitmap) {
      if (!ready) {  // push -> pull: the bitmap of the vertices at depth L
        for (uint32_t w0 = gw * kConvWords; w0 < words; w0 += nw * kConvWords) {
          int l[kConvWords];
#pragma unroll
          for (int k = 0; k < kConvWords; ++k) {
            const uint32_t v = (w0 + k) * 32 + lane;
            l[k] = v < (uint32_t)V ? a.labels[v] : -1;
          }
#pragma unroll
          for (int k = 0; k < kConvWords; ++k) {
            const uint32_t bal = __ballot_sync(0xffffffffu, l[k] == (int)L);
            if (lane == 0 && w0 + k < words) cur[w0 + k] = bal;
          }
        }
        if (!(ok = grid_level_end(a.loop, &sh, slot, nbar))) break;
      }
      loop_pull(a, cur, nxt, L, &sh);
      ++pull;
    } else {
      if (!ready) {  // pull -> push: the ranges of the bitmap's vertices
        // kConvWords words per warp step: their row offsets in flight, one reservation
        for (uint32_t w0 = gw * kConvWords; w0 < words; w0 += nw * kConvWords) {
          const uint32_t mine = lane < kConvWords && w0 + lane < words ? cur[w0 + lane] : 0u;
          if (!__any_sync(0xffffffffu, mine != 0u)) continue;
          int b[kConvWords], d[kConvWords];
#pragma unroll
          for (int k = 0; k < kConvWords; ++k) {
            const uint32_t x = __shfl_sync(0xffffffffu, mine, k), v = (w0 + k) * 32 + lane;
            const bool in = (x >> lane) & 1u;
            b[k] = in ? ro[v] : 0;
            d[k] = in ? ro[v + 1] : 0;
          }
#pragma unroll
          for (int k = 0; k < kConvWords; ++k) d[k] -= b[k];
          append_ranges(q, &c->items[(L + 2) % 3], a.cap, &c->error, b, d);
        }
        if (!(ok = grid_level_end(a.loop, &sh, (L + 2) % 3, nbar))) break;
        items = sh.items;
      }
      loop_push(a, q, items, qn, &c->items[slot], L, m > (1ull << 18), &sh);
      ++push;
    }
    if (!(ok = grid_level_end(a.loop, &sh, slot, nbar))) break;
    const unsigned long long n_next = sh.count, m_next = sh.edges;
    vcount += n_next;
    vedges += m_next;
    bool next_bitmap = bitmap;
    if (a.dir == MG_DIR_PUSH) {
      next_bitmap = false;
    } else if (a.dir == MG_DIR_PULL) {
      next_bitmap = true;
    } else if (!bitmap) {
      // only while the frontier grows: near the end of a search the unvisited
      // edges are few, and a sweep over every vertex costs more than the push
      const double unvisited = (double)a.g.E - (double)vedges;
      if ((double)m_next > unvisited / (double)a.alpha && n_next > n) next_bitmap = true;
    } else if ((double)n_next < (double)V / (double)a.beta && n_next < n) {
      next_bitmap = false;
    }
    ready = next_bitmap == bitmap;
    items = sh.items;
    bitmap = next_bitmap;
    n = n_next;
    m = m_next;
    ++L;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    LoopOut *o = a.loop.out;
    o->level = L;
    o->push_levels = push;
    o->pull_levels = pull;
    o->frontier_size = (uint32_t)n;
    o->visited_count = vcount;
    o->visited_edges = vedges;
    o->barriers = nbar;
    o->error = ok ? *(volatile int32_t *)&c->error : (int32_t)MG_ERR_TIMEOUT;
  }
}

int bfs_loop_run(LoopRun &run, mg_graph *g, cudaStream_t s, const std::vector<int32_t> &roots, uint32_t max_iter,
                 const mg_options *o, int32_t *labels, bool timed) {
  BfsLoopArgs a;
  a.g = g->csr;
  a.labels = labels;
  a.visited = g->ws.visited;
  a.bm0 = g->ws.bm[0];
  a.bm1 = g->ws.bm[1];
  a.q0 = g->loop_queue;
  a.q1 = g->loop_queue + g->loop_cap;
  a.cap = (uint32_t)g->loop_cap;
  a.roots = nullptr;
  a.root = roots[0];
  a.nroots = (int32_t)roots.size();
  if (roots.size() > 1) {
    cudaError_t e = cudaMemcpyAsync(g->ws.queue[0], roots.data(), roots.size() * 4, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cuda_status(e, "bfs roots");
    a.roots = g->ws.queue[0];
  }
  a.max_iter = max_iter;
  a.dir = o->direction;
  a.alpha = (float)o->alpha;
  a.beta = (float)o->beta;
  a.loop = run.args(o);
  void *args[] = {&a};
  return run.launch((const void *)k_bfs_loop, args, timed, "bfs loop launch");
}

}  // namespace mg
