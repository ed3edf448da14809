// Connected components of a symmetric graph by concurrent union-find, giving
// the labels of the reference's cc program (Algorithms/CC/cc.h:32-349: every
// vertex starts with its own id and atomicMin-propagates it along out-edges
// to a fixpoint, so on a symmetric graph each vertex ends with the smallest
// id of its component). Links always put the larger root under the smaller,
// so a root is the smallest id of its tree and the final find() of a vertex is
// exactly that label. Directed graphs keep the GAS program (mg_cc in
// gas_algos.cu), whose semantics there are not components.
//
// Order of work (the sampling scheme of Sutton et al., "Optimizing Parallel
// Graph Connectivity Computation via Subgraph Sampling", IPDPS 2018, with its
// first round done without atomics: hanging every vertex under a smaller
// neighbour, which only its own thread writes, is a valid forest):
//   1. every vertex starts under its first neighbour if that is smaller (but for
//      one in eight, kCcBreak), else as a root;
//   2. every vertex links with its second neighbour, a root of step 1 with its
//      first as well; the trees are flattened;
//   3. the most frequent root among kCcProbe fixed sample vertices names the
//      large component;
//   4. every vertex not already under that root links the rest of its edges.
// An edge skipped in step 4 joins two vertices of the large component, or is
// linked from its other end, which is not in it; on power-law graphs step 4
// touches a small share of the edges.
//
// On a skewed graph (kCcLongShare) the links of steps 1 and 2 queue up on a few roots
// (sampling alone took 340 us at R-MAT 21). There a one-launch BFS from the hub,
// of at most kCcLevels levels, finds the large component instead: what it
// reached starts under its smallest id, every other vertex links all its edges
// as in step 4. Any connected set serves, so the cap on the levels keeps long
// paths out of the BFS without changing a label. R-MAT 21: 0.68 -> 0.20 ms,
// R-MAT 22: 1.61 -> 0.31 ms. Where the first run of a graph finds that the BFS reaches
// fewer than kCcReach of the edges (several large components: 8 R-MAT graphs of scale 10
// to 16 in one took 1.06 ms by it, 0.31 without), the graph keeps to the sampling.
#include <cuda_runtime.h>

#include <climits>
#include <optional>
#include <vector>

#include "algo_util.cuh"
#include "gas/driver.cuh"
#include "gas/engine.cuh"
#include "grid_loop.cuh"

namespace mg {

// Root of x with path halving. Parent ids only decrease along a path and a
// root only ever becomes a non-root, so the walk ends and every shortcut
// written points to an ancestor.
MG_DEVINL int32_t cc_find(int32_t *parent, int32_t x) {
  for (;;) {
    const int32_t p = __ldcg(&parent[x]);
    if (p == x) return x;
    const int32_t gp = __ldcg(&parent[p]);
    if (gp == p) return p;
    parent[x] = gp;
    x = gp;
  }
}

// Links the components of a and b: the larger root is hooked under the smaller
// with atomicMin, which always succeeds. If the larger one was no longer a
// root (another link hooked it to `old` first), its tree and the smaller root
// still have to be joined: link old with the smaller root next. Every round
// hooks something, parent values only decrease, and the retries are bounded
// all the same (a failure is reported, not looped on).
MG_DEVINL bool cc_unite(int32_t *parent, int32_t a, int32_t b, unsigned long long limit) {
  for (unsigned long long it = 0; it < limit; ++it) {
    a = cc_find(parent, a);
    b = cc_find(parent, b);
    if (a == b) return true;
    const int32_t hi = a > b ? a : b, lo = a > b ? b : a;
    const int32_t old = atomicMin(&parent[hi], lo);
    if (old == hi) return true;
    a = old;
    b = lo;
  }
  return false;
}

// cc_unite for a whole warp (lanes with `pending` link a and b), one atomic per
// distinct larger root: the lane with the smallest other root hooks it, the
// lanes that hold the same larger root go on to join their other root with that
// one. Neighbouring vertices of a grid hang under the same few roots, and their
// hooks would queue up on one address (1200x1200 road grid with a third of its edges
// missing: 343 us for a run, 477 with a hook per lane). For the first neighbours
// alone: the lanes wait for one another, and second neighbours of a lattice form a
// chain through the warp (3000x3000 lattice: 1.24 ms, 1.57 with them by warps too).
MG_DEVINL bool cc_unite_warp(int32_t *parent, int32_t a, int32_t b, bool pending, unsigned long long limit) {
  const int lane = lane_id();
  for (unsigned long long it = 0; it < limit; ++it) {
    if (pending) {
      a = cc_find(parent, a);
      b = cc_find(parent, b);
      pending = a != b;
    }
    if (!__any_sync(0xffffffffu, pending)) return true;
    const int32_t hi = pending ? max(a, b) : -1 - lane, lo = min(a, b);
    const uint32_t same = __match_any_sync(0xffffffffu, hi);
    const int32_t least = __reduce_min_sync(same, lo);
    const uint32_t holders = __match_any_sync(0xffffffffu, ((unsigned long long)(uint32_t)hi << 32) | (uint32_t)lo);
    if (!pending) continue;
    if (lo != least) {
      a = lo;
      b = least;
    } else if (lane == __ffs(holders) - 1) {
      const int32_t old = atomicMin(&parent[hi], lo);
      pending = old != hi;
      a = old;
      b = lo;
    } else {
      pending = false;  // the same pair as the lane that hooks it
    }
  }
  return !__any_sync(0xffffffffu, pending);
}

constexpr int kCcSample = 2;    // neighbours linked per vertex before the large component is picked
constexpr int kCcProbe = 1024;  // sample vertices voting for the large component (one CTA)

// One vertex in 2^kCcBreak, spread by a multiplicative hash, stays a root in step 1 and
// links its first neighbour in step 2: on a lattice or a path every first neighbour is
// the one before, and the trees of step 1 were chains as long as it (road grids with 2 %
// of the edges dropped: 1000x1000 386 -> 293 us, 1200x1200 604 -> 480, 3000x3000 1.88 ->
// 1.11 ms, 1.13 with one vertex in four; a path of 4 M vertices 7.5 -> 0.63 ms). Two
// rounds of links with a flattening between them take 395 us, 464 us and 1.16 ms on those
// grids, 0.21 against 0.38 ms on a 1200x1200 lattice with no edge missing, and 450 against
// 335 us on a 1200x1200 grid with 35 % missing.
constexpr int kCcBreak = 3;
MG_DEVINL bool cc_breaks(int32_t v) { return ((uint32_t)v * 0x9E3779B1u) >> (32 - kCcBreak) == 0u; }

// Step 1: parent[v] = min(v, first neighbour).
__global__ void __launch_bounds__(kNT) k_cc_start(const int32_t *ro, const int32_t *col, int32_t *parent, int32_t V,
                                                  Ctl *ctl) {
  unsigned long long my_bytes = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const int b = ro[v], e = ro[v + 1];
    parent[v] = b < e && !cc_breaks(v) ? min(v, col[b]) : v;
    my_bytes += b < e ? 16 : 12;  // two offsets, the neighbour id, the parent
  }
  add_bytes(ctl, KID_CC, my_bytes);
}

// Step 2: vertex v links with its second neighbour, and with its first when
// step 1 left it a root.
__global__ void __launch_bounds__(kNT) k_cc_sample(const int32_t *ro, const int32_t *col, int32_t *parent, int32_t V,
                                                   Ctl *ctl) {
  const unsigned long long limit = ctl->spin_limit;
  bool ok = true;
  unsigned long long my_bytes = 0;
  for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31u); v0 < V;
       v0 += (int64_t)gridDim.x * blockDim.x) {
    const int v = (int)v0 + lane_id();
    const int b = v < V ? ro[v] : 0, e = v < V ? ro[v + 1] : 0;
    const int u0 = b < e ? col[b] : -1, u1 = b + 1 < e ? col[b + 1] : -1;
    const bool own0 = u0 > v || (u0 >= 0 && cc_breaks(v));  // step 1 left v a root
    my_bytes += 8 + (own0 ? 12 : b < e ? 4 : 0) + (u1 >= 0 ? 12 : 0);  // offsets; neighbour ids, parents read
    ok &= cc_unite_warp(parent, v, u0, own0, limit);
    if (u1 >= 0) ok &= cc_unite(parent, v, u1, limit);
  }
  if (!ok) raise_error(ctl, MG_ERR_TIMEOUT);
  add_bytes(ctl, KID_CC, my_bytes);
}

// Step 3: the root held by most of kCcProbe fixed sample vertices (ties: the
// smaller root). Written to *giant. Where parent[] is not quite flat (k_cc_flatten) it
// may be an inner vertex of the large tree; that serves as well, since all step 4 needs
// is that the vertices it skips hang under one and the same vertex.
__global__ void __launch_bounds__(kCcProbe) k_cc_giant(const int32_t *parent, int32_t V, int32_t *giant) {
  __shared__ int32_t s_lab[kCcProbe];
  __shared__ unsigned long long s_best[kCcProbe / 32];
  const int t = threadIdx.x;
  // fixed multiplicative-hash sample of the vertex ids
  const int v = (int)(((unsigned long long)(t + 1) * 2654435761ull) % (unsigned long long)V);
  s_lab[t] = parent[v];
  __syncthreads();
  const int mine = s_lab[t];
  int cnt = 0;
  for (int k = 0; k < kCcProbe; ++k) cnt += s_lab[k] == mine;
  // largest count, then smallest root: pack (count, ~root) and take the max
  unsigned long long key = ((unsigned long long)cnt << 32) | (uint32_t)(~(uint32_t)mine);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
    key = other > key ? other : key;
  }
  if (lane_id() == 0) s_best[warp_id()] = key;
  __syncthreads();
  if (t < 32) {
    key = s_best[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
      key = other > key ? other : key;
    }
    if (t == 0) *giant = (int32_t)(~(uint32_t)(key & 0xffffffffu));
  }
}

// Step 4: vertices outside the large component link their edges from the skip-th on. A
// warp takes 32 consecutive vertices; lists up to 32 edges are walked by their
// own lane, longer ones by the whole warp (32 edges per step).
__global__ void __launch_bounds__(kNT) k_cc_rest(const int32_t *ro, const int32_t *col, int32_t *parent, int32_t V,
                                                 const int32_t *giant, int skip, Ctl *ctl) {
  const unsigned long long limit = ctl->spin_limit;
  const int32_t big = *giant;
  const int lane = lane_id();
  bool ok = true;
  unsigned long long my_bytes = 0;
  const uint32_t groups = ((uint32_t)V + 31) / 32;
  for (uint32_t grp = (blockIdx.x * blockDim.x + threadIdx.x) / 32; grp < groups;
       grp += (gridDim.x * blockDim.x) / 32) {
    const int v = (int)(grp * 32) + lane;
    bool work = false;
    int b = 0, e = 0;
    if (v < V) {
      my_bytes += 12;  // parent, two offsets
      b = ro[v] + skip;
      e = ro[v + 1];
      work = b < e && __ldcg(&parent[v]) != big;
    }
    if (work && e - b <= 32) {
      for (int k = b; k < e; ++k) {
        my_bytes += 4;
        if (!cc_unite(parent, v, col[k], limit)) ok = false;
      }
    }
    uint32_t heavy = __ballot_sync(0xffffffffu, work && e - b > 32);
    while (heavy) {
      const int h = __ffs(heavy) - 1;
      heavy &= heavy - 1;
      const int hv = (int)(grp * 32) + h;
      const int hb = __shfl_sync(0xffffffffu, b, h), he = __shfl_sync(0xffffffffu, e, h);
      for (int k = hb + lane; k < he; k += 32) {
        my_bytes += 4;
        if (!cc_unite(parent, hv, col[k], limit)) ok = false;
      }
    }
  }
  if (!ok) raise_error(ctl, MG_ERR_TIMEOUT);
  add_bytes(ctl, KID_CC, my_bytes);
}

// Every vertex's root (in the end the smallest id of its component) to `out`.
// Between the steps that is `parent` itself: there a path halving that read an
// older ancestor may still replace a root just written, which only makes the
// tree less flat; the labels therefore go to an array of their own.
__global__ void __launch_bounds__(kNT) k_cc_flatten(int32_t *parent, int32_t *out, int32_t V, Ctl *ctl) {
  unsigned long long my_bytes = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    out[v] = cc_find(parent, v);
    my_bytes += 12;  // the vertex's parent, its root's parent, the write
  }
  add_bytes(ctl, KID_CC, my_bytes);
}

// The smallest vertex a BFS reached, then every vertex's start: under it, or a root.
__global__ void __launch_bounds__(kNT) k_cc_low(const int32_t *depth, int32_t V, int32_t *low) {
  int m = INT_MAX;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V && m == INT_MAX; v += gridDim.x * blockDim.x)
    if (depth[v] >= 0) m = v;  // a thread's vertices ascend
  m = __reduce_min_sync(0xffffffffu, m);
  if (lane_id() == 0 && m < *(volatile int32_t *)low) atomicMin(low, m);
}

__global__ void __launch_bounds__(kNT) k_cc_seed(const int32_t *depth, int32_t V, const int32_t *low, int32_t *parent,
                                                 Ctl *ctl) {
  const int32_t root = *low;
  unsigned long long my_bytes = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    parent[v] = depth[v] >= 0 ? root : v;
    my_bytes += 8;
  }
  add_bytes(ctl, KID_CC, my_bytes);
}

// Share of the edges in long lists (kLongList) from which the BFS finds the large
// component: R-MAT graphs have 0.15 (scale 10) to 0.65, and the hub is in their large
// component. A hub alone says nothing about the rest: from a vertex of 200 leaves beside
// a road grid with 2 % of the edges dropped 16 levels reach little, and the BFS and the
// other edges' hooks take 445 us (1200x1200) and 1.32 ms (3000x3000), the sampling 375 us
// and 1.14 ms. (Sparse R-MAT 21 graphs, one or two edges drawn a vertex, with / without
// the BFS: 175 / 306, 167 / 483 us.)
constexpr double kCcLongShare = 0.1;
constexpr uint32_t kCcLevels = 16;
// Share of the edges whose tails the BFS must reach: two R-MAT graphs of scales 10 and 11
// side by side (it reaches two thirds) 250 us, 137 by sampling. In one R-MAT graph it
// reaches all but a few edges.
constexpr double kCcReach = 0.8;

// Union-find CC on a symmetric graph (called by mg_cc).
int cc_union_find(mg_graph *g, int32_t *labels, mg_stats *stats, const mg_options *o) {
  cudaStream_t s = run_stream(g, o);
  int st = prepare_run(g, s);
  if (st != MG_OK) return st;
  const int32_t V = g->csr.V;
  if (V < 1) return set_error(MG_ERR_ARG, "cc: empty graph");
  int32_t *parent = g->ws.vbuf[0];
  Ctl *ctl = g->ws.ctl;
  bool by_bfs = g->hub >= 0 && o->use_cuda_graph && !prof_on() && o->spin_limit >= kSpinLimitDefault &&
                g->hub_degree <= kLoopPullList &&
                g->cc_by_bfs != 0 && (double)g->long_list_edges > kCcLongShare * (double)g->edges;
  std::optional<LoopRun> run;
  if (by_bfs) run.emplace(g, s);
  cudaError_t e = cudaEventRecord(g->ev0, s);
  if (e != cudaSuccess) return cuda_status(e, "event record");
  int32_t *giant = reinterpret_cast<int32_t *>(g->ws.scan);  // scratch word (the scan buffer is free here)
  const int vgrid = g->num_sms * 8;
  // the last pass writes the caller's buffer when it is this GPU's memory
  const bool direct = o->outputs_on_device != 0 && on_device(g, labels);
  int32_t *out = direct ? labels : g->ws.vbuf[1];
  k_ctl_init<<<1, 32, 0, s>>>(ctl, 1u, 1u, (unsigned long long)o->spin_limit, MODE_QUEUE, ctl_flags(nullptr));
  int32_t *depth = g->ws.gather_tmp;
  if (by_bfs) {
    mg_options bo;
    mg_options_init(&bo);
    st = bfs_loop_run(*run, g, s, {g->hub}, kCcLevels, &bo, depth, false);
    if (st != MG_OK && st != kLoopRefused) return st;
    by_bfs = st == MG_OK;
    if (by_bfs && g->cc_by_bfs < 0) {
      // the graph's first run: later ones queue the rest without waiting here
      if ((st = run->finish(cudaSuccess, "cc")) != MG_OK) return st;
      by_bfs = (double)g->loop_out->visited_edges >= kCcReach * (double)g->edges;
      g->cc_by_bfs = by_bfs ? 1 : 0;
    }
  }
  if (by_bfs) {
    k_fill_i32<<<1, 32, 0, s>>>(giant, INT_MAX, 1);
    k_cc_low<<<vgrid, kNT, 0, s>>>(depth, V, giant);
    k_cc_seed<<<vgrid, kNT, 0, s>>>(depth, V, giant, parent, ctl);
    k_cc_rest<<<vgrid, kNT, 0, s>>>(g->csr.row_offsets, g->csr.col, parent, V, giant, 0, ctl);
    count_launch(6);
  } else {
    MG_LAUNCH(KID_CC, s, (k_cc_start<<<vgrid, kNT, 0, s>>>(g->csr.row_offsets, g->csr.col, parent, V, ctl)));
    MG_LAUNCH(KID_CC, s, (k_cc_sample<<<vgrid, kNT, 0, s>>>(g->csr.row_offsets, g->csr.col, parent, V, ctl)));
    MG_LAUNCH(KID_CC, s, (k_cc_flatten<<<vgrid, kNT, 0, s>>>(parent, parent, V, ctl)));
    MG_LAUNCH(KID_CC, s, (k_cc_giant<<<1, kCcProbe, 0, s>>>(parent, V, giant)));
    MG_LAUNCH(KID_CC, s, (k_cc_rest<<<vgrid, kNT, 0, s>>>(g->csr.row_offsets, g->csr.col, parent, V, giant, kCcSample,
                                                          ctl)));
    count_launch(7);
  }
  MG_LAUNCH(KID_CC, s, (k_cc_flatten<<<vgrid, kNT, 0, s>>>(parent, out, V, ctl)));
  if ((st = launch_check("cc union-find")) != MG_OK) return st;
  e = cudaEventRecord(g->ev1, s);
  if (e != cudaSuccess) return cuda_status(e, "event record");
  Ctl c;
  if ((st = read_ctl(g, s, &c)) != MG_OK) return st;
  prof_flush(s, c.kbytes);
  if (by_bfs && (st = run->finish(cudaSuccess, "cc")) != MG_OK) return st;
  if (c.error) return set_error(c.error, std::string("cc: device reported ") + mg_status_string(c.error));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, g->ev0, g->ev1);
  finish_run(g, 1);
  if (stats) {
    stats->iterations = 1;
    stats->push_iterations = 1;
    stats->pull_iterations = 0;
    stats->converged = 1;
    stats->device_ms = ms;
    stats->residual = 0.0;
    stats->vertices_reached = g->nodes;
    stats->edges_traversed = g->edges;
  }
  return direct ? MG_OK : copy_out(s, labels, out, (size_t)V * 4, o->outputs_on_device != 0);
}

}  // namespace mg
