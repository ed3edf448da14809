// Personalised PageRank with its adjoint (no reference counterpart): the
// forward solve and the gradients of a loss with respect to the teleport
// vectors and the edge weights.
//
// Forward:  R = (1-d) T + d P^T R,  R, T in [V][nvec] (row-major), P[u,v] = w(e(u,v))
//           solved by power iteration pulled over the in-edges (CSC):
//           R'[v,:] = (1-d) T[v,:] + d * sum_{u->v} w(u,v) R[u,:]
// Adjoint:  for L with G = dL/dR, lambda = G + d P lambda, pulled over the
//           out-edges (CSR): lambda'[u,:] = G[u,:] + d * sum_{u->v} w(u,v) lambda[v,:]
//           dL/dT = (1-d) lambda,  dL/dw(u,v) = d * <lambda[v,:], R[u,:]>
// Both solves stop when the L1 change over all entries is <= tolerance times
// the L1 norm of their right-hand side (T or G; for teleport columns that are
// distributions that is tolerance * nvec), or after iter_num iterations.
//
// Layout and work split: the solve's rows are padded to nv = nvec rounded up to
// a multiple of 4, so every row is 16-byte aligned and falls into G pieces of 4
// columns (nv/4 rounded up to a power of two). A group of 8 lanes (16 for more
// than 32 columns) owns one chunk of one vertex's adjacency (PprGroup): an edge
// costs one coalesced row read, and a warp works on 4 (2) chunks at once. The chunks are taken in descending
// order of length (vertex order within a length), so the groups of a warp run
// the same number of steps. Adjacencies longer than kPprChunk are cut into
// chunks whose partial rows are added in chunk order by a fix-up pass
// (deterministic). The forward solve reads the weights gathered into CSC order
// once per solve.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <optional>
#include <vector>

#include "algo_util.cuh"
#include "gas/driver.cuh"
#include "gas/engine.cuh"
#include "grid_loop.cuh"

namespace mg {

// Longest chunk. On a graph of up to kPprSmall edges the chunks are as long as the
// square root of the longest list, to a power of two from 64 on: a chunk is summed
// step by step, a cut list's partial rows one after the other, and the longer of
// the two chains is the iteration there (R-MAT 12, 32 columns, forward and
// backward: 3.25 ms with chunks of 256, 1.84 with 64; R-MAT 18, 12 columns: 6.5 /
// 7.1 ms with 128).
constexpr int64_t kPprSmall = 1 << 21;
constexpr int kPprChunk = 256;
constexpr int kPprMaxVec = 64;

struct PprArgs {
  const int32_t *idx;              // adjacency of the solve (CSC forward, CSR adjoint)
  const float *w;                  // weights in the order of idx
  const float *rhs;                // T (forward) or G (adjoint), [V][nv]
  float alpha, d;                  // X' = alpha*rhs + d*sum(...)
  float *x0, *x1, *partial;
  const int32_t *cv, *cb, *ce, *cslot, *mv, *mfirst;
  // nfull: chunks that have edges (they come first); columns [nvec, nv) are padding and
  // stay 0 (their sums may not: 0 times an infinite weight), so they add nothing to a residual
  int32_t nchunks, nfull, nmulti, nvec, nv, V;
  Ctl *ctl;
};

template <int NC>
MG_DEVINL void ppr_finalize_row(const PprArgs &a, int v, const float (&acc)[NC], const float *xold, float *xnew,
                                double &res) {
  const int lane = lane_id();
#pragma unroll
  for (int q = 0; q < NC; ++q) {
    const int c = lane + 32 * q;
    if (c < a.nv) {
      const int64_t o = (int64_t)v * a.nv + c;
      const float xn = c < a.nvec ? fmaf(a.d, acc[q], a.alpha * a.rhs[o]) : 0.f;
      res += (double)fabsf(xn - xold[o]);
      xnew[o] = xn;
    }
  }
}

// A group of kPprStep lanes (16 when a row has more than 8 pieces) takes a chunk
// in steps of kPprStep edges. Its lanes are G column pieces x ES edge slots: the
// lane of slot e takes the step's edges e, e + ES, ..., and the slots' sums are
// added at the end of the chunk (one slot from 17 columns on).
constexpr int kPprStep = 8;
template <int G>
struct PprGroup {
  static constexpr int kLanes = G < kPprStep ? kPprStep : G;
  static constexpr int kPer = 32 / kLanes;      // chunks per warp
  static constexpr int kSlots = kLanes / G;     // edge slots
  static constexpr int kEdges = kPprStep / kSlots;  // edges of a step per lane
  int gl, piece, slot;
  MG_DEVINL PprGroup() : gl(lane_id() & (kLanes - 1)), piece(gl % G), slot(gl / G) {}
  // the step's edges [k, k + kPprStep): lane l holds edge k + l (-1 past the end)
  MG_DEVINL void load(const int32_t *idx, const float *wgt, int k, int e, int &u, float &w) const {
    const int p = k + (gl & (kPprStep - 1));
    u = p < e ? __ldcs(idx + p) : -1;
    w = p < e && wgt ? __ldcs(wgt + p) : 0.f;
  }
  template <typename T>
  MG_DEVINL T of(T x, int j) const {  // the value of this lane's j-th edge of the step
    return __shfl_sync(0xffffffffu, x, j * kSlots + slot, kLanes);
  }
  MG_DEVINL float sum_slots(float x) const {
#pragma unroll
    for (int o = G; o < kLanes; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  }
};

// One iteration's sweep over the chunks. A step's row loads are in flight
// together, its indices and weights were loaded one step ahead (one coalesced
// load per group each, passed on by shuffles). Vertices without edges keep
// alpha*rhs: both iterates hold it after the first two iterations, and from
// then on their chunks are not visited.
template <int G, bool RO>
MG_DEVINL void ppr_sweep(const PprArgs &a, uint32_t L, uint32_t gw, uint32_t nw, double &res,
                         unsigned long long &my_bytes) {
  using P = PprGroup<G>;
  const P g;
  const float *xold = (L & 1) ? a.x1 : a.x0;
  float *xnew = (L & 1) ? a.x0 : a.x1;
  const int col = g.piece * 4;
  const bool cok = col < a.nv;
  const uint32_t n = (uint32_t)(L < 2 ? a.nchunks : a.nfull);
  for (uint32_t c0 = gw * P::kPer; c0 < n; c0 += nw * P::kPer) {
    const uint32_t c = c0 + lane_id() / P::kLanes;
    const bool has = c < n;
    const int v = has ? a.cv[c] : 0, b = has ? a.cb[c] : 0, e = has ? a.ce[c] : 0;
    const int slot = has ? a.cslot[c] : 0;
    const int steps = (__reduce_max_sync(0xffffffffu, e - b) + kPprStep - 1) / kPprStep;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    int u, un;
    float w, wn;
    g.load(a.idx, a.w, b, e, u, w);
    for (int s = 0; s < steps; ++s) {
      g.load(a.idx, a.w, b + (s + 1) * kPprStep, e, un, wn);
      float4 row[P::kEdges];
#pragma unroll
      for (int j = 0; j < P::kEdges; ++j) {
        const int t = g.of(u, j);
        row[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t >= 0 && cok) {
          const float4 *r = reinterpret_cast<const float4 *>(xold + (int64_t)t * a.nv + col);
          row[j] = RO ? __ldg(r) : *r;
        }
      }
#pragma unroll
      for (int j = 0; j < P::kEdges; ++j) {
        const float wt = g.of(w, j);
        acc.x = fmaf(wt, row[j].x, acc.x);
        acc.y = fmaf(wt, row[j].y, acc.y);
        acc.z = fmaf(wt, row[j].z, acc.z);
        acc.w = fmaf(wt, row[j].w, acc.w);
      }
      u = un;
      w = wn;
    }
    acc = make_float4(g.sum_slots(acc.x), g.sum_slots(acc.y), g.sum_slots(acc.z), g.sum_slots(acc.w));
    if (!has) continue;
    if (g.gl == 0) my_bytes += (unsigned long long)(e - b) * (8ull + 4ull * a.nv);
    if (g.slot != 0 || !cok) continue;
    if (slot < 0) {
      const int64_t o = (int64_t)v * a.nv + col;
      const float4 r = *reinterpret_cast<const float4 *>(a.rhs + o);
      const float4 xo = *reinterpret_cast<const float4 *>(xold + o);
      float4 xn;
      xn.x = fmaf(a.d, acc.x, a.alpha * r.x);
      xn.y = fmaf(a.d, acc.y, a.alpha * r.y);
      xn.z = fmaf(a.d, acc.z, a.alpha * r.z);
      xn.w = fmaf(a.d, acc.w, a.alpha * r.w);
      if (col + 1 >= a.nvec) xn.y = 0.f;
      if (col + 2 >= a.nvec) xn.z = 0.f;
      if (col + 3 >= a.nvec) xn.w = 0.f;
      res += (double)fabsf(xn.x - xo.x) + (double)fabsf(xn.y - xo.y) + (double)fabsf(xn.z - xo.z) +
             (double)fabsf(xn.w - xo.w);
      *reinterpret_cast<float4 *>(xnew + o) = xn;
      if (g.piece == 0) my_bytes += 12ull * a.nv;
    } else {
      *reinterpret_cast<float4 *>(a.partial + (int64_t)slot * a.nv + col) = acc;
    }
  }
}

template <int G>
__global__ void __launch_bounds__(kNT, 4) k_ppr_iter(PprArgs a) {
  Ctl *ctl = a.ctl;
  if (!ctl->active) return;
  double res = 0.0;
  unsigned long long my_bytes = 0;
  ppr_sweep<G, true>(a, ctl->level, blockIdx.x * kNW + warp_id(), gridDim.x * kNW, res, my_bytes);
  add_bytes(ctl, KID_PPR, my_bytes);
  res = cta_sum_f64(res);
  if (threadIdx.x == 0 && res != 0.0) atomicAdd(&ctl->acc[1], res);
}

// Split vertices: partial rows added in chunk order.
template <int NC>
MG_DEVINL void ppr_fix(const PprArgs &a, uint32_t L, uint32_t gw, uint32_t nw, double &res) {
  const float *xold = (L & 1) ? a.x1 : a.x0;
  float *xnew = (L & 1) ? a.x0 : a.x1;
  const int lane = lane_id();
  for (uint32_t m = gw; m < (uint32_t)a.nmulti; m += nw) {
    const int v = a.mv[m];
    float acc[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q) acc[q] = 0.f;
    // eight partial rows loaded at once, then added in chunk order (a hub has
    // hundreds of chunks; one dependent load per chunk made this the tail)
    int s = a.mfirst[m];
    const int se = a.mfirst[m + 1];
    for (; s + 8 <= se; s += 8) {
      float t[8][NC];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int q = 0; q < NC; ++q) {
          const int col = lane + 32 * q;
          t[j][q] = col < a.nv ? a.partial[(int64_t)(s + j) * a.nv + col] : 0.f;
        }
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int q = 0; q < NC; ++q) acc[q] += t[j][q];
    }
    for (; s < se; ++s)
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        const int col = lane + 32 * q;
        if (col < a.nv) acc[q] += a.partial[(int64_t)s * a.nv + col];
      }
    ppr_finalize_row<NC>(a, v, acc, xold, xnew, res);
  }
}

template <int NC>
__global__ void __launch_bounds__(kNT) k_ppr_fixup(PprArgs a) {
  Ctl *ctl = a.ctl;
  if (!ctl->active) return;
  double res = 0.0;
  ppr_fix<NC>(a, ctl->level, blockIdx.x * kNW + warp_id(), gridDim.x * kNW, res);
  res = cta_sum_f64(res);
  if (threadIdx.x == 0 && res != 0.0) atomicAdd(&ctl->acc[1], res);
}

// A whole solve in one cooperative launch (grid_loop.cuh): one barrier per
// iteration, two where adjacencies are cut, one more for the norm of the
// right-hand side. For solves whose iteration is short beside the launches of
// the level loop.
template <int G>
__global__ void __launch_bounds__(kLoopNT, 1) k_ppr_loop(PprArgs a, double tol, uint32_t max_iter, GridLoop loop) {
  __shared__ LoopShared sh;
  const uint32_t tid = blockIdx.x * kLoopNT + threadIdx.x, nt = gridDim.x * kLoopNT;
  const uint32_t nw = nt / 32, gw = warp_id() * gridDim.x + blockIdx.x;
  LoopCtl *c = loop.c;
  if (threadIdx.x == 0) {
    sh.my_count = sh.my_edges = sh.my_mask = 0;
    sh.fail = 0;
  }
  // slot 1 takes the norm, slot 0 the first iteration
  if (blockIdx.x == 0 && threadIdx.x < 3) {
    c->residual[threadIdx.x] = 0.0;
    if (threadIdx.x == 0) c->error = 0;
  }
  uint32_t nbar = 0, L = 0;
  __syncthreads();
  bool ok = grid_level_end(loop, &sh, 2, nbar);
  double sum = 0.0;
  for (int64_t i = tid; i < (int64_t)a.V * a.nv; i += nt) sum += fabs((double)a.rhs[i]);
  sum = cta_sum_f64(sum);
  if (threadIdx.x == 0 && sum != 0.0) atomicAdd(&c->residual[1], sum);
  ok = ok && grid_level_end(loop, &sh, 1, nbar);
  const double norm = sh.residual;
  // (the slots below start at 2: iteration L uses slot (L + 2) % 3, cleared two barriers earlier)
  double last = 0.0;
  bool more = max_iter > 0;
  unsigned long long my_bytes = 0;
  while (ok && more) {
    const uint32_t slot = (L + 2) % 3;
    // slot of the next iteration: last read before the previous one
    if (blockIdx.x == 0 && threadIdx.x == 0) c->residual[(L + 3) % 3] = 0.0;
    double res = 0.0;
    ppr_sweep<G, false>(a, L, gw, nw, res, my_bytes);
    if (a.nmulti) {
      if (!(ok = grid_level_end(loop, &sh, slot, nbar))) break;
      ppr_fix<(G > 8 ? 2 : 1)>(a, L, gw, nw, res);
    }
    res = cta_sum_f64(res);
    if (threadIdx.x == 0 && res != 0.0) atomicAdd(&c->residual[slot], res);
    if (!(ok = grid_level_end(loop, &sh, slot, nbar))) break;
    last = sh.residual;
    ++L;
    more = last > tol * norm && L < max_iter;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    LoopOut *o = loop.out;
    o->level = L;
    o->residual = last;
    o->norm = norm;
    o->barriers = nbar;
    o->error = ok ? *(volatile int32_t *)&c->error : (int32_t)MG_ERR_TIMEOUT;
  }
}

// ctl->acc[2] holds the L1 norm of the right-hand side (k_ppr_rhs_norm).
__global__ void k_ppr_level_end(Ctl *ctl, double tol, cudaGraphConditionalHandle h, int use_handle) {
  if (threadIdx.x != 0) return;
  if (ctl->active) {
    const double res = ctl->acc[1];
    ctl->acc[1] = 0.0;
    ctl->residual = res;
    ctl->level += 1;
    ctl->push_levels += 1;
    ctl->active = (res > tol * ctl->acc[2] && ctl->level < ctl->max_iter && ctl->error == 0) ? 1u : 0u;
  }
  if (use_handle) cudaGraphSetConditional(h, ctl->active);
}

// dL/dw(u,v) = d <lambda[v,:], R[u,:]>: a group of lanes per out-edge chunk of
// the CSR chunk plan (a row, or at most kPprChunk edges of a long row), laid out
// as in ppr_sweep: R[u,:] held in registers, a step's lambda rows in flight, the
// dot products reduced over a slot's pieces. R has the caller's row stride nvec.
template <int G>
__global__ void __launch_bounds__(kNT, 4) k_ppr_edge_grad(const int32_t *cv, const int32_t *cb, const int32_t *ce,
                                                          int32_t n, const int32_t *idx, int32_t nvec, int32_t nv,
                                                          const float *lam, const float *R, float d, float *grad_w,
                                                          Ctl *ctl) {
  using P = PprGroup<G>;
  const P g;
  const int col = g.piece * 4;
  const uint32_t nw = gridDim.x * kNW;
  unsigned long long my_bytes = 0;
  for (uint32_t c0 = (blockIdx.x * kNW + warp_id()) * P::kPer; c0 < (uint32_t)n; c0 += nw * P::kPer) {
    const uint32_t c = c0 + lane_id() / P::kLanes;
    const bool has = c < (uint32_t)n;
    const int u = has ? cv[c] : 0, b = has ? cb[c] : 0, e = has ? ce[c] : 0;
    float ru[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) ru[q] = has && col + q < nvec ? R[(int64_t)u * nvec + col + q] : 0.f;
    const int steps = (__reduce_max_sync(0xffffffffu, e - b) + kPprStep - 1) / kPprStep;
    int v, vn;
    float none;
    g.load(idx, nullptr, b, e, v, none);
    for (int s = 0; s < steps; ++s) {
      const int k = b + s * kPprStep;
      g.load(idx, nullptr, k + kPprStep, e, vn, none);
      float4 row[P::kEdges];
#pragma unroll
      for (int j = 0; j < P::kEdges; ++j) {
        const int t = g.of(v, j);
        row[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t >= 0 && col < nv) row[j] = __ldg(reinterpret_cast<const float4 *>(lam + (int64_t)t * nv + col));
      }
#pragma unroll
      for (int j = 0; j < P::kEdges; ++j) {
        float dot = fmaf(row[j].w, ru[3], fmaf(row[j].z, ru[2], fmaf(row[j].y, ru[1], row[j].x * ru[0])));
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        // the slot's lane j (of its pieces, in turn) writes the edge
        const int i = k + j * P::kSlots + g.slot;
        if (g.piece == j % G && i < e) grad_w[i] = d * dot;
      }
      v = vn;
    }
    if (has && g.gl == 0) my_bytes += 4ull * nvec + (unsigned long long)(e - b) * (8ull + 4ull * nv);
  }
  add_bytes(ctl, KID_PPR, my_bytes);
}

// L1 norm of the right-hand side into ctl->acc[2] (FP64 accumulation).
__global__ void k_ppr_rhs_norm(const float *rhs, int64_t n, Ctl *ctl) {
  double sum = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    sum += fabs((double)rhs[i]);
  sum = cta_sum_f64(sum);
  if (threadIdx.x == 0 && sum != 0.0) atomicAdd(&ctl->acc[2], sum);
}

// dst[i][0..nd) = s * src[i][0..ns) for V rows, columns past ns zero: to and
// from the padded rows of a solve.
__global__ void k_rows_f32(const float *src, int32_t ns, float *dst, int32_t nd, float s, int64_t V) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V * nd; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = ns == nd ? 0 : i / nd;
    const int32_t c = ns == nd ? 0 : (int32_t)(i - r * nd);
    dst[i] = ns == nd ? s * src[i] : c < ns ? s * src[r * ns + c] : 0.f;
  }
}

__global__ void k_copy_f32(const float *src, float *dst, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

__global__ void k_gather_f32(const int32_t *idx, const float *src, float *dst, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = src[idx[i]];
}

// Chunk plan for the solve over `off` (host copy of the offsets): the chunks in
// descending order of length, by a counting sort over the lengths (stable, so a
// length's chunks stay in vertex order and read neighbouring indices). Partial
// slots and split vertices stay in vertex order.
static int build_plan(mg_graph *g, const std::vector<int32_t> &off, mg_graph::PprPlan *p, cudaStream_t s) {
  const int64_t V = g->nodes;
  int64_t longest = 0;
  for (int64_t v = 0; v < V; ++v) longest = std::max<int64_t>(longest, off[v + 1] - off[v]);
  int32_t chunk = g->edges <= kPprSmall ? 64 : kPprChunk;
  while (chunk < kPprChunk && (int64_t)chunk * chunk < longest) chunk *= 2;
  std::vector<int64_t> at((size_t)chunk + 2, 0);  // at[chunk - len + 1]: chunks of a length, then their first place
  for (int64_t v = 0; v < V; ++v) {
    const int32_t len = off[v + 1] - off[v];
    if (len > chunk) at[1] += len / chunk;
    if (len <= chunk || len % chunk) at[chunk - (len <= chunk ? len : len % chunk) + 1] += 1;
  }
  const int64_t n_empty = at[chunk + 1];
  for (int i = 1; i < chunk + 2; ++i) at[i] += at[i - 1];
  const size_t n = (size_t)at[chunk + 1];
  std::vector<int32_t> cv(n), cb(n), ce(n), cs(n), mv, mf;
  int32_t slots = 0;
  auto put = [&](int64_t v, int32_t b, int32_t e, int32_t slot) {
    const int64_t i = at[chunk - (e - b)]++;
    cv[i] = (int32_t)v;
    cb[i] = b;
    ce[i] = e;
    cs[i] = slot;
  };
  for (int64_t v = 0; v < V; ++v) {
    const int32_t b = off[v], e = off[v + 1];
    if (e - b <= chunk) {
      put(v, b, e, -1);
    } else {
      mv.push_back((int32_t)v);
      mf.push_back(slots);
      for (int32_t x = b; x < e; x += std::min(chunk, e - x)) put(v, x, x + std::min(chunk, e - x), slots++);
    }
  }
  mf.push_back(slots);
  int st;
  const size_t nc = std::max<size_t>(n, 1), nm = std::max<size_t>(mv.size(), 1);
  if ((st = device_alloc(g, (void **)&p->cv, nc * 4)) != MG_OK ||
      (st = device_alloc(g, (void **)&p->cb, nc * 4)) != MG_OK ||
      (st = device_alloc(g, (void **)&p->ce, nc * 4)) != MG_OK ||
      (st = device_alloc(g, (void **)&p->cslot, nc * 4)) != MG_OK ||
      (st = device_alloc(g, (void **)&p->mv, nm * 4)) != MG_OK ||
      (st = device_alloc(g, (void **)&p->mfirst, (nm + 1) * 4)) != MG_OK)
    return st;
  cudaError_t e = cudaSuccess;
  if (!cv.empty()) {
    e = cudaMemcpyAsync(p->cv, cv.data(), cv.size() * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(p->cb, cb.data(), cb.size() * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(p->ce, ce.data(), ce.size() * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(p->cslot, cs.data(), cs.size() * 4, cudaMemcpyHostToDevice, s);
  }
  if (e == cudaSuccess && !mv.empty()) e = cudaMemcpyAsync(p->mv, mv.data(), mv.size() * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(p->mfirst, mf.data(), mf.size() * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, "ppr plan upload");
  p->nchunks = (int32_t)cv.size();
  p->nfull = (int32_t)(cv.size() - (size_t)n_empty);
  p->nmulti = (int32_t)mv.size();
  p->nslots = slots;
  return MG_OK;
}

// Row stride of a solve's matrices.
static int32_t ppr_stride(int32_t nvec) { return (nvec + 3) & ~3; }
// Lanes per chunk: a power of two of 4-column lanes that covers a row.
static int ppr_group(int32_t nv) {
  int gsz = 1;
  while (gsz * 4 < nv) gsz *= 2;
  return gsz;
}

static int ppr_prepare(mg_graph *g, int32_t nv, cudaStream_t s) {
  int st;
  if (!g->ppr_plan[0].cv) {
    const int64_t V = g->nodes;
    std::vector<int32_t> co((size_t)V + 1), ro((size_t)V + 1);
    cudaError_t e = cudaMemcpyAsync(co.data(), g->csr.csc_offsets, (V + 1) * 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ro.data(), g->csr.row_offsets, (V + 1) * 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "ppr plan read");
    if ((st = build_plan(g, co, &g->ppr_plan[0], s)) != MG_OK) return st;
    if ((st = build_plan(g, ro, &g->ppr_plan[1], s)) != MG_OK) return st;
  }
  if (g->ppr_cap_nvec < nv) {
    const size_t V = (size_t)g->nodes;
    const int32_t slots = std::max(std::max(g->ppr_plan[0].nslots, g->ppr_plan[1].nslots), 1);
    if ((st = device_alloc(g, (void **)&g->ppr_x[0], V * nv * 4)) != MG_OK ||
        (st = device_alloc(g, (void **)&g->ppr_x[1], V * nv * 4)) != MG_OK ||
        (st = device_alloc(g, (void **)&g->ppr_rhs, V * nv * 4)) != MG_OK ||
        (st = device_alloc(g, (void **)&g->ppr_partial, (size_t)slots * nv * 4)) != MG_OK)
      return st;
    g->ppr_cap_nvec = nv;
  }
  if (!g->ppr_w && (st = device_alloc(g, (void **)&g->ppr_w, (size_t)g->edges * 4 + 64)) != MG_OK) return st;
  return MG_OK;
}

static bool is_device_ptr(const void *p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

// (vertices + edges) times row width up to which a solve is one launch (forward
// and backward, level loop / one launch: R-MAT 9, 32 columns 2.33 / 1.96 ms,
// R-MAT 14, 2 columns 2.27 / 2.10, R-MAT 16, 7 columns 3.34 / 2.86, R-MAT 18,
// 12 columns 6.54 / 6.90).
constexpr int64_t kPprLoopWork = 1ll << 24;

static int ppr_one_launch(LoopRun &run, mg_graph *g, PprArgs a, uint32_t max_iter, const mg_options *o, const char *name,
                          LoopResult *res) {
  GridLoop loop = run.args(o);
  double tol = o->tolerance;
  void *args[] = {&a, &tol, &max_iter, &loop};
  const void *kernel;
  switch (ppr_group(a.nv)) {
    case 1: kernel = (const void *)k_ppr_loop<1>; break;
    case 2: kernel = (const void *)k_ppr_loop<2>; break;
    case 4: kernel = (const void *)k_ppr_loop<4>; break;
    case 8: kernel = (const void *)k_ppr_loop<8>; break;
    default: kernel = (const void *)k_ppr_loop<16>;
  }
  memset(&res->ctl, 0, sizeof(res->ctl));
  int st = run.launch(kernel, args, true, name);
  if (st != MG_OK || (st = run.finish(cudaSuccess, name)) != MG_OK) return st;
  res->ctl.level = g->loop_out->level;
  res->ctl.residual = g->loop_out->residual;
  res->ctl.acc[2] = g->loop_out->norm;
  float ms = 0.f;
  cudaEventElapsedTime(&ms, g->ev0, g->ev1);
  res->ms = ms;
  return MG_OK;
}

// Runs one power-iteration solve; on return the solution is in *result.
static int ppr_solve(mg_graph *g, int dir, const float *w, const float *rhs, float alpha, int32_t nvec,
                     const mg_options *o, cudaStream_t s, const char *name, float **result, LoopResult *res) {
  const mg_graph::PprPlan &p = g->ppr_plan[dir];
  // The level loop is captured once and replayed: its kernels read the inputs
  // from the graph's own buffers, so callers may pass different pointers.
  const int32_t nv = ppr_stride(nvec);
  const int64_t n = (int64_t)g->nodes * nv;
  // Short iterations: one launch. The level loop serves the rest, the host-driven
  // runs and callers that shorten the waits.
  std::optional<LoopRun> run;
  if (o->use_cuda_graph && !prof_on() && o->spin_limit >= kSpinLimitDefault && (g->nodes + g->edges) * nv <= kPprLoopWork)
    run.emplace(g, s);
  k_rows_f32<<<g->num_sms * 8, 256, 0, s>>>(rhs, nvec, g->ppr_rhs, nv, 1.0f, g->nodes);
  // the weights in the order the solve reads its adjacency (CSC order for the
  // forward pull, so no edge-id indirection per edge and iteration)
  if (dir == 0) k_gather_f32<<<g->num_sms * 4, 256, 0, s>>>(g->csr.csc_eid, w, g->ppr_w, g->edges);
  else k_copy_f32<<<g->num_sms * 4, 256, 0, s>>>(w, g->ppr_w, g->edges);
  count_launch(2);
  w = g->ppr_w;
  rhs = g->ppr_rhs;
  PprArgs a;
  a.idx = dir == 0 ? g->csr.csc_rows : g->csr.col;
  a.w = w;
  a.rhs = rhs;
  a.alpha = alpha;
  a.d = (float)o->damping;
  a.x0 = g->ppr_x[0];
  a.x1 = g->ppr_x[1];
  a.partial = g->ppr_partial;
  a.cv = p.cv;
  a.cb = p.cb;
  a.ce = p.ce;
  a.cslot = p.cslot;
  a.mv = p.mv;
  a.mfirst = p.mfirst;
  a.nchunks = p.nchunks;
  a.nfull = p.nfull;
  a.nmulti = p.nmulti;
  a.nvec = nvec;
  a.nv = nv;
  a.V = g->csr.V;
  a.ctl = g->ws.ctl;
  // start from the right-hand side
  k_copy_f32<<<g->num_sms * 4, 256, 0, s>>>(rhs, a.x0, n);
  count_launch();
  const uint32_t max_iter = (uint32_t)std::max<int32_t>(0, std::min<int32_t>(o->iter_num, 100000));
  if (run) {
    const int st = ppr_one_launch(*run, g, a, max_iter, o, name, res);
    *result = (res->ctl.level & 1) ? a.x1 : a.x0;
    if (st != kLoopRefused) return st;
  }
  k_ctl_init<<<1, 32, 0, s>>>(a.ctl, 1u, max_iter, (unsigned long long)o->spin_limit, MODE_QUEUE, ctl_flags(nullptr));
  k_ppr_rhs_norm<<<g->num_sms * 4, 256, 0, s>>>(rhs, n, a.ctl);
  count_launch(2);
  const int grid = persistent_grid(g, o, 4);
  const double tol = o->tolerance;
  LevelBody body = [=](cudaStream_t ss, cudaGraphConditionalHandle h, int use_h) {
    switch (ppr_group(nv)) {
      case 1: MG_LAUNCH(KID_PPR, ss, k_ppr_iter<1><<<grid, kNT, 0, ss>>>(a)); break;
      case 2: MG_LAUNCH(KID_PPR, ss, k_ppr_iter<2><<<grid, kNT, 0, ss>>>(a)); break;
      case 4: MG_LAUNCH(KID_PPR, ss, k_ppr_iter<4><<<grid, kNT, 0, ss>>>(a)); break;
      case 8: MG_LAUNCH(KID_PPR, ss, k_ppr_iter<8><<<grid, kNT, 0, ss>>>(a)); break;
      default: MG_LAUNCH(KID_PPR, ss, k_ppr_iter<16><<<grid, kNT, 0, ss>>>(a));
    }
    if (nv > 32) MG_LAUNCH(KID_PPR, ss, k_ppr_fixup<2><<<grid, kNT, 0, ss>>>(a));
    else MG_LAUNCH(KID_PPR, ss, k_ppr_fixup<1><<<grid, kNT, 0, ss>>>(a));
    MG_LAUNCH(KID_OTHER, ss, k_ppr_level_end<<<1, 32, 0, ss>>>(a.ctl, tol, h, use_h));
  };
  char key[160];
  // (ppr_cap_nvec: a wider solve replaced the buffers the cached graph's arguments point to)
  snprintf(key, sizeof(key), "%s/%d/%d/%d/%.9g/%.17g/%.17g", name, grid, nvec, g->ppr_cap_nvec, (double)alpha, o->damping,
           tol);
  int st = run_level_loop(g, s, key, 3, body, o->use_cuda_graph != 0, res);
  if (st != MG_OK) return st;
  finish_run(g, res->ctl.level);
  if (res->ctl.error)
    return set_error(res->ctl.error, std::string(name) + ": device reported " + mg_status_string(res->ctl.error));
  *result = (res->ctl.level & 1) ? a.x1 : a.x0;
  return MG_OK;
}

static void ppr_stats(mg_stats *stats, const LoopResult &res, double tol, mg_graph *g) {
  const double tol_total = tol * res.ctl.acc[2];
  if (!stats) return;
  stats->iterations = (int32_t)res.ctl.level;
  stats->push_iterations = 0;
  stats->pull_iterations = (int32_t)res.ctl.level;
  stats->converged = res.ctl.residual <= tol_total ? 1 : 0;
  stats->device_ms = res.ms;
  stats->residual = res.ctl.residual;
  stats->vertices_reached = g->nodes;
  stats->edges_traversed = g->edges * (int64_t)res.ctl.level;
}

static const mg_options *opts_or_default(const mg_options *o, mg_options *d) {
  if (o) return o;
  mg_options_init(d);
  d->tolerance = 1e-7;
  return d;
}

}  // namespace mg

using namespace mg;

extern "C" {

int mg_ppr_forward(mg_graph *g, const float *edge_weights, const float *teleport, int32_t nvec, float *ranks,
                   mg_stats *stats, const mg_options *opts) {
  clear_error();
  if (!g) return set_error(MG_ERR_ARG, "graph is NULL");
  if (nvec < 1 || nvec > kPprMaxVec) return set_error(MG_ERR_ARG, "nvec must be in [1, 64]");
  if (!g->directed)
    return set_error(MG_ERR_UNSUPPORTED, "personalised PageRank needs the transpose: create the graph with directed=1");
  if (!edge_weights || !teleport || !ranks) return set_error(MG_ERR_ARG, "NULL pointer");
  if (!is_device_ptr(edge_weights) || !is_device_ptr(teleport) || !is_device_ptr(ranks))
    return set_error(MG_ERR_ARG, "mg_ppr_forward takes device pointers");
  mg_options d;
  const mg_options *o = opts_or_default(opts, &d);
  if (!(o->damping >= 0.0 && o->damping < 1.0)) return set_error(MG_ERR_ARG, "damping must be in [0, 1)");
  cudaStream_t s = run_stream(g, o);
  int st = prepare_run(g, s);
  if (st != MG_OK || (st = ppr_prepare(g, ppr_stride(nvec), s)) != MG_OK) return st;
  float *x = nullptr;
  LoopResult res;
  if ((st = ppr_solve(g, 0, edge_weights, teleport, (float)(1.0 - o->damping), nvec, o, s, "ppr_fwd", &x, &res)) !=
      MG_OK)
    return st;
  ppr_stats(stats, res, o->tolerance, g);
  const int32_t nv = ppr_stride(nvec);
  if (nv == nvec) return copy_out(s, ranks, x, (size_t)g->nodes * nvec * 4, true);
  // into the other iterate's buffer when a kernel cannot write `ranks`
  const bool direct = on_device(g, ranks);
  float *out = direct ? ranks : x == g->ppr_x[0] ? g->ppr_x[1] : g->ppr_x[0];
  k_rows_f32<<<g->num_sms * 8, 256, 0, s>>>(x, nv, out, nvec, 1.0f, g->nodes);
  count_launch();
  if ((st = launch_check("ppr forward")) != MG_OK) return st;
  if (!direct) return copy_out(s, ranks, out, (size_t)g->nodes * nvec * 4, true);
  return cuda_status(cudaStreamSynchronize(s), "ppr forward");
}

int mg_ppr_backward(mg_graph *g, const float *edge_weights, const float *ranks, const float *grad_ranks, int32_t nvec,
                    float *grad_edge_weights, float *grad_teleport, mg_stats *stats, const mg_options *opts) {
  clear_error();
  if (!g) return set_error(MG_ERR_ARG, "graph is NULL");
  if (nvec < 1 || nvec > kPprMaxVec) return set_error(MG_ERR_ARG, "nvec must be in [1, 64]");
  if (!g->directed)
    return set_error(MG_ERR_UNSUPPORTED, "personalised PageRank needs the transpose: create the graph with directed=1");
  if (!edge_weights || !ranks || !grad_ranks) return set_error(MG_ERR_ARG, "NULL pointer");
  if (!is_device_ptr(edge_weights) || !is_device_ptr(ranks) || !is_device_ptr(grad_ranks) ||
      (grad_edge_weights && !is_device_ptr(grad_edge_weights)) || (grad_teleport && !is_device_ptr(grad_teleport)))
    return set_error(MG_ERR_ARG, "mg_ppr_backward takes device pointers");
  mg_options d;
  const mg_options *o = opts_or_default(opts, &d);
  if (!(o->damping >= 0.0 && o->damping < 1.0)) return set_error(MG_ERR_ARG, "damping must be in [0, 1)");
  cudaStream_t s = run_stream(g, o);
  int st = prepare_run(g, s);
  if (st != MG_OK || (st = ppr_prepare(g, ppr_stride(nvec), s)) != MG_OK) return st;
  float *lam = nullptr;
  LoopResult res;
  if ((st = ppr_solve(g, 1, edge_weights, grad_ranks, 1.0f, nvec, o, s, "ppr_adj", &lam, &res)) != MG_OK) return st;
  const int grid = persistent_grid(g, o, 4);
  if (grad_edge_weights) {
    const mg_graph::PprPlan &pl = g->ppr_plan[1];  // chunks of the out-edge rows
    const int32_t nv = ppr_stride(nvec);
    auto launch = [&](auto kernel) {
      kernel<<<grid, kNT, 0, s>>>(pl.cv, pl.cb, pl.ce, pl.nfull, g->csr.col, nvec, nv, lam, ranks, (float)o->damping,
                                  grad_edge_weights, g->ws.ctl);
    };
    switch (ppr_group(nv)) {
      case 1: launch(k_ppr_edge_grad<1>); break;
      case 2: launch(k_ppr_edge_grad<2>); break;
      case 4: launch(k_ppr_edge_grad<4>); break;
      case 8: launch(k_ppr_edge_grad<8>); break;
      default: launch(k_ppr_edge_grad<16>);
    }
    count_launch();
  }
  if (grad_teleport) {
    k_rows_f32<<<g->num_sms * 8, 256, 0, s>>>(lam, ppr_stride(nvec), grad_teleport, nvec, (float)(1.0 - o->damping),
                                              g->nodes);
    count_launch();
  }
  ppr_stats(stats, res, o->tolerance, g);
  return cuda_status(cudaStreamSynchronize(s), "ppr backward");
}

}  // extern "C"
