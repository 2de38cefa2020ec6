// pm_cc.cu -- Connected Components of a symmetric graph by union-find.
//
// numa-Components.C computes labels by min-label propagation (CC_F
// 55-106, loop 233-281): labels start at the vertex id (387-391) and each
// round lowers a label to the least label among its neighbours.  On a
// symmetric graph the fixpoint is the minimum vertex id of each connected
// component, a value independent of the schedule, so any exact algorithm
// that yields that minimum gives the reference's labels bit for bit.
//
// This file computes it with a concurrent union-find in the scheme of
// Afforest (Sutton, Ben-Nun and Barak, IPDPS 2018), in one cooperative launch:
//   1. every vertex hangs under its first neighbour when that is smaller (its
//      own entry only: no atomics; rows are usually sorted, so this is mostly
//      the least neighbour), and the trees are compressed;
//   2. every vertex links to its second neighbour, and the trees are
//      compressed again;
//   3. the root shared by most of kModeSamples spread vertices is taken as the
//      largest intermediate component L;
//   4. every vertex not under L links to all its neighbours.  A vertex of L
//      skips them: an edge between L and another component is also stored the
//      other way round (the graph is symmetric), and the other endpoint, not
//      in L, links it; an edge inside L needs nothing;
//   5. a last compression points every vertex at its root.
// Links always hang the larger root under the smaller one (with a CAS in steps
// 2 and 4), so parent[v] <= v holds throughout, a root is the least id of its
// tree, and the final root of each component is its minimum vertex id: exactly
// the labels of the propagation.  The parent array is the caller's label array.
// Label propagation stays available (tunable PM_TUNE_CC_MODE = 1) and is
// what directed and partitioned handles use.
//
// What bounds it: the dependent reads id -> parent -> parent of a few million
// vertices.  Each thread therefore follows kStep vertices side by side, in the
// links too, and the compressions read parents through L1 (a stale parent is an
// ancestor too), where most trees end.  Symmetrised 2^22-vertex, 128 M-edge
// R-MAT: 407 us as eight kernels, 244 in one launch whose links went one after
// another, 180 here; the grid without 30 % of its edges 775, 1336 and 734 us
// (with half the eight kernels' threads its links, 944 us of it, took as many
// more steps in a row).
#include <algorithm>

#include "pm_rounds.cuh"

namespace pm {

constexpr int kModeSamples = kRoundThreads;
constexpr int kFewEdges = 16;  // of a row that its own lane links in step 4

__device__ __forceinline__ int32_t ld_parent(const int32_t *p, int32_t v) {
  return *((volatile const int32_t *)p + v);
}

// Hangs the root of u's tree and the root of v's tree together, the larger
// under the smaller (Afforest's link).
__device__ __forceinline__ void uf_link(int32_t *parent, int32_t u, int32_t v) {
  int32_t p1 = ld_parent(parent, u), p2 = ld_parent(parent, v);
  while (p1 != p2) {
    const int32_t high = max(p1, p2), low = min(p1, p2);
    const int32_t p_high = ld_parent(parent, high);
    if (p_high == low) break;  // already hung there
    if (p_high == high && atomicCAS(parent + high, high, low) == high) break;  // high was a root
    p1 = ld_parent(parent, ld_parent(parent, high));
    p2 = ld_parent(parent, low);
  }
}

// The same for kStep pairs of parents (p1[u], p2[u]) side by side: their chains
// of dependent reads overlap.  Pairs that are equal are linked already.
__device__ __forceinline__ void uf_link_each(int32_t *parent, int32_t (&p1)[kStep], int32_t (&p2)[kStep]) {
  for (;;) {
    int32_t above[kStep], low[kStep];
    bool more = false;
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      low[u] = min(p1[u], p2[u]);
      above[u] = p1[u] != p2[u] ? ld_parent(parent, max(p1[u], p2[u])) : low[u];
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const int32_t high = max(p1[u], p2[u]);
      // a root is hung under low; when another thread was first, above is its choice
      if (above[u] == high && above[u] != low[u]) {
        above[u] = atomicCAS(parent + high, high, low[u]);
        if (above[u] == high) above[u] = low[u];
      }
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const bool open = above[u] != low[u];
      p1[u] = open ? ld_parent(parent, above[u]) : low[u];
      p2[u] = open ? ld_parent(parent, low[u]) : low[u];
      more |= open;
    }
    if (!more) break;
  }
}

// Steps a compression takes before it stores its jumps, and before it reads
// past L1 as well: most trees are no deeper than the first.  Once every thread
// does both, all chains shorten together (pointer doubling): a path of n
// vertices in id order takes log n steps, not n.  With both at 8 a 2048 x 2048
// grid takes 403 us and one without 30 % of its edges 885; with both at 2 191
// and 784, but a symmetrised 2^21-vertex graph of mostly near neighbours 227
// instead of 183; as they are 229, 734 and 169.
constexpr int kPublish = 2, kPastL1 = 8;

// parent[v] := root of v, for every v.  Writes only v's own entry; a reader of
// parent[v] meanwhile sees either the old value or the root, both ancestors.
__device__ __forceinline__ void uf_compress(int32_t *parent, int64_t n) {
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v0 = gtid; v0 < n; v0 += kStep * gsize) {
    int32_t old[kStep], p[kStep], q[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) old[u] = p[u] = __ldca(parent + min(v0 + u * gsize, n - 1));
#pragma unroll
    for (int u = 0; u < kStep; ++u) q[u] = __ldca(parent + p[u]);
    for (int step = 0;; ++step) {
      bool more = false;
#pragma unroll
      for (int u = 0; u < kStep; ++u)
        if (p[u] != q[u]) {
          p[u] = q[u];
          if (step >= kPublish && v0 + u * gsize < n) parent[v0 + u * gsize] = p[u];
          q[u] = step < kPastL1 ? __ldca(parent + q[u]) : ld_parent(parent, q[u]);
          more |= p[u] != q[u];
        }
      if (!more) break;
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u)
      if (v0 + u * gsize < n && p[u] != old[u]) parent[v0 + u * gsize] = p[u];
  }
}

// The root most of kModeSamples spread vertices share (ties: the smaller
// root), by every block for itself; the vertices are v = i * n / S.
__device__ __forceinline__ int32_t uf_mode(const int32_t *parent, int64_t n) {
  __shared__ int32_t s_root[kModeSamples];
  __shared__ unsigned long long s_best;
  const int i = threadIdx.x;
  const int32_t root = __ldca(parent + (int64_t)i * n / kModeSamples);  // compressed: its parent is its root
  s_root[i] = root;
  if (i == 0) s_best = ~0ull;
  __syncthreads();
  int cnt = 0;
#pragma unroll 8
  for (int j = 0; j < kModeSamples; ++j) cnt += s_root[j] == root;
  // key: larger count first, then smaller root
  const unsigned long long key = ((unsigned long long)(kModeSamples - cnt) << 32) | (uint32_t)root;
  if (key < s_best) atomicMin(&s_best, key);
  __syncthreads();
  return (int32_t)(uint32_t)(s_best & 0xffffffffull);
}

__global__ void __launch_bounds__(kRoundThreads, 2) k_uf(GraphView g, int32_t *parent, unsigned long long *edges) {
  cg::grid_group grid = cg::this_grid();
  const int lane = lane_id();
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (int64_t)gridDim.x * blockDim.x;
  const int64_t n = g.n;
  if (gtid == 0) *edges = 0;
  unsigned long long mine = 0;
  // 1. first neighbours
  for (int64_t v0 = gtid; v0 < n; v0 += kStep * gsize) {
    int32_t o0[kStep], o1[kStep], d[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const int64_t v = min(v0 + u * gsize, n - 1);
      o0[u] = __ldg(g.out.off + v);
      o1[u] = __ldg(g.out.off + v + 1);
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) d[u] = o0[u] < o1[u] ? checked_id(g, __ldg(g.out.idx + o0[u])) : INT32_MAX;
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const int64_t v = v0 + u * gsize;
      if (v < n) {
        parent[v] = min(d[u], (int32_t)v);
        mine += d[u] != INT32_MAX;
      }
    }
  }
  grid.sync();
  uf_compress(parent, n);
  grid.sync();
  // 2. second neighbours
  for (int64_t v0 = gtid; v0 < n; v0 += kStep * gsize) {
    int32_t o0[kStep], o1[kStep], d[kStep], pv[kStep], pd[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const int64_t v = min(v0 + u * gsize, n - 1);
      o0[u] = __ldg(g.out.off + v) + 1;
      o1[u] = v0 + u * gsize < n ? __ldg(g.out.off + v + 1) : 0;
      pv[u] = ld_parent(parent, (int32_t)v);
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) d[u] = o0[u] < o1[u] ? checked_id(g, __ldg(g.out.idx + o0[u])) : -1;
#pragma unroll
    for (int u = 0; u < kStep; ++u) pd[u] = d[u] >= 0 ? ld_parent(parent, d[u]) : 0;
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      mine += d[u] >= 0;
      if (d[u] < 0) pd[u] = pv[u];
    }
    uf_link_each(parent, pv, pd);
  }
  grid.sync();
  uf_compress(parent, n);
  grid.sync();
  // 3. and 4.: a warp takes 32 * kStep vertices; a vertex outside the largest
  // component links its neighbours itself when they are few, side by side with
  // the lane's other vertices, else the whole warp does
  const int32_t L = uf_mode(parent, n);
  grid.sync();  // every block has chosen, from the same trees: they agree on L
  for (int64_t base = gtid - lane; base < n; base += kStep * gsize) {
    int32_t p[kStep], o0[kStep], o1[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const int64_t v = min(base + u * gsize + lane, n - 1);
      p[u] = ld_parent(parent, (int32_t)v);
      o0[u] = __ldg(g.out.off + v);
      o1[u] = base + u * gsize + lane < n ? __ldg(g.out.off + v + 1) : 0;
    }
    int32_t few = 0;  // the longest of this lane's short rows
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      if (p[u] == L || o0[u] > o1[u]) o1[u] = o0[u];  // nothing to do
      if (o1[u] - o0[u] <= kFewEdges) few = max(few, o1[u] - o0[u]);
    }
    for (int32_t k = 0; k < few; ++k) {
      int32_t d[kStep], pd[kStep];
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        const bool on = k < o1[u] - o0[u] && o1[u] - o0[u] <= kFewEdges;
        d[u] = on ? checked_id(g, __ldg(g.out.idx + o0[u] + k)) : -1;
        mine += on && k >= 2;  // the first two were counted above
      }
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        pd[u] = d[u] >= 0 ? ld_parent(parent, d[u]) : p[u];
      }
      uf_link_each(parent, p, pd);
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      if (o1[u] - o0[u] <= kFewEdges) o1[u] = o0[u];
      unsigned todo = __ballot_sync(0xffffffffu, o0[u] < o1[u]);
      while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1;
        const int32_t v = (int32_t)(base + u * gsize + l);
        const EdgePos e1 = __shfl_sync(0xffffffffu, o1[u], l);
        const EdgePos first = __shfl_sync(0xffffffffu, o0[u], l);
        for (EdgePos e = first + lane; e < e1; e += 32) {
          uf_link(parent, v, checked_id(g, __ldg(g.out.idx + e)));
          mine += e >= first + 2;  // the first two were counted above
        }
      }
    }
  }
  mine = warp_sum(mine);
  if (lane == 0 && mine) atomicAdd(edges, mine);
  grid.sync();
  uf_compress(parent, n);
}

void run_cc_union_find(pm_graph *g, int32_t *d_labels, pm_traversal_stats *st) {
  Engine &E = g->E;
  unsigned long long *edges = &E.d_cnt->edges;
  static const int per_sm = round_occupancy(k_uf);
  E.prof.begin("cc", E.stream);
  PM_LAUNCH_COOP(k_uf, round_grid(E, per_sm), kRoundThreads, E.stream, E.g, d_labels, edges);
  E.prof.end(E.stream);
  if (st) {
    // this launch raises no error word: only its own count is read
    PM_CUDA(cudaMemcpyAsync(&E.h_cnt->edges, edges, sizeof *edges, cudaMemcpyDeviceToHost, E.stream));
    PM_CUDA(cudaStreamSynchronize(E.stream));
    pm_traversal_stats s{};
    s.rounds = 3;  // union-find passes over the vertices
    s.dense_rounds = 0;
    s.edges_visited = (int64_t)E.h_cnt->edges;  // edges linked
    s.reached = g->n;
    *st = s;
  }
}

}  // namespace pm
