// pm_min.cu -- minimum propagation on whole graphs, every round in one
// cooperative launch: BellmanFord (BF_F numa-BellmanFord.C:61-95, loop
// 166-211) and the label propagation of Components on directed graphs (CC_F
// numa-Components.C:55-119, loop 233-281).  The options of these applications
// (pull or DENSE_FORWARD rounds, delta-stepping, warp-aggregated pushes) and
// partitions run the host loops of pm_apps.cu.
//
// A round pushes val[s] (+ weight) over the frontier's out-edges from queues
// whose rows are cut to bounded pieces (pm_rounds.cuh); the next frontier is
// what fell.  Rounds below the threshold learn that from the atomics' results
// (a stamp keeps a vertex from being queued twice).  BellmanFord's rounds at or
// above it issue atomics without results, skipped when the target's value as this SM
// last saw it is already no larger (values only fall, so one seen earlier is
// never below the current one), and find what fell by comparing with a copy
// taken at the round's start.  Labels pull in those rounds (labels_pull).
//
// What bounds it: the gathers of the targets' values in the one or two rounds
// that push most of the graph (200 G edges/s), and, on small graphs, the
// barriers.  BellmanFord on the symmetrised 2^22-vertex, 128 M-edge R-MAT
// (weights 1..22): 1.69 ms as a host loop -> 1.16 ms here.  Labels: a vertex
// order with locality has six or seven dense rounds, in which pushes lost to the
// host loop's pulls: 2^23 vertices, 76 M edges, most of them to near ids, 2.50 ms
// as a host loop, 3.85 with dense rounds pushed, 1.69 pulled; a directed 2^22-vertex
// R-MAT 1.48, 0.86 and 0.84 ms.
#include "pm_rounds.cuh"
#include "pm_sorted.cuh"

namespace pm {

struct MinWork {
  int32_t *val, *before, *stamp;
  RoundQueue q[2];
  RoundCount *count;  // three slots, level % 3
  RoundsEnd *end;
  // labels: the rows by in-degree, longest first (pm_sorted.cuh)
  const int32_t *order;
  const int2 *long_pieces;  // {vertex, first in-edge of the piece} of the rows [0, rc)
  int32_t np, rc, rh, rm;
};

// The least of m and the labels of in-edges e, e + width, ... below e1.
__device__ __forceinline__ int32_t labels_least(const GraphView &g, const int32_t *val, int32_t m, EdgePos e, EdgePos e1,
                                                int width) {
  for (; e < e1; e += kStep * width) {
    int s[kStep];
    int32_t x[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) s[u] = e + u * width < e1 ? checked_id(g, __ldg(g.in.idx + e + u * width)) : -1;
#pragma unroll
    for (int u = 0; u < kStep; ++u) x[u] = s[u] >= 0 ? val[s[u]] : INT32_MAX;
#pragma unroll
    for (int u = 0; u < kStep; ++u) m = min(m, x[u]);
  }
  return m;
}

// One dense round of label propagation: every vertex takes the least label of
// its in-neighbours, in the frontier or not (one that is not was pushed when
// it fell: taking it again changes nothing), and is queued when it fell.  A
// label another warp lowers meanwhile may be read before or after: the vertex
// that lowered it is in the next frontier.  The rows are split as the
// multi-source BFS splits its own: pieces of the longest by a CTA each, then a
// warp or kSubLanes lanes per row, the short ones in vertex order.
__device__ __forceinline__ void labels_pull(const GraphView &g, const MinWork &w, int32_t level, const RoundQueue &q,
                                            RoundCount *c, unsigned long long &size, unsigned long long &edges) {
  const int lane = lane_id();
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (int64_t)gridDim.x * blockDim.x;
  auto queue_one = [&](bool fell, int v) {  // by the whole warp
    const bool act[kStep] = {fell, false, false, false};
    const int d[kStep] = {v, 0, 0, 0};
    const int deg[kStep] = {fell ? __ldg(g.out.off + v + 1) - __ldg(g.out.off + v) : 0, 0, 0, 0};
    size += fell;
    edges += (unsigned)deg[0];
    round_append(act, d, deg, q, c);
  };
  for (int p = blockIdx.x; p < w.np; p += gridDim.x) {
    const int2 pc = __ldg(w.long_pieces + p);
    const EdgePos e1 = edge_end((EdgePos)pc.y, kOrderPiece, (EdgePos)__ldg(g.in.off + pc.x + 1));
    int32_t m = labels_least(g, w.val, INT32_MAX, (EdgePos)pc.y + threadIdx.x, e1, kRoundThreads);
    m = __reduce_min_sync(0xffffffffu, m);
    bool fell = false;  // queued by the first of the row's pieces to lower it
    if (lane == 0 && m < *((volatile int32_t *)w.val + pc.x) && m < atomicMin(w.val + pc.x, m))
      fell = atomicExch(w.stamp + pc.x, level) != level;
    queue_one(fell, pc.x);
  }
  const int64_t n1 = w.rh - w.rc, n2 = ((int64_t)(w.rm - w.rh) * kSubLanes + 31) / 32;
  for (int64_t t = gtid >> 5; t < n1 + n2; t += gsize >> 5) {
    const bool whole = t < n1;  // the same for the whole warp
    const int r = whole ? w.rc + (int)t : w.rh + (int)((t - n1) * (32 / kSubLanes)) + lane / kSubLanes;
    const int width = whole ? 32 : kSubLanes, sub = whole ? lane : lane % kSubLanes;
    int v = 0;
    int32_t own = 0, m = INT32_MAX;
    if (r < (whole ? w.rh : w.rm)) {
      v = __ldg(w.order + r);
      own = w.val[v];
      m = labels_least(g, w.val, own, (EdgePos)__ldg(g.in.off + v) + sub, __ldg(g.in.off + v + 1), width);
    }
    for (int d = width / 2; d > 0; d >>= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, d));
    const bool fell = sub == 0 && m < own;
    if (fell) w.val[v] = m;
    queue_one(fell, v);
  }
  constexpr int64_t kTile = (int64_t)kRoundThreads * kStep;
  for (int64_t base = blockIdx.x * kTile; base < g.n; base += gridDim.x * kTile) {
    bool act[kStep];
    int v[kStep], deg[kStep];
    EdgePos o[kStep], o1[kStep];
    int32_t own[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const int64_t x = base + u * kRoundThreads + threadIdx.x;
      v[u] = (int)min(x, (int64_t)g.n - 1);
      o[u] = __ldg(g.in.off + v[u]);
      o1[u] = x < g.n ? (EdgePos)__ldg(g.in.off + v[u] + 1) : o[u];
      own[u] = w.val[v[u]];
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      act[u] = false;
      deg[u] = 0;
      if (o1[u] - o[u] >= kSortShort) continue;  // above
      const int32_t m = labels_least(g, w.val, own[u], o[u], o1[u], 1);
      act[u] = m < own[u];
      if (act[u]) {
        w.val[v[u]] = m;
        deg[u] = __ldg(g.out.off + v[u] + 1) - __ldg(g.out.off + v[u]);
        ++size;
        edges += (unsigned)deg[u];
      }
    }
    round_append_block(act, v, deg, q, c);
  }
}

// W: val + weight from the source src (BellmanFord); otherwise every vertex
// starts with its id and in the frontier (labels).
template <bool W>
__global__ void __launch_bounds__(kRoundThreads, 2) k_min_rounds(GraphView g, const int32_t *__restrict__ weight,
                                                                 MinWork w, RoundsEnd from, int32_t src, int64_t threshold) {
  cg::grid_group grid = cg::this_grid();
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (int64_t)gridDim.x * blockDim.x;
  constexpr int64_t kTile = (int64_t)kRoundThreads * kStep;
  const bool fresh = from.level == 1;
  if (fresh)
    for (int64_t v = gtid; v < g.n; v += gsize) {
      w.val[v] = W ? (v == src ? 0 : kDevBFInf) : (int32_t)v;
      w.stamp[v] = 0;
    }
  if (W && fresh && blockIdx.x == 0 && threadIdx.x < 32) round_start(g, src, w.q[0], w.count);
  // the vertices of the block's tiles for which in(v) holds become the frontier
  // q, counted in c
  auto collect = [&](auto &&in, const RoundQueue &q, RoundCount *c) {
    unsigned long long size = 0, edges = 0;
    for (int64_t base = blockIdx.x * kTile; base < g.n; base += gridDim.x * kTile) {
      bool act[kStep];
      int v[kStep], deg[kStep];
#pragma unroll
      for (int i = 0; i < kStep; ++i) {
        const int64_t x = base + i * kRoundThreads + threadIdx.x;
        v[i] = (int)min(x, (int64_t)g.n - 1);
        act[i] = in(v[i]) && x < g.n;
      }
#pragma unroll
      for (int i = 0; i < kStep; ++i) {
        deg[i] = act[i] ? __ldg(g.out.off + v[i] + 1) - __ldg(g.out.off + v[i]) : 0;
        size += act[i];
        edges += (unsigned)deg[i];
      }
      round_append_block(act, v, deg, q, c);
    }
    round_count_add(size, edges, c);
  };
  if (!W && fresh) collect([](int) { return true; }, w.q[0], w.count);
  grid.sync();
  // a source's value as its piece or row is taken: one lowered later in the
  // round is in the next frontier and pushes again
  auto value_of = [&](int s) { return *((volatile int32_t *)w.val + s); };
  PM_ROUND_STATS(st, gtid, from);
  int32_t level = from.level;
  bool more = false;
  for (;; ++level) {
    RoundCount *cur = w.count + (level - 1) % 3, *nxt = w.count + level % 3;
    const RoundCount f = round_read(cur);
    const unsigned long long fsize = f.size, fedges = f.edges;
    if (fsize == 0 || level > (int64_t)g.n + 2) break;  // level - 1 rounds are done
    more = level - from.level == kRoundsPerLaunch;
    if (more) break;
    const bool dense = (long long)(fsize + fedges) >= threshold;
    const RoundQueue &q = w.q[(level - 1) & 1], &qn = w.q[level & 1];
    if (gtid == 0) {
      st.rounds++;
      st.dense_rounds += dense;
      st.edges_visited += (int64_t)fedges;
      w.count[(level + 1) % 3] = RoundCount{};
    }
    if (!W && dense) {
      unsigned long long size = 0, edges = 0;
      labels_pull(g, w, level, qn, nxt, size, edges);
      round_count_add(size, edges, nxt);
    } else if (dense) {
      for (int64_t v0 = gtid; v0 < g.n; v0 += kStep * gsize) {  // four loads in flight
        int32_t x[kStep];
#pragma unroll
        for (int i = 0; i < kStep; ++i) x[i] = w.val[min(v0 + i * gsize, (int64_t)g.n - 1)];
#pragma unroll
        for (int i = 0; i < kStep; ++i)
          if (v0 + i * gsize < g.n) w.before[v0 + i * gsize] = x[i];
      }
      grid.sync();
      round_push(g, q, f.rows, f.pieces, value_of,
                 [&](const int (&x)[kStep], const EdgePos (&e)[kStep], const int (&d)[kStep], const bool (&ok)[kStep]) {
                   int32_t nv[kStep], seen[kStep];
#pragma unroll
                   for (int u = 0; u < kStep; ++u) nv[u] = x[u] + (W && ok[u] ? __ldg(weight + e[u]) : 0);
#pragma unroll
                   for (int u = 0; u < kStep; ++u) seen[u] = ok[u] ? __ldca(w.val + d[u]) : 0;
#pragma unroll
                   for (int u = 0; u < kStep; ++u)
                     if (ok[u] && nv[u] < seen[u]) atomicMin(w.val + d[u], nv[u]);
                 });
      grid.sync();
      collect([&](int v) { return __ldcs(w.val + v) < __ldcs(w.before + v); }, qn, nxt);
    } else {
      unsigned long long size = 0, edges = 0;
      round_push(g, q, f.rows, f.pieces, value_of,
                 [&](const int (&x)[kStep], const EdgePos (&e)[kStep], const int (&d)[kStep], const bool (&ok)[kStep]) {
                   bool act[kStep];
                   int deg[kStep];
                   int32_t nv[kStep];
#pragma unroll
                   for (int u = 0; u < kStep; ++u) {
                     nv[u] = x[u] + (W && ok[u] ? __ldg(weight + e[u]) : 0);
                     act[u] = ok[u] && nv[u] < *((volatile int32_t *)w.val + d[u]);
                   }
#pragma unroll
                   for (int u = 0; u < kStep; ++u) act[u] = act[u] && nv[u] < atomicMin(w.val + d[u], nv[u]);
#pragma unroll
                   for (int u = 0; u < kStep; ++u) act[u] = act[u] && atomicExch(w.stamp + d[u], level) != level;
#pragma unroll
                   for (int u = 0; u < kStep; ++u) {
                     deg[u] = act[u] ? __ldg(g.out.off + d[u] + 1) - __ldg(g.out.off + d[u]) : 0;
                     size += act[u];
                     edges += (unsigned)deg[u];
                   }
                   round_append(act, d, deg, qn, nxt);
                 });
      round_count_add(size, edges, nxt);
    }
    grid.sync();
  }
  if (gtid == 0) *w.end = RoundsEnd{st, level, more, 0, 0};
}

template <bool W>
static pm_traversal_stats run_min(pm_graph *g, const int32_t *weight, int32_t src, int32_t *d_val, int64_t threshold,
                                  const char *tag) {
  Engine &E = g->E;
  const size_t pieces = round_pieces(g->m);
  MinWork w{};
  w.val = d_val;
  if (W) w.before = (int32_t *)g->scratch_buf(37, (size_t)g->n * 4);
  w.stamp = E.defer;
  int2 *pc = (int2 *)g->scratch_buf(0, 2 * pieces * sizeof(int2));
  for (int k = 0; k < 2; ++k) {
    w.q[k].rows = g->subset(k).queue;
    w.q[k].pieces = pc + k * pieces;
  }
  w.count = (RoundCount *)g->scratch_buf(30, 3 * sizeof(RoundCount));
  w.end = (RoundsEnd *)E.h_cnt;
  if (!W) {
    const RowOrder &o = ensure_row_order(g, false);
    w.order = o.order.as<int32_t>();
    w.long_pieces = o.pieces.as<int2>();
    w.np = o.npieces;
    w.rc = o.cuts[0];
    w.rh = o.cuts[1];
    w.rm = o.cuts[2];
  }
  if (!W) PM_CUDA(cudaMemsetAsync(w.count, 0, 3 * sizeof(RoundCount), E.stream));
  static const int per_sm = round_occupancy(k_min_rounds<W>);
  E.prof.begin(tag, E.stream);
  const pm_traversal_stats st = run_rounds(E, [&](const RoundsEnd &from) {
    PM_LAUNCH_COOP((k_min_rounds<W>), round_grid(E, per_sm), kRoundThreads, E.stream, E.g, weight, w, from, src,
                   threshold);
    E.prof.end(E.stream);
  });
  E.prof.set_passes((int)st.rounds);
  return st;
}

void run_bellman_ford_rounds(pm_graph *g, int32_t src, int32_t *d_dist, int64_t threshold, pm_traversal_stats *st) {
  pm_traversal_stats s = run_min<true>(g, g->w_i32_out.as<int32_t>(), src, d_dist, threshold, "bellman_ford");
  if (s.rounds > g->n + 1) fail(PM_ERR_INVALID_ARG, "BellmanFord did not converge");
  s.reached = 1;
  if (st) *st = s;
}

void run_cc_rounds(pm_graph *g, int32_t *d_labels, int64_t threshold, pm_traversal_stats *st) {
  pm_traversal_stats s = run_min<false>(g, nullptr, -1, d_labels, threshold, "cc");
  s.reached = g->n;
  if (st) *st = s;
}

}  // namespace pm
