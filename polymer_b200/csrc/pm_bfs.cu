// pm_bfs.cu -- breadth-first search on whole graphs, every round in one
// cooperative launch (BFS_F numa-BFS.C:59-79, loop 258-296; the host loop of
// pm_apps.cu serves partitions and the cuda_graphs tunable set to 0).
//
// A round takes the direction rule |F| + outdeg(F) >= threshold from counts
// the round before left on the device.  Sparse rounds push from queues whose
// rows are cut to bounded pieces (pm_rounds.cuh) and claim vertices by CAS on
// parents -- the claim also keeps a vertex from being queued twice, so no
// bitmap is kept; dense rounds pull from the frontier bitmap, a thread per
// unvisited vertex, four in-edges at a time, the parent being the first
// in-neighbour in CSC order that is in the frontier.
//
// What bounds it: the latency chain of its rounds (a barrier of about 2 us
// each, the dependent loads id -> bit -> claim), and for the large dense
// rounds the reads of parents, offsets and first in-edges of every unvisited
// vertex.  16 sources on the symmetrised 2^22-vertex, 128 M-edge R-MAT:
// 7.62 ms as a CUDA graph with a WHILE node (eight kernels a round)
// -> 4.2 ms here, of which the first dense round of each is a third.  Two CTAs
// per SM (64 registers): 3.94 ms of kernels, three with spills 4.77.
#include "pm_rounds.cuh"

namespace pm {

struct BfsWork {
  int32_t *parents, *depth;
  uint32_t *bits[2];     // frontier of even / odd levels, valid after a dense round
  RoundQueue q[2];
  RoundCount *count;     // three slots, level % 3
  RoundsEnd *end;
};

// One dense round: next = the unvisited vertices with an in-neighbour in cur.
// A thread takes kStep vertices (a warp kStep words of the bitmap) and reads
// their parents, offsets and first two in-edges side by side: most vertices
// of a large round are settled by those.
__device__ __forceinline__ void bfs_pull(const GraphView &g, const BfsWork &w, const uint32_t *cur, uint32_t *next,
                                         int32_t level, unsigned long long &size, unsigned long long &edges) {
  const int lane = lane_id();
  const int64_t ntot = ((int64_t)g.n + 31) & ~31ll, gsize = (int64_t)gridDim.x * blockDim.x;
  auto in_cur = [&](int s) { return s >= 0 && ((cur[s >> 5] >> (s & 31)) & 1u); };
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ntot; t += kStep * gsize) {
    int parent[kStep];
    EdgePos e[kStep], e1[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) parent[u] = t + u * gsize < g.n ? w.parents[t + u * gsize] : 0;
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      e[u] = e1[u] = 0;
      if (parent[u] == -1) {
        e[u] = __ldg(g.in.off + t + u * gsize);
        e1[u] = __ldg(g.in.off + t + u * gsize + 1);
      } else {
        parent[u] = -1;  // visited: no edges to scan
      }
    }
    {
      int a[kStep], b[kStep];
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        a[u] = e[u] < e1[u] ? checked_id(g, __ldg(g.in.idx + e[u])) : -1;
        b[u] = e[u] + 1 < e1[u] ? checked_id(g, __ldg(g.in.idx + e[u] + 1)) : -1;
      }
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        const bool ha = in_cur(a[u]), hb = in_cur(b[u]);
        parent[u] = ha ? a[u] : hb ? b[u] : -1;
        e[u] = edge_end(e[u], 2, e1[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      if (t - lane + u * gsize >= ntot) break;  // the same for the whole warp
      const int v = (int)(t + u * gsize);
      const EdgePos lim = edge_end(e[u], kPullScan, e1[u]);
      while (e[u] < lim && parent[u] < 0) {
        int s[kStep];
        bool hit[kStep];
#pragma unroll
        for (int k = 0; k < kStep; ++k) s[k] = e[u] + k < lim ? checked_id(g, __ldg(g.in.idx + e[u] + k)) : -1;
#pragma unroll
        for (int k = 0; k < kStep; ++k) hit[k] = in_cur(s[k]);
#pragma unroll
        for (int k = kStep - 1; k >= 0; --k)
          if (hit[k]) parent[u] = s[k];
        e[u] = edge_end(e[u], kStep, lim);
      }
      // rows still open: the warp scans each together
      unsigned open = __ballot_sync(0xffffffffu, parent[u] < 0 && e[u] < e1[u]);
      while (open) {
        const int l = __ffs(open) - 1;
        open &= open - 1;
        const EdgePos o1 = __shfl_sync(0xffffffffu, e1[u], l);
        int found = -1;
        for (EdgePos o = __shfl_sync(0xffffffffu, e[u], l); o < o1 && found < 0; o += 32 * kStep) {
          int s[kStep];
          bool hit[kStep];
#pragma unroll
          for (int k = 0; k < kStep; ++k) {
            const EdgePos x = o + 32 * k + lane;
            s[k] = x < o1 ? checked_id(g, __ldg(g.in.idx + x)) : -1;
          }
#pragma unroll
          for (int k = 0; k < kStep; ++k) hit[k] = in_cur(s[k]);
#pragma unroll
          for (int k = kStep - 1; k >= 0; --k) {
            const unsigned hits = __ballot_sync(0xffffffffu, hit[k]);
            if (hits) found = __shfl_sync(0xffffffffu, s[k], __ffs(hits) - 1);
          }
        }
        if (lane == l) parent[u] = found;
      }
      const unsigned word = __ballot_sync(0xffffffffu, parent[u] >= 0);
      if (lane == 0) next[v >> 5] = word;
      if (parent[u] >= 0) {
        w.parents[v] = parent[u];
        w.depth[v] = level;
        ++size;
        edges += (unsigned)(__ldg(g.out.off + v + 1) - __ldg(g.out.off + v));
      }
    }
  }
}

__global__ void __launch_bounds__(kRoundThreads, 2) k_bfs(GraphView g, BfsWork w, RoundsEnd from, int32_t src,
                                                          int64_t threshold) {
  cg::grid_group grid = cg::this_grid();
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (int64_t)gridDim.x * blockDim.x;
  PM_ROUND_STATS(st, gtid, from);
  if (from.level == 1) {
    for (int64_t v = gtid; v < g.n; v += gsize) {
      w.parents[v] = v == src ? src : -1;
      w.depth[v] = v == src ? 0 : -1;
    }
    if (blockIdx.x == 0 && threadIdx.x < 32) round_start(g, src, w.q[0], w.count);
    grid.sync();
  }
  bool have_bits = from.have_bits, more = false;
  int32_t level = from.level;
  for (;; ++level) {
    RoundCount *cur = w.count + (level - 1) % 3, *nxt = w.count + level % 3;
    RoundCount f = round_read(cur);
    const unsigned long long fsize = f.size, fedges = f.edges;
    more = fsize != 0 && level - from.level == kRoundsPerLaunch;
    if (fsize == 0 || more) break;
    const bool dense = (long long)(fsize + fedges) >= threshold;
    const RoundQueue &q = w.q[(level - 1) & 1], &qn = w.q[level & 1];
    uint32_t *bits = w.bits[(level - 1) & 1], *bits_next = w.bits[level & 1];
    if (gtid == 0) {
      st.rounds++;
      st.dense_rounds += dense;
      st.edges_visited += (int64_t)fedges;
      st.reached += (int64_t)fsize;
      w.count[(level + 1) % 3] = RoundCount{};
    }
    unsigned long long size = 0, edges = 0;
    if (dense) {
      if (!have_bits) {
        for (int64_t i = gtid; i < ((int64_t)g.n + 31) / 32; i += gsize) bits[i] = 0u;
        grid.sync();
        round_queue_to_bits(q, f.rows, f.pieces, bits);
        grid.sync();
      }
      bfs_pull(g, w, bits, bits_next, level, size, edges);
    } else {
      if (have_bits) {
        round_bits_to_queue(g, bits, q, cur);
        grid.sync();
        f = round_read(cur);
      }
      round_push(
          g, q, f.rows, f.pieces, [](int s) { return s; },
          [&](const int (&s)[kStep], const EdgePos (&)[kStep], const int (&d)[kStep], const bool (&ok)[kStep]) {
            bool act[kStep];
            int deg[kStep];
#pragma unroll
            for (int u = 0; u < kStep; ++u) act[u] = ok[u] && *((volatile int32_t *)w.parents + d[u]) == -1;
#pragma unroll
            for (int u = 0; u < kStep; ++u) act[u] = act[u] && atomicCAS(w.parents + d[u], -1, s[u]) == -1;
#pragma unroll
            for (int u = 0; u < kStep; ++u) {
              deg[u] = 0;
              if (act[u]) {
                w.depth[d[u]] = level;
                deg[u] = __ldg(g.out.off + d[u] + 1) - __ldg(g.out.off + d[u]);
                ++size;
                edges += (unsigned)deg[u];
              }
            }
            round_append(act, d, deg, qn, nxt);
          });
    }
    have_bits = dense;
    round_count_add(size, edges, nxt);
    grid.sync();
  }
  if (gtid == 0) *w.end = RoundsEnd{st, level, more, have_bits, 0};
}

void run_bfs_rounds(pm_graph *g, int32_t src, int32_t *d_parents, int32_t *d_depth, int64_t threshold,
                    pm_traversal_stats *st) {
  Engine &E = g->E;
  const size_t pieces = round_pieces(g->m);
  BfsWork w;
  w.parents = d_parents;
  w.depth = d_depth;
  int2 *pc = (int2 *)g->scratch_buf(0, 2 * pieces * sizeof(int2));
  for (int k = 0; k < 2; ++k) {
    w.bits[k] = g->subset(k).bits;
    w.q[k].rows = g->subset(k).queue;
    w.q[k].pieces = pc + k * pieces;
  }
  w.count = (RoundCount *)g->scratch_buf(30, 3 * sizeof(RoundCount));
  w.end = (RoundsEnd *)E.h_cnt;
  static const int per_sm = round_occupancy(k_bfs);
  E.prof.begin("bfs", E.stream);
  const pm_traversal_stats s = run_rounds(E, [&](const RoundsEnd &from) {
    PM_LAUNCH_COOP(k_bfs, round_grid(E, per_sm), kRoundThreads, E.stream, E.g, w, from, src, threshold);
    E.prof.end(E.stream);
  });
  if (st) *st = s;
}

}  // namespace pm
