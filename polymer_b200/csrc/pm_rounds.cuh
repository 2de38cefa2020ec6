// pm_rounds.cuh -- traversals whose rounds run inside one cooperative launch:
// what BFS and BellmanFord share.  The direction rule needs the frontier's
// size and out-degree sum after every round; a host loop reads them back
// (about 20 us of idle GPU per round), and a CUDA graph with a WHILE node
// still pays eight small launches a round.  Here a round costs one grid
// barrier (about 2 us) beyond its own work.
#pragma once
#include <cooperative_groups.h>

#include "pm_graph.cuh"

namespace pm {

namespace cg = cooperative_groups;

constexpr int kRoundThreads = 512;
constexpr int kShortRow = 32;      // out-degree below which a frontier vertex is queued whole
constexpr int kPushChunk = 256;    // edges of one queued piece of a longer row

// A frontier as a sparse round reads it: vertices with short rows, and the
// longer rows cut into pieces, so that every warp's share is bounded by
// 32 short rows or one piece whatever the degrees.
struct RoundQueue {
  int32_t *rows;    // vertices with 1 .. kShortRow - 1 out-edges
  int2 *pieces;     // (vertex, first out-edge of the piece relative to the row)
};

// What a round counts of the frontier it makes.  Three slots take turns: the
// one a round reads, the one it fills, the one it clears for the next.
struct RoundCount {
  unsigned long long size, edges;  // |F| and the sum of out-degrees of F
  unsigned rows, pieces;           // queue lengths
};

// Rounds of one launch.  A traversal can take as many rounds as the graph has
// vertices (a path; a negative cycle until it is given up), and a launch that
// ran them all would hold the GPU for minutes: after this many it returns, the
// host looks at RoundsEnd and launches it again from the queue or bitmap it
// left.  A round takes 3 us or more, a launch and a wait about 15 us.
constexpr int kRoundsPerLaunch = 1024;

// How a launch ended, in pinned memory, and where the next one goes on.
struct RoundsEnd {
  pm_traversal_stats stats;
  int32_t level;       // the next round
  int32_t more;        // its frontier is not empty
  int32_t have_bits;   // the frontier is held as a bitmap (else as a queue)
  int32_t flushed;     // multi-source BFS: levels below have their depths written
};
static_assert(sizeof(RoundsEnd) <= 3 * sizeof(Counters), "written to the pinned counter words");

// Queue room for any frontier of a graph with m edges: vertices with long
// rows number at most m / kShortRow.
inline size_t round_pieces(int64_t m) { return (size_t)(m / kShortRow + m / kPushChunk + 1); }

constexpr int kStep = 4;  // edges or vertices a lane has in flight

__device__ __forceinline__ int round_pieces_of(int deg) { return edge_pieces(deg, kPushChunk); }

// Writes the pieces of the lanes' long rows (n pieces of v from slot at on):
// a lane writes a few itself, a hub's are written by the whole warp.
__device__ __forceinline__ void round_write_pieces(const RoundQueue &q, int v, int n, unsigned at) {
  const int lane = lane_id();
  if (n <= 4)
    for (int k = 0; k < n; ++k) q.pieces[at + k] = make_int2(v, k * kPushChunk);
  unsigned longs = __ballot_sync(0xffffffffu, n > 4);
  while (longs) {
    const int l = __ffs(longs) - 1;
    longs &= longs - 1;
    const int hv = __shfl_sync(0xffffffffu, v, l), hn = __shfl_sync(0xffffffffu, n, l);
    const unsigned ha = __shfl_sync(0xffffffffu, at, l);
    for (int k = lane; k < hn; k += 32) q.pieces[ha + k] = make_int2(hv, k * kPushChunk);
  }
}

// Appends the lanes' vertices d[u] (act[u]: there is one, with out-degree
// deg[u]) to q: one reservation per queue and warp.  All lanes call it.
__device__ __forceinline__ void round_append(const bool (&act)[kStep], const int (&d)[kStep], const int (&deg)[kStep],
                                             const RoundQueue &q, RoundCount *c) {
  int rows = 0, pieces = 0;
#pragma unroll
  for (int u = 0; u < kStep; ++u)
    if (act[u]) {
      rows += deg[u] > 0 && deg[u] < kShortRow;
      pieces += deg[u] >= kShortRow ? round_pieces_of(deg[u]) : 0;
    }
  if (!__any_sync(0xffffffffu, rows | pieces)) return;
  int rtot, ptot;
  const int rpos = warp_excl_scan(rows, &rtot), ppos = warp_excl_scan(pieces, &ptot);
  unsigned rb = 0, pb = 0;
  if (lane_id() == 0) {
    if (rtot) rb = atomicAdd(&c->rows, (unsigned)rtot);
    if (ptot) pb = atomicAdd(&c->pieces, (unsigned)ptot);
  }
  unsigned ra = __shfl_sync(0xffffffffu, rb, 0) + rpos, pa = __shfl_sync(0xffffffffu, pb, 0) + ppos;
#pragma unroll
  for (int u = 0; u < kStep; ++u) {
    if (act[u] && deg[u] > 0 && deg[u] < kShortRow) q.rows[ra++] = d[u];
    if (ptot) {  // the same for the whole warp
      const int n = act[u] && deg[u] >= kShortRow ? round_pieces_of(deg[u]) : 0;
      round_write_pieces(q, d[u], n, pa);
      pa += n;
    }
  }
}

// The same for the vertices of a block's tile: one reservation per block and
// queue.  All threads of the block call it.
__device__ __forceinline__ void round_append_block(const bool (&act)[kStep], const int (&v)[kStep],
                                                   const int (&deg)[kStep], const RoundQueue &q, RoundCount *c) {
  constexpr int kWarps = kRoundThreads / 32;
  __shared__ unsigned s_rows[kWarps], s_pieces[kWarps];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  int rows = 0, pieces = 0;
#pragma unroll
  for (int u = 0; u < kStep; ++u)
    if (act[u]) {
      rows += deg[u] > 0 && deg[u] < kShortRow;
      pieces += deg[u] >= kShortRow ? round_pieces_of(deg[u]) : 0;
    }
  int rtot, ptot;
  const int rpos = warp_excl_scan(rows, &rtot), ppos = warp_excl_scan(pieces, &ptot);
  if (lane == 0) {
    s_rows[wid] = rtot;
    s_pieces[wid] = ptot;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int rall, pall;
    const int re = warp_excl_scan(lane < kWarps ? (int)s_rows[lane] : 0, &rall);
    const int pe = warp_excl_scan(lane < kWarps ? (int)s_pieces[lane] : 0, &pall);
    unsigned rb = 0, pb = 0;
    if (lane == 0) {
      if (rall) rb = atomicAdd(&c->rows, (unsigned)rall);
      if (pall) pb = atomicAdd(&c->pieces, (unsigned)pall);
    }
    rb = __shfl_sync(0xffffffffu, rb, 0);
    pb = __shfl_sync(0xffffffffu, pb, 0);
    if (lane < kWarps) {
      s_rows[lane] = rb + re;
      s_pieces[lane] = pb + pe;
    }
  }
  __syncthreads();
  unsigned ra = s_rows[wid] + rpos, pa = s_pieces[wid] + ppos;
#pragma unroll
  for (int u = 0; u < kStep; ++u) {
    if (act[u] && deg[u] > 0 && deg[u] < kShortRow) q.rows[ra++] = v[u];
    if (ptot) {
      const int n = act[u] && deg[u] >= kShortRow ? round_pieces_of(deg[u]) : 0;
      round_write_pieces(q, v[u], n, pa);
      pa += n;
    }
  }
  __syncthreads();  // the arrays are free again
}

// The three counts cleared and the frontier {v} queued, by one warp.
__device__ __forceinline__ void round_start(const GraphView &g, int v, const RoundQueue &q, RoundCount *c) {
  if (lane_id() < 3) c[lane_id()] = RoundCount{};
  __syncwarp();
  const int deg0 = __ldg(g.out.off + v + 1) - __ldg(g.out.off + v);
  const bool act[kStep] = {lane_id() == 0, false, false, false};
  const int d[kStep] = {v, 0, 0, 0}, deg[kStep] = {deg0, 0, 0, 0};
  round_append(act, d, deg, q, c);
  if (lane_id() == 0) {
    c->size = 1;
    c->edges = (unsigned)deg0;
  }
}

// Adds the block's sums to the count: one atomic per block and word.
__device__ __forceinline__ void round_count_add(unsigned long long size, unsigned long long edges, RoundCount *c) {
  __shared__ unsigned long long s_size[kRoundThreads / 32], s_edges[kRoundThreads / 32];
  size = warp_sum(size);
  edges = warp_sum(edges);
  if (lane_id() == 0) {
    s_size[threadIdx.x >> 5] = size;
    s_edges[threadIdx.x >> 5] = edges;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < kRoundThreads / 32; ++i) {
      size += s_size[i];
      edges += s_edges[i];
    }
    if (size) atomicAdd(&c->size, size);
    if (edges) atomicAdd(&c->edges, edges);
  }
  __syncthreads();  // the arrays are free again
}

// A round's counts, by one lane per warp.  Reading them through shared memory
// or with plain loads saves the warps' requests for the same words (5 us a
// round), but the compiler then takes the queue lengths for uniform and the
// push loops it makes from them run at half the speed (BellmanFord at 2^22
// vertices 1.16 -> 1.81 ms with the same instructions and L2 traffic).
__device__ __forceinline__ RoundCount round_read(const RoundCount *c) {
  const volatile RoundCount *v = c;
  RoundCount f{};
  if (lane_id() == 0) {
    f.size = v->size;
    f.edges = v->edges;
    f.rows = v->rows;
    f.pieces = v->pieces;
  }
  f.size = __shfl_sync(0xffffffffu, f.size, 0);
  f.edges = __shfl_sync(0xffffffffu, f.edges, 0);
  f.rows = __shfl_sync(0xffffffffu, f.rows, 0);
  f.pieces = __shfl_sync(0xffffffffu, f.pieces, 0);
  return f;
}

// For every out-edge e = s -> d of the queued frontier: relax(x, e, d, ok) on
// kStep edges per lane at a time (ok marks those there are), all lanes of a
// warp together; x = src(s), read once per piece or row.  A relax does its
// loads, atomics and appends for the four edges side by side: a step costs
// one chain of latencies, not four.  A small frontier is spread thinner (an
// eighth of a piece, or a single row, per warp) so that its round is one step.
template <class Src, class Relax>
__device__ __forceinline__ void round_push(const GraphView &g, const RoundQueue &q, unsigned rows, unsigned pieces,
                                           Src &&src, Relax &&relax) {
  const int lane = lane_id();
  const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
  const unsigned parts = pieces <= warps / 8 ? 8 : pieces <= warps / 2 ? 2 : 1, part_len = kPushChunk / parts;
  for (unsigned i = warp; i < pieces * parts; i += warps) {
    const int2 p = q.pieces[i / parts];
    const EdgeSpan share =
        edge_share(__ldg(g.out.off + p.x), __ldg(g.out.off + p.x + 1), (EdgePos)p.y, i % parts, part_len);
    const int x = src(p.x);
    for (EdgePos b = share.begin; b < share.end; b += 32 * kStep) {
      int xs[kStep], d[kStep];
      EdgePos e[kStep];
      bool ok[kStep];
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        xs[u] = x;
        e[u] = b + 32 * u + lane;
        ok[u] = e[u] < share.end;
        d[u] = ok[u] ? checked_id(g, __ldg(g.out.idx + e[u])) : 0;
      }
      relax(xs, e, d, ok);
    }
  }
  const unsigned per = rows <= warps ? 1 : rows <= warps * 8 ? 8 : 32;  // rows a warp takes
  for (unsigned base = warp * per; base < rows; base += warps * per) {
    int x = 0, o = 0, deg = 0;
    if (lane < (int)per && base + lane < rows) {
      const int v = q.rows[base + lane];
      o = __ldg(g.out.off + v);
      deg = __ldg(g.out.off + v + 1) - o;
      x = src(v);
    }
    int total;
    const int pos = warp_excl_scan(deg, &total);
    for (int b = 0; b < total; b += 32 * kStep) {
      int xs[kStep], d[kStep];
      EdgePos e[kStep];
      bool ok[kStep];
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        const int k = b + 32 * u + lane;
        ok[u] = k < total;
        int j = 0;  // last vertex whose first flat edge is <= k
        if (b + 32 * u < total) {  // the same for the whole warp
#pragma unroll
          for (int step = 16; step > 0; step >>= 1)
            if (__shfl_sync(0xffffffffu, pos, j + step) <= k) j += step;
          xs[u] = __shfl_sync(0xffffffffu, x, j);
          e[u] = (EdgePos)__shfl_sync(0xffffffffu, o, j) + (EdgePos)(k - __shfl_sync(0xffffffffu, pos, j));
        }
        d[u] = ok[u] ? checked_id(g, __ldg(g.out.idx + e[u])) : 0;
      }
      relax(xs, e, d, ok);
    }
  }
}

// Frontier bitmap -> queue, a word of 32 vertices per thread: the vertices are
// counted, the block reserves its slots, and they are written.  All threads of
// the grid call it; a barrier must follow before the queue is read.
__device__ __forceinline__ void round_bits_to_queue(const GraphView &g, const uint32_t *bits, const RoundQueue &q,
                                                    RoundCount *c) {
  const int64_t words = ((int64_t)g.n + 31) / 32, gsize = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < words; base += gsize) {
    const int64_t i = base + threadIdx.x;
    uint32_t word = i < words ? bits[i] : 0u;
    if (i == words - 1 && (g.n & 31)) word &= (1u << (g.n & 31)) - 1u;
    // each warp takes the set bits of its words, kStep per lane and step
    while (__any_sync(0xffffffffu, word != 0u)) {
      bool act[kStep];
      int v[kStep], deg[kStep];
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        act[u] = word != 0u;
        v[u] = act[u] ? (int)(i * 32) + __ffs(word) - 1 : 0;
        word &= word - 1u;
      }
#pragma unroll
      for (int u = 0; u < kStep; ++u) deg[u] = act[u] ? __ldg(g.out.off + v[u] + 1) - __ldg(g.out.off + v[u]) : 0;
      round_append(act, v, deg, q, c);
    }
  }
}
// Queue -> frontier bitmap (already cleared).  A frontier vertex without
// out-edges is in no queue and in no edge's way.
__device__ __forceinline__ void round_queue_to_bits(const RoundQueue &q, unsigned rows, unsigned pieces,
                                                    uint32_t *bits) {
  const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x, gsize = gridDim.x * blockDim.x;
  for (unsigned i = gtid; i < rows; i += gsize) atomicOr(bits + (q.rows[i] >> 5), 1u << (q.rows[i] & 31));
  for (unsigned i = gtid; i < pieces; i += gsize) {
    const int2 p = q.pieces[i];
    if (p.y == 0) atomicOr(bits + (p.x >> 5), 1u << (p.x & 31));
  }
}

// Blocks of a traversal: enough threads for the vertices and, at eight edges
// each, the edges; the resident limit at most (a small grid's barrier is
// cheaper).
inline int round_grid(const Engine &E, int per_sm) {
  const int64_t want = std::max<int64_t>(E.g.n, E.g.m / 8) / kRoundThreads + 1;
  return (int)std::min<int64_t>(want, (int64_t)E.num_sms * per_sm);
}
// A kernel's statistics: thread 0 of the grid alone keeps and writes them (in
// shared memory: a copy in every thread's registers costs spills).
#define PM_ROUND_STATS(st, gtid, from)      \
  __shared__ pm_traversal_stats st;         \
  if ((gtid) == 0) st = (from).stats

// Launches launch(from) until the traversal has ended; `from` starts at round 1.
// The stream is idle afterwards.
template <class Launch>
inline pm_traversal_stats run_rounds(Engine &E, Launch &&launch) {
  const RoundsEnd *end = (const RoundsEnd *)E.h_cnt;  // pinned: the kernels write it over the bus
  RoundsEnd from{};
  from.level = 1;
  do {
    launch(from);
    PM_CUDA(cudaStreamSynchronize(E.stream));
    from = *end;
  } while (from.more);
  return from.stats;
}
template <class K>
int round_occupancy(K kernel) {
  int per_sm = 0;
  PM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kRoundThreads, 0));
  return std::max(1, per_sm);
}

}  // namespace pm
