// pm_batch.cu -- batched workloads: multi-source BellmanFord, 64 int32
// distance lanes per vertex (personalised PageRank: pm_ppr.cu; multi-source
// BFS: pm_msbfs.cu; the parts of a disjoint union: pm_parts.cu).
#include <cub/cub.cuh>

#include "pm_sorted.cuh"

namespace pm {

using u64 = unsigned long long;

// ===========================================================================
// Multi-source BellmanFord, up to 64 sources (BF_F of numa-BellmanFord.C:
// 61-85 with one int32 distance lane per source).  dist is vertex-major,
// 64 lanes per vertex (256 bytes, one warp-wide pair of 128-byte rows);
// active[v] has bit l set when lane l of v fell in the last round.  A round
// follows BF's direction rule on the union frontier (|F| + outdeg(F) >=
// threshold is dense):
//  * dense: eight lanes of a warp (or, for long rows, all) own a CSC row; for
//    each in-edge whose source has active lanes they gather the source's row
//    and take its minimum with the weight added;
//  * sparse: the frontier's out-edges are cut into 32-edge chunks (a scan of
//    the queued out-degrees); for each edge eight lanes of the warp relax the
//    target's with atomicMin and OR those that fell into its next active word.
// Distances only fall, so reading a row another warp is lowering in the same
// round is harmless: the lower value is a real path length and the lane that
// fell is in the next frontier either way.
//
// What bounds it: the instructions around the pull's row gathers (72 % of the
// issue slots at 22 % of the L2's rate with half a warp per row and a test per
// lane; a load, two shuffles and eight add-and-minimum instructions per four
// rows now).  50 sources, 1.5 M vertices, 42 M edges: 9.0 ms with a warp per
// row in vertex order, 6.65 with half a warp per row by in-degree, 4.0 here
// (a dense round 1.25 -> 0.72 ms; the pushes, a warp per edge and two in flight
// before, 0.54 -> about 0.3).
// ===========================================================================
constexpr int kLanes = 64;
// Resident CTAs per SM of the pull: with eight, a row in flight per group of
// lanes, 50 sources on a 1.5 M-vertex, 42 M-edge R-MAT take 4.33 ms; with six
// and two rows in flight 4.44, with five and three 4.72, with four and four
// 4.82.
constexpr int kBfCtas = 8;
constexpr int kBfPushCtas = 6;  // of the push (four, two edges in flight per group: 1 % slower)

// active -> queue of frontier vertices with out-edges (and their degrees);
// size = |F|, edges = outdeg(F), aux = queue length, left in *host (pinned) by
// the last block, which clears c and the ticket for the next round; next is
// cleared for the round, too.  A block takes 1024 vertices at a time, four side
// by side per thread, and reserves their queue slots with one atomic (an atomic
// per warp and 32 vertices took 60 us for a frontier of most of 1.5 M vertices).
__global__ void __launch_bounds__(256) k_bf_multi_frontier(const u64 *__restrict__ active,
                                                           const int32_t *__restrict__ out_off, int64_t n,
                                                           int32_t *__restrict__ queue, int32_t *__restrict__ qdeg,
                                                           u64 *next, Counters *c, u64 *ticket, Counters *host) {
  __shared__ unsigned s_count[8];
  __shared__ unsigned long long s_at, s_size[8], s_edges[8];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  constexpr int U = 4;
  unsigned long long size = 0, edges = 0;
  for (int64_t base = (int64_t)blockIdx.x * (256 * U); base < n; base += (int64_t)gridDim.x * (256 * U)) {
    bool act[U];
    int deg[U];
    unsigned push[U];
    int count = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t v = base + u * 256 + threadIdx.x;
      act[u] = v < n && active[v] != 0ull;
      if (v < n) next[v] = 0ull;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t v = base + u * 256 + threadIdx.x;
      deg[u] = act[u] ? __ldg(out_off + v + 1) - __ldg(out_off + v) : 0;
      size += act[u];
      edges += (unsigned)deg[u];
      push[u] = __ballot_sync(0xffffffffu, deg[u] > 0);
      count += __popc(push[u]);
    }
    if (lane == 0) s_count[wid] = (unsigned)count;
    __syncthreads();
    unsigned before = 0, all = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      before += i < wid ? s_count[i] : 0u;
      all += s_count[i];
    }
    if (threadIdx.x == 0 && all) s_at = atomicAdd(&c->aux, (unsigned long long)all);
    __syncthreads();
    unsigned long long pos = s_at + before;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (deg[u] > 0) {
        const unsigned long long at = pos + __popc(push[u] & ((1u << lane) - 1u));
        queue[at] = (int32_t)(base + u * 256 + threadIdx.x);
        qdeg[at] = deg[u];
      }
      pos += __popc(push[u]);
    }
    __syncthreads();  // s_count and s_at are free again
  }
  size = warp_sum(size);
  edges = warp_sum(edges);
  if (lane == 0) {
    s_size[wid] = size;
    s_edges[wid] = edges;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) {
      size += s_size[i];
      edges += s_edges[i];
    }
    if (size) atomicAdd(&c->size, size);
    if (edges) atomicAdd(&c->edges, edges);
    __threadfence();
    if (atomicAdd(ticket, 1ull) == gridDim.x - 1) {
      host->size = atomicExch(&c->size, 0ull);
      host->edges = atomicExch(&c->edges, 0ull);
      host->aux = atomicExch(&c->aux, 0ull);
      *ticket = 0ull;
      __threadfence_system();
    }
  }
}

// Eight of a row's 64 distances: 32 bytes, one load.
struct Oct {
  int32_t x[8];
};
__device__ __forceinline__ Oct ld_oct(const int32_t *p) {
  Oct v;
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v.x[0]), "=r"(v.x[1]), "=r"(v.x[2]), "=r"(v.x[3]), "=r"(v.x[4]), "=r"(v.x[5]), "=r"(v.x[6]),
                 "=r"(v.x[7])
               : "l"(p));
  return v;
}

// The same past L1: what other warps' atomics have made of it.
__device__ __forceinline__ Oct ld_oct_fresh(const int32_t *p) {
  Oct v;
  asm volatile("ld.volatile.global.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x[0]), "=r"(v.x[1]), "=r"(v.x[2]), "=r"(v.x[3])
               : "l"(p));
  asm volatile("ld.volatile.global.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x[4]), "=r"(v.x[5]), "=r"(v.x[6]), "=r"(v.x[7])
               : "l"(p + 4));
  return v;
}

constexpr int kBfSub = 8;  // lanes per row

// Eight lanes per edge, each group of them eight of the chunk's 32 edges one
// after another: a warp has four targets' rows in flight.
__global__ void __launch_bounds__(256, kBfPushCtas) k_bf_multi_push(const int32_t *__restrict__ out_off,
                                                       const int32_t *__restrict__ out_idx,
                                                       const int32_t *__restrict__ w_out,
                                                       const int32_t *__restrict__ queue,
                                                       const int32_t *__restrict__ qoff, int q, int64_t total,
                                                       int32_t *dist, const u64 *__restrict__ active,
                                                       u64 *next_active) {
  const int lane = lane_id(), sub = lane % kBfSub;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t chunk = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); chunk * 32 < total;
       chunk += warps) {
    const int64_t t0 = chunk * 32;
    // last queue entry whose first edge is <= t0 (qoff is increasing: every
    // queued vertex has at least one out-edge)
    int lo = 0, hi = q - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(qoff + mid) <= t0) lo = mid;
      else hi = mid - 1;
    }
    // queue entries starting inside the chunk mark their first position
    const int bi = lo + 1 + lane;
    unsigned start = 0;
    if (bi < q) {
      const int64_t p = (int64_t)__ldg(qoff + bi) - t0;
      if (p < 32) start = 1u << p;
    }
    start = __reduce_or_sync(0xffffffffu, start);
    const int64_t t = t0 + lane;
    const bool valid = t < total;
    int s = -1, d = 0;
    int32_t w = 0;
    if (valid) {
      const int qi = lo + __popc(start << (31 - lane));
      s = __ldg(queue + qi);
      const int64_t e = (int64_t)__ldg(out_off + s) + (t - __ldg(qoff + qi));
      d = __ldg(out_idx + e);
      w = __ldg(w_out + e);
    }
    int cur = -1;
    unsigned on = 0;  // the active lanes among this thread's eight of the source's
    Oct from;
    for (int j = 0; j < kBfSub; ++j) {
      const int sj = __shfl_sync(0xffffffffu, s, j, kBfSub);
      const int dj = __shfl_sync(0xffffffffu, d, j, kBfSub);
      const int32_t wj = __shfl_sync(0xffffffffu, w, j, kBfSub);
      if (sj >= 0 && sj != cur) {
        cur = sj;
        on = __ldg(reinterpret_cast<const uint8_t *>(active + sj) + sub);
        if (on) from = ld_oct(dist + (int64_t)sj * kLanes + 8 * sub);
      }
      if (sj < 0 || !on) continue;
      // A lane below the distance read here lowers it with an atomic whose
      // result is unused and is marked active: it fell, or another push
      // lowered it further meanwhile (an extra relaxation next round, the same
      // distances).
      int32_t *to = dist + (int64_t)dj * kLanes + 8 * sub;
      const Oct old = ld_oct_fresh(to);
      unsigned fell = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int32_t nv = on >> i & 1u ? from.x[i] + wj : kDevBFInf;
        if (nv < kDevBFInf && nv < old.x[i]) {
          atomicMin(to + i, nv);
          fell |= 1u << i;
        }
      }
      if (fell) atomicOr(reinterpret_cast<unsigned *>(next_active + dj) + sub / 4, fell << 8 * (sub % 4));
    }
  }
}

constexpr int kBfSmallWeight = 1 << 30;

// The least dist[s] + w over this group's in-edges whose sources have active
// lanes: kBfSub edges from e on, then from e + step on, ... below e1.  Eight
// lanes hold a source's row (thread t lanes 8 t .. 8 t + 7), so that one load
// instruction brings four rows.  A lane of such a source that is not active is
// relaxed too: its distance, when finite, is a path's length that was pushed
// when it fell, and pushing it again changes nothing.  An infinite one must
// not be pushed over a negative weight, nor where the sum would wrap: a batch
// with such a weight tests each value.  self: the group's own row, named by
// the places without an edge.  All lanes of the warp call it; the groups may
// have different rows and lengths.  col: dist at this thread's lanes.
__device__ __forceinline__ Oct bf_multi_relax(const int32_t *__restrict__ in_idx, const int32_t *__restrict__ w_in,
                                              const int32_t *col, const u64 *__restrict__ active, int self, EdgePos e,
                                              EdgePos e1, int step) {
  const int t = lane_id() & 7, shift = lane_id() & 24;
  Oct m;
#pragma unroll
  for (int i = 0; i < 8; ++i) m.x[i] = kDevBFInf;
  for (; __any_sync(0xffffffffu, e < e1); e += step) {
    int s = self;
    bool act = false;
    int32_t w = 0;
    if (e + t < e1) {
      s = __ldcs(in_idx + e + t);
      act = __ldg(active + s) != 0ull;
      w = __ldcs(w_in + e + t);
    }
    unsigned todo = (__ballot_sync(0xffffffffu, act) >> shift) & 0xffu;
    const bool plain = __all_sync(0xffffffffu, (unsigned)w <= (unsigned)kBfSmallWeight);
    int j = 0;  // a group that is done repeats its last edge (or place)
    while (__any_sync(0xffffffffu, todo != 0u)) {
      if (todo) j = __ffs(todo) - 1;
      todo &= todo - 1u;
      const int sj = __shfl_sync(0xffffffffu, s, j, 8);
      const int32_t wj = __shfl_sync(0xffffffffu, w, j, 8);
      const Oct v = ld_oct(col + (int64_t)sj * kLanes);
      if (plain) {
#pragma unroll
        for (int i = 0; i < 8; ++i) m.x[i] = __viaddmin_s32(v.x[i], wj, m.x[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (v.x[i] < kDevBFInf) m.x[i] = min(m.x[i], v.x[i] + wj);
      }
    }
  }
  return m;
}
// The four groups' minima of one row, on all of them.
__device__ __forceinline__ Oct bf_multi_join(Oct m) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m.x[i] = min(m.x[i], __shfl_xor_sync(0xffffffffu, m.x[i], 8));
    m.x[i] = min(m.x[i], __shfl_xor_sync(0xffffffffu, m.x[i], 16));
  }
  return m;
}

constexpr int kBfPiece = 512;  // in-edges of one warp's piece of a heavy row

// Dense round, a warp per item: 512-edge pieces of the heavy rows (in-degree >
// g.heavy_deg; they lower the row with atomicMin and OR the fallen lanes into
// next_active, which starts at zero), then the light rows in order of
// in-degree (order: pm_sorted.cu; null: by id), a warp for each of [0, rh) and
// kBfSub lanes for each of [rh, rl).  A light row is relaxed in full by its lanes, which
// write its next_active bytes.
__global__ void __launch_bounds__(256, kBfCtas) k_bf_multi_pull(GraphView g, const int32_t *__restrict__ w_in,
                                                                int32_t *dist, const u64 *__restrict__ active,
                                                                u64 *next_active, int64_t heavy_pieces,
                                                                const int32_t *__restrict__ order, int rh, int rl,
                                                                int k) {
  const int lane = lane_id(), group = lane / kBfSub, t = lane % kBfSub;
  // threads past the k sources read the last used thread's lanes, no further
  // sector, and write nothing (thread 0's, out of order, make the load slower:
  // 50 sources 4.60 instead of 4.20 ms)
  const bool used = 8 * t < k;
  const int32_t *col = dist + 8 * min(t, (k - 1) / 8);
  int64_t item = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (item < heavy_pieces) {
    const int c = (int)(item / (kChunkEdges / kBfPiece));
    const int piece = (int)(item % (kChunkEdges / kBfPiece));
    const int r = __ldg(g.in.hrow + c);
    const int row_end = __ldg(g.in.off + r + 1);
    const int64_t first = (int64_t)__ldg(g.in.off + r) + (int64_t)(c - __ldg(g.in.hfirst + r)) * kChunkEdges +
                          (int64_t)piece * kBfPiece;
    if (first >= row_end) return;
    const EdgePos e0 = (EdgePos)first, e1 = edge_end(e0, kBfPiece, row_end);
    const Oct m = bf_multi_join(bf_multi_relax(g.in.idx, w_in, col, active, r, e0 + kBfSub * group, e1, 32));
    if (group != 0 || !used) return;
    unsigned fell = 0;
    int32_t *p = dist + (int64_t)r * kLanes + 8 * t;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (m.x[i] < *(const volatile int32_t *)(p + i) && m.x[i] < atomicMin(p + i, m.x[i])) fell |= 1u << i;
    if (fell) atomicOr(reinterpret_cast<unsigned *>(next_active + r) + t / 4, fell << 8 * (t % 4));
    return;
  }
  item -= heavy_pieces;
  const bool whole = item < rh;  // the same for the whole warp
  const int64_t r = whole ? item : rh + (32 / kBfSub) * (item - rh) + group;
  int v = 0;
  EdgePos e0 = 0, e1 = 0;
  bool mine = r < rl;
  if (mine) {
    v = order ? __ldg(order + r) : (int)r;
    e0 = __ldg(g.in.off + v);
    e1 = __ldg(g.in.off + v + 1);
    mine = e1 - e0 <= (EdgePos)g.heavy_deg;
    if (!mine) e1 = e0;
  }
  if (!__any_sync(0xffffffffu, mine)) return;
  Oct m = bf_multi_relax(g.in.idx, w_in, col, active, v, whole ? e0 + kBfSub * group : e0, e1, whole ? 32 : kBfSub);
  if (whole) m = bf_multi_join(m);
  if (!mine || !used || (whole && group != 0)) return;
  int4 *row = reinterpret_cast<int4 *>(dist + (int64_t)v * kLanes) + 2 * t;
  const int4 a = row[0], b = row[1];
  const unsigned fell = (m.x[0] < a.x) | (m.x[1] < a.y) << 1 | (m.x[2] < a.z) << 2 | (m.x[3] < a.w) << 3 |
                        (m.x[4] < b.x) << 4 | (m.x[5] < b.y) << 5 | (m.x[6] < b.z) << 6 | (m.x[7] < b.w) << 7;
  if (!fell) return;
  row[0] = make_int4(min(m.x[0], a.x), min(m.x[1], a.y), min(m.x[2], a.z), min(m.x[3], a.w));
  row[1] = make_int4(min(m.x[4], b.x), min(m.x[5], b.y), min(m.x[6], b.z), min(m.x[7], b.w));
  reinterpret_cast<uint8_t *>(next_active + v)[t] = (uint8_t)fell;
}

__global__ void k_bf_multi_init(int32_t *dist, u64 *active, int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * kLanes; i += stride)
    dist[i] = kDevBFInf;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) active[i] = 0ull;
}

__global__ void k_bf_multi_seed(const int32_t *sources, int k, int32_t *dist, u64 *active) {
  const int l = threadIdx.x;
  if (l < k) {
    const int v = sources[l];
    dist[(int64_t)v * kLanes + l] = 0;
    atomicOr(active + v, 1ull << l);
  }
}

// One count per block: the warps' sums meet in shared memory and thread 0
// adds the block's total (blockDim = 32 x 8), so a transpose of millions of
// tiles issues one atomic per block instead of one per warp.
__device__ __forceinline__ void block_count_add(unsigned long long v, unsigned long long *dst) {
  __shared__ unsigned long long s_part[8];
  v = warp_sum(v);
  const int w = threadIdx.y;  // one warp per threadIdx.y (blockDim.x == 32)
  if (threadIdx.x == 0) s_part[w] = v;
  __syncthreads();
  if (threadIdx.x == 0 && w == 0) {
    unsigned long long t = 0;
    for (int i = 0; i < (int)blockDim.y; ++i) t += s_part[i];
    if (t) atomicAdd(dst, t);
  }
}

// dist vertex-major (n x 64) -> out source-major (k x n), through 32x32
// tiles (grid-stride over the vertex tiles); c->size counts the finite
// distances (reached (source, vertex) pairs).
__global__ void __launch_bounds__(256) k_bf_multi_transpose(const int32_t *__restrict__ dist, int64_t n, int k,
                                                            int32_t *__restrict__ out, Counters *c) {
  __shared__ int32_t tile[32][33];
  const int l0 = blockIdx.y * 32;
  unsigned long long reached = 0;
  for (int64_t v0 = (int64_t)blockIdx.x * 32; v0 < n; v0 += (int64_t)gridDim.x * 32) {
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
      const int64_t v = v0 + r;
      tile[r][threadIdx.x] = v < n ? dist[v * kLanes + l0 + threadIdx.x] : kDevBFInf;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
      const int l = l0 + r;
      const int64_t v = v0 + threadIdx.x;
      if (l < k && v < n) {
        const int32_t x = tile[threadIdx.x][r];
        out[(int64_t)l * n + v] = x;
        reached += x < kDevBFInf;
      }
    }
    __syncthreads();
  }
  block_count_add(reached, &c->size);
}

void run_bf_multi(pm_graph *g, const int32_t *d_sources, int k, int32_t *d_dist_out, int64_t threshold,
                  pm_traversal_stats *st) {
  Engine &E = g->E;
  const int64_t n = g->n;
  int32_t *dist = (int32_t *)g->scratch_buf(0, (size_t)n * kLanes * 4);
  u64 *act = (u64 *)g->scratch_buf(1, (size_t)n * 8);
  u64 *nxt = (u64 *)g->scratch_buf(2, (size_t)n * 8);
  int32_t *qdeg = (int32_t *)g->scratch_buf(3, (size_t)n * 4);
  int32_t *qoff = (int32_t *)g->scratch_buf(4, (size_t)n * 4);
  int32_t *queue = g->subset(0).queue;
  size_t tmp_bytes = 0;
  PM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, qdeg, qoff, (int)n, E.stream));
  void *tmp = g->scratch_buf(5, std::max<size_t>(tmp_bytes, 16));
  PM_LAUNCH(k_bf_multi_init, E.grid_for(n * kLanes, 256, 16), 256, 0, E.stream, dist, act, n);
  PM_LAUNCH(k_bf_multi_seed, 1, 64, 0, E.stream, d_sources, k, dist, act);
  static const int push_per_sm = [] {
    int r = 0;
    PM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_bf_multi_push, 256, 0));
    return std::max(r, 1);
  }();
  const int64_t heavy_pieces = (int64_t)E.g.in.nchunks * (kChunkEdges / kBfPiece);
  // without memory for the order, a warp per row in vertex order
  const RowOrder *o = find_row_order(g, false);
  const int32_t *order = o ? o->order.as<int32_t>() : nullptr;
  const int rh = o ? o->cuts[1] : (int)n, rl = o ? o->cuts[3] : (int)n;
  const int64_t items = heavy_pieces + rh + ((int64_t)(rl - rh) * kBfSub + 31) / 32;
  const unsigned pull_grid = (unsigned)((items + 7) / 8);
  const int32_t *w_in = g->w_i32_in.as<int32_t>(), *w_out = g->w_i32_out.as<int32_t>();
  pm_traversal_stats s{};
  E.tag = "bellman_ford_multi";
  PM_CUDA(cudaMemsetAsync(E.d_cnt, 0, 3 * sizeof(Counters), E.stream));
  for (;;) {
    // a round trip: this launch and a wait (with the counters copied back and
    // two words cleared by memsets it took about 35 us)
    PM_LAUNCH(k_bf_multi_frontier, E.grid_for((n + 3) / 4, 256, 8), 256, 0, E.stream, act, E.g.out.off, n, queue, qdeg,
              nxt, E.d_cnt + 1, &E.d_cnt[2].aux, E.h_cnt);
    PM_CUDA(cudaStreamSynchronize(E.stream));
    const int64_t size = (int64_t)E.h_cnt->size, edges = (int64_t)E.h_cnt->edges, q = (int64_t)E.h_cnt->aux;
    if (size == 0) break;
    if (s.rounds > n + 1) fail(PM_ERR_INVALID_ARG, "BellmanFord did not converge");
    s.edges_visited += edges;
    const bool dense = size + edges >= threshold;
    E.prof.begin(E.tag, E.stream);
    if (dense) {
      if (items > 0)
        PM_LAUNCH(k_bf_multi_pull, pull_grid, 256, 0, E.stream, E.g, w_in, dist, act, nxt, heavy_pieces,
                  order, rh, rl, k);
    } else {
      if (q > 0) {
        PM_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, qdeg, qoff, (int)q, E.stream));
        const int64_t chunks = (edges + 31) / 32;
        const int grid = (int)std::max<int64_t>(
            1, std::min<int64_t>((chunks + 7) / 8, (int64_t)E.num_sms * push_per_sm));
        PM_LAUNCH(k_bf_multi_push, grid, 256, 0, E.stream, E.g.out.off, E.g.out.idx, w_out, queue, qoff, (int)q,
                  edges, dist, act, nxt);
      }
    }
    E.prof.end(E.stream);
    s.rounds++;
    s.dense_rounds += dense;
    std::swap(act, nxt);
  }
  PM_CUDA(cudaMemsetAsync(E.d_cnt + 2, 0, sizeof(Counters), E.stream));
  dim3 tb(32, 8), tg((unsigned)std::min<int64_t>((n + 31) / 32, (int64_t)E.num_sms * 16), 2);
  PM_LAUNCH(k_bf_multi_transpose, tg, tb, 0, E.stream, dist, n, k, d_dist_out, E.d_cnt + 2);
  s.reached = (int64_t)E.read_counters()[2].size;
  if (st) *st = s;
}

}  // namespace pm
