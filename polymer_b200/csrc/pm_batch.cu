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
//  * dense: a warp owns a CSC row, thread t owns lanes t and t+32; for each
//    in-edge whose source has active lanes it gathers the source's row and
//    relaxes those lanes; the row's new active word is written in full;
//  * sparse: the frontier's out-edges are cut into 32-edge chunks (a scan of
//    the queued out-degrees); for each edge the warp relaxes the active lanes
//    of the target with atomicMin and ORs the lanes that fell into the
//    target's next active word.
// Distances only fall, so reading a row another warp is lowering in the same
// round is harmless: the lower value is a real path length and the lane that
// fell is in the next frontier either way.
// ===========================================================================
constexpr int kLanes = 64;
constexpr int kBfUnroll = 4;      // pull: in-edges whose row gathers are in flight together per half-warp
// Resident CTAs per SM of the pull: 50 sources on a 1.5 M-vertex, 42 M-edge
// R-MAT take 8.37 ms with four (58 registers), 7.11 with five, 6.64 with six
// (40 registers) and 6.75 with eight; a warp per row in vertex order, two
// 128-byte loads a row, took 8.87 to 9.16.
constexpr int kBfCtas = 6;
constexpr int kBfPushUnroll = 2;  // push: out-edges whose target rows are read together per warp

// active -> queue of frontier vertices with out-edges (and their degrees);
// c->size = |F|, c->edges = outdeg(F), c->aux = queue length.
__global__ void k_bf_multi_frontier(const u64 *__restrict__ active, const int32_t *__restrict__ out_off,
                                    int64_t n, int32_t *__restrict__ queue, int32_t *__restrict__ qdeg,
                                    Counters *c) {
  const int lane = lane_id();
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  unsigned long long size = 0, edges = 0;
  for (int64_t base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; base < n;
       base += warps * 32) {
    const int64_t v = base + lane;
    int deg = 0;
    bool act = false;
    if (v < n) {
      act = active[v] != 0ull;
      if (act) deg = __ldg(out_off + v + 1) - __ldg(out_off + v);
    }
    size += act;
    edges += (unsigned)deg;
    const unsigned push = __ballot_sync(0xffffffffu, deg > 0);
    if (push) {
      unsigned long long pos = 0;
      if (lane == 0) pos = atomicAdd(&c->aux, (unsigned long long)__popc(push));
      pos = shfl_idx(pos, 0) + __popc(push & ((1u << lane) - 1u));
      if (deg > 0) {
        queue[pos] = (int32_t)v;
        qdeg[pos] = deg;
      }
    }
  }
  size = warp_sum(size);
  edges = warp_sum(edges);
  if (lane == 0 && size) {
    atomicAdd(&c->size, size);
    atomicAdd(&c->edges, edges);
  }
}

__global__ void __launch_bounds__(256) k_bf_multi_push(const int32_t *__restrict__ out_off,
                                                       const int32_t *__restrict__ out_idx,
                                                       const int32_t *__restrict__ w_out,
                                                       const int32_t *__restrict__ queue,
                                                       const int32_t *__restrict__ qoff, int q, int64_t total,
                                                       int32_t *dist, const u64 *__restrict__ active,
                                                       u64 *next_active) {
  const int lane = lane_id();
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
    const int cnt = (int)min((int64_t)32, total - t0);
    int cur = -1;
    u64 a = 0;
    int32_t slo = 0, shi = 0;
    for (int j0 = 0; j0 < cnt; j0 += kBfPushUnroll) {
      // kBfPushUnroll edges at a time: the targets' rows are read, and their
      // atomics issued, before any result is waited for.
      int dj[kBfPushUnroll];
      int32_t nlo[kBfPushUnroll], nhi[kBfPushUnroll], olo[kBfPushUnroll], ohi[kBfPushUnroll];
#pragma unroll
      for (int u = 0; u < kBfPushUnroll; ++u) {
        const int j = min(j0 + u, cnt - 1);
        const bool take = j0 + u < cnt;
        const int sj = __shfl_sync(0xffffffffu, s, j);
        dj[u] = __shfl_sync(0xffffffffu, d, j);
        const int32_t wj = __shfl_sync(0xffffffffu, w, j);
        if (sj != cur) {
          cur = sj;
          a = __ldg(active + sj);
          slo = dist[(int64_t)sj * kLanes + lane];
          shi = dist[(int64_t)sj * kLanes + 32 + lane];
        }
        nlo[u] = take && ((a >> lane) & 1ull) ? slo + wj : kDevBFInf;
        nhi[u] = take && ((a >> (32 + lane)) & 1ull) ? shi + wj : kDevBFInf;
        olo[u] = nlo[u] < kDevBFInf ? *(volatile int32_t *)(dist + (int64_t)dj[u] * kLanes + lane) : 0;
        ohi[u] = nhi[u] < kDevBFInf ? *(volatile int32_t *)(dist + (int64_t)dj[u] * kLanes + 32 + lane) : 0;
      }
      // A lane below the distance read above lowers it with an atomic
      // whose result is unused and is marked active: it fell, or another
      // push lowered it further meanwhile (an extra relaxation next round,
      // the same distances).
#pragma unroll
      for (int u = 0; u < kBfPushUnroll; ++u) {
        if (nlo[u] < olo[u]) atomicMin(dist + (int64_t)dj[u] * kLanes + lane, nlo[u]);
        if (nhi[u] < ohi[u]) atomicMin(dist + (int64_t)dj[u] * kLanes + 32 + lane, nhi[u]);
      }
#pragma unroll
      for (int u = 0; u < kBfPushUnroll; ++u) {
        const u64 mask = (u64)__ballot_sync(0xffffffffu, nlo[u] < olo[u]) |
                         ((u64)__ballot_sync(0xffffffffu, nhi[u] < ohi[u]) << 32);
        if (lane == 0 && mask) atomicOr(next_active + dj[u], mask);
      }
    }
  }
}

// The least dist[s] + w over this half-warp's in-edges whose sources have
// active lanes: 16 edges from e on, then from e + step on, ... below e1.  Half
// a warp holds a source's row (int4: lanes 4 t .. 4 t + 3 of the 64 on its
// thread t), so one load brings a row to each half and a step has kBfUnroll
// rows per half in flight.  All lanes of the warp call it; the halves may have
// different rows and lengths.
__device__ __forceinline__ int4 bf_multi_relax(const int32_t *__restrict__ in_idx, const int32_t *__restrict__ w_in,
                                               const int32_t *dist, const u64 *__restrict__ active, int e, int e1,
                                               int step) {
  const int t = lane_id() & 15, quad = t * 4, shift = lane_id() & 16;
  int4 m = make_int4(kDevBFInf, kDevBFInf, kDevBFInf, kDevBFInf);
  for (; __any_sync(0xffffffffu, e < e1); e += step) {
    int s = 0;
    u64 act = 0;
    int32_t w = 0;
    if (e + t < e1) {
      s = __ldcs(in_idx + e + t);
      act = __ldg(active + s);
      w = __ldcs(w_in + e + t);
    }
    unsigned todo = (__ballot_sync(0xffffffffu, act != 0) >> shift) & 0xffffu;
    while (__any_sync(0xffffffffu, todo != 0u)) {
      int4 v[kBfUnroll];
      unsigned on[kBfUnroll];
      int32_t wj[kBfUnroll];
#pragma unroll
      for (int u = 0; u < kBfUnroll; ++u) {
        const int j = todo ? __ffs(todo) - 1 : 0;
        const bool take = todo != 0u;
        todo &= todo - 1u;
        const int sj = __shfl_sync(0xffffffffu, s, j, 16);
        const unsigned lo = __shfl_sync(0xffffffffu, (unsigned)act, j, 16),
                       hi = __shfl_sync(0xffffffffu, (unsigned)(act >> 32), j, 16);
        wj[u] = __shfl_sync(0xffffffffu, w, j, 16);
        on[u] = take ? ((quad < 32 ? lo >> quad : hi >> (quad - 32)) & 15u) : 0u;
        v[u] = make_int4(0, 0, 0, 0);
        if (on[u]) v[u] = *reinterpret_cast<const int4 *>(dist + (int64_t)sj * kLanes + quad);
      }
#pragma unroll
      for (int u = 0; u < kBfUnroll; ++u) {
        if (on[u] & 1u) m.x = min(m.x, v[u].x + wj[u]);
        if (on[u] & 2u) m.y = min(m.y, v[u].y + wj[u]);
        if (on[u] & 4u) m.z = min(m.z, v[u].z + wj[u]);
        if (on[u] & 8u) m.w = min(m.w, v[u].w + wj[u]);
      }
    }
  }
  return m;
}
// Both halves' minima of one row, on both.
__device__ __forceinline__ int4 bf_multi_join(int4 m) {
  m.x = min(m.x, __shfl_xor_sync(0xffffffffu, m.x, 16));
  m.y = min(m.y, __shfl_xor_sync(0xffffffffu, m.y, 16));
  m.z = min(m.z, __shfl_xor_sync(0xffffffffu, m.z, 16));
  m.w = min(m.w, __shfl_xor_sync(0xffffffffu, m.w, 16));
  return m;
}

// The 64-bit mask whose bits 4 t .. 4 t + 3 are the nibble of the half's
// thread t, on every lane of that half.
__device__ __forceinline__ u64 bf_multi_mask(unsigned nibble) {
  const int t = lane_id() & 15;
  unsigned lo = t < 8 ? nibble << (4 * t) : 0u, hi = t < 8 ? 0u : nibble << (4 * (t - 8));
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) {
    lo |= __shfl_xor_sync(0xffffffffu, lo, d);
    hi |= __shfl_xor_sync(0xffffffffu, hi, d);
  }
  return (u64)lo | ((u64)hi << 32);
}

constexpr int kBfPiece = 512;  // in-edges of one warp's piece of a heavy row

// Dense round, a warp per item: 512-edge pieces of the heavy rows (in-degree >
// g.heavy_deg; they lower the row with atomicMin and OR the fallen lanes into
// next_active, which starts at zero), then the light rows in order of
// in-degree (order: pm_sorted.cu), a warp for each of [0, rh) and half a warp
// for each of [rh, rl).  A light row is relaxed in full by its lanes, which
// write its next_active word.
__global__ void __launch_bounds__(256, kBfCtas) k_bf_multi_pull(GraphView g, const int32_t *__restrict__ w_in,
                                                                int32_t *dist, const u64 *__restrict__ active,
                                                                u64 *next_active, int64_t heavy_pieces,
                                                                const int32_t *__restrict__ order, int rh, int rl) {
  const int lane = lane_id(), half = lane >> 4, t = lane & 15;
  int64_t item = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (item < heavy_pieces) {
    const int c = (int)(item / (kChunkEdges / kBfPiece));
    const int piece = (int)(item % (kChunkEdges / kBfPiece));
    const int r = __ldg(g.in.hrow + c);
    const int row_end = __ldg(g.in.off + r + 1);
    const int64_t first = (int64_t)__ldg(g.in.off + r) + (int64_t)(c - __ldg(g.in.hfirst + r)) * kChunkEdges +
                          (int64_t)piece * kBfPiece;
    if (first >= row_end) return;
    const int e0 = (int)first, e1 = min(row_end - e0, kBfPiece) + e0;
    const int4 m = bf_multi_join(bf_multi_relax(g.in.idx, w_in, dist, active, e0 + 16 * half, e1, 32));
    unsigned fell = 0;
    if (half == 0) {
      int32_t *p = dist + (int64_t)r * kLanes + 4 * t;
      const volatile int32_t *seen = p;
      if (m.x < seen[0] && m.x < atomicMin(p, m.x)) fell |= 1u;
      if (m.y < seen[1] && m.y < atomicMin(p + 1, m.y)) fell |= 2u;
      if (m.z < seen[2] && m.z < atomicMin(p + 2, m.z)) fell |= 4u;
      if (m.w < seen[3] && m.w < atomicMin(p + 3, m.w)) fell |= 8u;
    }
    const u64 mask = bf_multi_mask(fell);
    if (lane == 0 && mask) atomicOr(next_active + r, mask);
    return;
  }
  item -= heavy_pieces;
  const bool whole = item < rh;  // the same for the whole warp
  const int64_t r = whole ? item : rh + 2 * (item - rh) + half;
  int v = 0, e0 = 0, e1 = 0;
  bool mine = r < rl;
  if (mine) {
    v = __ldg(order + r);
    e0 = __ldg(g.in.off + v);
    e1 = __ldg(g.in.off + v + 1);
    mine = e1 - e0 <= g.heavy_deg;
    if (!mine) e1 = e0;
  }
  if (!__any_sync(0xffffffffu, mine)) return;
  int4 *row = reinterpret_cast<int4 *>(dist + (int64_t)v * kLanes) + t;
  const int4 old = *row;
  int4 m = bf_multi_relax(g.in.idx, w_in, dist, active, whole ? e0 + 16 * half : e0, e1, whole ? 32 : 16);
  if (whole) m = bf_multi_join(m);
  const unsigned fell = !mine ? 0u : (m.x < old.x) | (m.y < old.y) << 1 | (m.z < old.z) << 2 | (m.w < old.w) << 3;
  const bool write = !whole || half == 0;
  if (write && fell) *row = make_int4(min(m.x, old.x), min(m.y, old.y), min(m.z, old.z), min(m.w, old.w));
  const u64 mask = bf_multi_mask(fell);
  if (mine && write && t == 0 && mask) next_active[v] = mask;
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
  const RowOrder &o = ensure_row_order(g, false);
  const int rh = o.cuts[1], rl = o.cuts[3];
  const int64_t items = heavy_pieces + rh + (rl - rh + 1) / 2;
  const unsigned pull_grid = (unsigned)((items + 7) / 8);
  const int32_t *w_in = g->w_i32_in.as<int32_t>(), *w_out = g->w_i32_out.as<int32_t>();
  pm_traversal_stats s{};
  E.tag = "bellman_ford_multi";
  for (;;) {
    PM_CUDA(cudaMemsetAsync(E.d_cnt, 0, 3 * sizeof(Counters), E.stream));
    PM_LAUNCH(k_bf_multi_frontier, E.grid_for(n, 256, 8), 256, 0, E.stream, act, E.g.out.off, n, queue, qdeg,
              E.d_cnt + 1);
    const Counters *h = E.read_counters();
    const int64_t size = (int64_t)h[1].size, edges = (int64_t)h[1].edges, q = (int64_t)h[1].aux;
    if (size == 0) break;
    if (s.rounds > n + 1) fail(PM_ERR_INVALID_ARG, "BellmanFord did not converge");
    s.edges_visited += edges;
    const bool dense = size + edges >= threshold;
    E.prof.begin(E.tag, E.stream);
    PM_CUDA(cudaMemsetAsync(nxt, 0, (size_t)n * 8, E.stream));
    if (dense) {
      if (items > 0)
        PM_LAUNCH(k_bf_multi_pull, pull_grid, 256, 0, E.stream, E.g, w_in, dist, act, nxt, heavy_pieces,
                  o.order.as<int32_t>(), rh, rl);
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
