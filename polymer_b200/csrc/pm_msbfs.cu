// pm_msbfs.cu -- multi-source BFS, up to 64 sources (BFS_F of
// numa-BFS.C:59-79 with the parent test replaced by per-source visited bits),
// every level in one cooperative launch.
//
// Level t's word of a vertex holds the sources that reach it at exactly that
// level; visited[v] the sources that reached v so far; depth[l * n + v] is v's
// level from source l.  The levels' words stay in a ring of kSlots-or-fewer
// slots, and the depths are written from them in one coalesced pass.
// Sparse levels push: every frontier vertex ORs the bits its out-neighbours
// lack into their next words, from queues cut to bounded pieces
// (pm_rounds.cuh).  Dense levels pull: a vertex that lacks sources ORs its
// in-neighbours' words until nothing it lacks is left to find -- hubs come
// first in most rows, so from the second dense level on a few in-edges settle
// a vertex.  The long rows are taken in order of degree (pm_sorted.cuh's
// order), each kind by as many lanes as suit it, so no warp is left with a long
// row; the short ones in vertex order, a thread each.
// Either way a level only adds bits that visited lacks.  visited takes a dense
// level's bits when the next level looks at the vertex, so no pass over the
// vertices follows a level.
//
// What bounds it: the first dense level, which has to look at most edges (an
// 8-byte gather each), and the k x n depths (1 GB for 64 sources at 2^22
// vertices).  64 sources, symmetrised 2^22-vertex, 128 M-edge R-MAT: 2.80 to
// 3.23 ms as host-driven rounds of whole-row pulls -> 1.9 to 2.1 ms (the first
// dense level 0.6 ms, 214 G gathers/s; the depths 0.2 ms).  Two CTAs per SM:
// three (40 registers, with spills) take 2 % less there, but 0.85 instead of 0.80 ms
// on a directed 2^21-vertex graph and 0.36 instead of 0.30 on 0.3 M vertices,
// where the barriers count.
#include "pm_rounds.cuh"
#include "pm_sorted.cuh"

namespace pm {

using u64 = unsigned long long;

constexpr int kSlots = 16;        // level words kept before their depths are written

struct MsbfsWork {
  u64 *ring;       // slots x n: level t in slot t % slots
  int slots;
  u64 *visited;
  int32_t *touched;  // vertices a sparse level reached, each once
  RoundQueue q[2];
  RoundCount *count;   // three slots, level % 3, and the call's sums
  unsigned *ntouched;  // three slots, level % 3
  const int32_t *order;  // rows by in-degree, longest first
  const int2 *long_pieces;  // {vertex, first in-edge of the piece} of the rows [0, rc)
  int32_t np, rc, rh, rm;
  EdgePos short_rows;    // rows below this length are taken in vertex order
  const int32_t *sources;
  int k;
  int32_t *depth;
  RoundsEnd *end;
};

// OR over the lanes of `width` consecutive lanes.
template <int WIDTH>
__device__ __forceinline__ u64 lanes_or(u64 x) {
#pragma unroll
  for (int d = WIDTH / 2; d > 0; d >>= 1)
    x |= (u64)__shfl_xor_sync(0xffffffffu, (unsigned)x, d) |
         ((u64)__shfl_xor_sync(0xffffffffu, (unsigned)(x >> 32), d) << 32);
  return x;
}

// The bits of `need` found among the words of in-edges e, e + WIDTH, ... of
// WIDTH lanes' common row; all lanes of the warp call it (rows may differ by
// group), lanes whose row is done wait.
template <int WIDTH>
__device__ __forceinline__ u64 msbfs_scan(const GraphView &g, const u64 *front, u64 need, EdgePos e, EdgePos e1) {
  u64 got = 0;
  bool open = need != 0 && e1 > 0;
  while (__any_sync(0xffffffffu, open)) {
    u64 x = 0;
    if (open) {
      int s[kStep];
#pragma unroll
      for (int u = 0; u < kStep; ++u) s[u] = e + u * WIDTH < e1 ? checked_id(g, __ldg(g.in.idx + e + u * WIDTH)) : -1;
#pragma unroll
      for (int u = 0; u < kStep; ++u)
        if (s[u] >= 0) x |= front[s[u]];
      e += kStep * WIDTH;
    }
    got |= lanes_or<WIDTH>(x) & need;
    open = open && got != need && e - (lane_id() % WIDTH) < e1;
  }
  return got;
}

// Sums a thread keeps: the level's |F| and out-degrees, and over the whole call
// the (source, vertex) pairs reached and their out-degrees.
struct MsbfsSums {
  u64 size = 0, edges = 0, reached = 0, outdeg = 0;
  // v got `bits`; first: its first of this level
  __device__ __forceinline__ void add(const GraphView &g, int v, u64 bits, bool first) {
    const unsigned deg = (unsigned)(__ldg(g.out.off + v + 1) - __ldg(g.out.off + v));
    const unsigned c = (unsigned)__popcll(bits);
    size += first;
    edges += first ? deg : 0u;
    reached += c;
    outdeg += (u64)c * deg;
  }
};

// One dense level.  pending: visited lacks the bits of front (a dense level
// went before).
__device__ __forceinline__ void msbfs_pull(const GraphView &g, const MsbfsWork &w, const u64 *front, u64 *next,
                                           u64 full, bool pending, MsbfsSums &sum) {
  const int lane = lane_id();
  // rows of the longest kind: a CTA per piece, ORed into the (zeroed) word.
  // Every piece may store visited: they store the same bits.
  for (int p = blockIdx.x; p < w.np; p += gridDim.x) {
    const int2 pc = __ldg(w.long_pieces + p);
    u64 vis = w.visited[pc.x];
    if (pending) {
      const u64 f = front[pc.x];
      vis |= f;
      if (threadIdx.x == 0 && f) w.visited[pc.x] = vis;
    }
    const u64 need = full & ~vis;
    if (need == 0) continue;
    const EdgePos e1 = edge_end((EdgePos)pc.y, kOrderPiece, (EdgePos)__ldg(g.in.off + pc.x + 1));
    u64 x = 0;
    for (EdgePos e = (EdgePos)pc.y + threadIdx.x; e < e1; e += kStep * kRoundThreads) {
      int s[kStep];
#pragma unroll
      for (int u = 0; u < kStep; ++u)
        s[u] = e + u * kRoundThreads < e1 ? checked_id(g, __ldg(g.in.idx + e + u * kRoundThreads)) : -1;
#pragma unroll
      for (int u = 0; u < kStep; ++u)
        if (s[u] >= 0) x |= front[s[u]];
    }
    x = lanes_or<32>(x) & need;
    if (lane == 0 && x) {
      const u64 old = atomicOr(next + pc.x, x);
      if (x & ~old) sum.add(g, pc.x, x & ~old, old == 0);
    }
  }
  // then a warp per row, kSubLanes lanes per row
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (int64_t)gridDim.x * blockDim.x;
  const int64_t n1 = w.rh - w.rc, n2 = ((int64_t)(w.rm - w.rh) * kSubLanes + 31) / 32;
  for (int64_t t = gtid >> 5; t < n1 + n2; t += gsize >> 5) {
    const bool whole = t < n1;  // the same for the whole warp
    const int r = whole ? w.rc + (int)t : w.rh + (int)((t - n1) * (32 / kSubLanes)) + lane / kSubLanes;
    const int sub = whole ? lane : lane % kSubLanes;
    int v = 0;
    EdgePos o = 0, o1 = 0;
    u64 need = 0;
    if (r < (whole ? w.rh : w.rm)) {
      v = w.order[r];
      u64 vis = w.visited[v];
      if (pending) {
        const u64 f = front[v];
        vis |= f;
        if (sub == 0 && f) w.visited[v] = vis;
      }
      need = full & ~vis;
      if (need) {
        o = __ldg(g.in.off + v);
        o1 = __ldg(g.in.off + v + 1);
      }
    }
    const u64 got = whole ? msbfs_scan<32>(g, front, need, o + sub, o1)
                          : msbfs_scan<kSubLanes>(g, front, need, o + sub, o1);
    if (sub == 0 && got) {
      next[v] = got;
      sum.add(g, v, got, true);
    }
  }
  // the short rows in vertex order, a thread each (their words and offsets are
  // read and written in whole lines; in order of degree, four lanes a row,
  // they took three quarters of a level)
  for (int64_t v0 = gtid; v0 < g.n; v0 += kStep * gsize) {
    u64 need[kStep], got[kStep];
    EdgePos o[kStep], o1[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const int64_t v = v0 + u * gsize;
      need[u] = got[u] = 0;
      o[u] = o1[u] = 0;
      if (v < g.n) {
        o[u] = __ldg(g.in.off + v);
        o1[u] = __ldg(g.in.off + v + 1);
        need[u] = w.visited[v];
        if (pending) got[u] = front[v];
      }
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      const int64_t v = v0 + u * gsize;
      const bool mine = o1[u] > o[u] && o1[u] - o[u] < w.short_rows;
      const u64 vis = need[u] | got[u];
      if (got[u] && mine) w.visited[v] = vis;
      need[u] = mine ? full & ~vis : 0ull;
      got[u] = 0;
      while (got[u] != need[u] && o[u] < o1[u]) {
        int s[kStep];
        u64 x = 0;
#pragma unroll
        for (int k = 0; k < kStep; ++k) s[k] = o[u] + k < o1[u] ? checked_id(g, __ldg(g.in.idx + o[u] + k)) : -1;
#pragma unroll
        for (int k = 0; k < kStep; ++k)
          if (s[k] >= 0) x |= front[s[k]];
        got[u] |= x & need[u];
        o[u] += kStep;
      }
      if (got[u]) {
        next[v] = got[u];
        sum.add(g, (int)v, got[u], true);
      }
    }
  }
}

// Bit i of a byte at bit 4 i.
__device__ __forceinline__ unsigned spread_nibbles(unsigned x) {
  x = (x | x << 12) & 0x000f000fu;
  x = (x | x << 6) & 0x03030303u;
  return (x | x << 3) & 0x11111111u;
}

// Writes the depths of levels [l0, l0 + cnt): cnt < kSlots, so a lane's level
// among them is four bits, kept as four planes of 64 lanes; fifteen stands for
// none.  Eight lanes at a time their planes become nibbles (a shift of each
// 64-bit plane per lane took 350 us of a 1.9 ms call, this about 200).
// first: all k rows are written (-1 where no level has the lane), else only
// the lanes found.
static_assert(kSlots <= 16, "fifteen levels and the mark for none in four bits");
__device__ __forceinline__ void msbfs_depths(const MsbfsWork &w, int64_t n, int32_t l0, int cnt, bool first) {
  const int64_t gsize = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gsize) {
    u64 p0 = 0, p1 = 0, p2 = 0, p3 = 0, found = 0;
#pragma unroll 4
    for (int j = 0; j < cnt; ++j) {
      const u64 x = w.ring[(int64_t)((l0 + j) % w.slots) * n + v];
      found |= x;
      if (j & 1) p0 |= x;
      if (j & 2) p1 |= x;
      if (j & 4) p2 |= x;
      if (j & 8) p3 |= x;
    }
    if (!first && found == 0) continue;
    p0 |= ~found;
    p1 |= ~found;
    p2 |= ~found;
    p3 |= ~found;
    int32_t *out = w.depth + v;
    for (int l = 0; l < w.k; l += 8) {
      const unsigned q = spread_nibbles((unsigned)(p0 >> l) & 255u) | spread_nibbles((unsigned)(p1 >> l) & 255u) << 1 |
                         spread_nibbles((unsigned)(p2 >> l) & 255u) << 2 | spread_nibbles((unsigned)(p3 >> l) & 255u) << 3;
#pragma unroll
      for (int i = 0; i < 8; ++i, out += n) {
        const int t = (int)(q >> (4 * i)) & 15;
        if (l + i < w.k && (first || t != 15)) *out = t == 15 ? -1 : l0 + t;
      }
    }
  }
}

__global__ void __launch_bounds__(kRoundThreads, 2) k_msbfs(GraphView g, MsbfsWork w, RoundsEnd from,
                                                            int64_t threshold) {
  cg::grid_group grid = cg::this_grid();
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (int64_t)gridDim.x * blockDim.x;
  const int64_t n = g.n;
  const u64 full = w.k == 64 ? ~0ull : (1ull << w.k) - 1ull;
  auto slot = [&](int32_t t) { return w.ring + (int64_t)(t % w.slots) * n; };
  const bool fresh = from.level == 1;
  if (fresh) {
    for (int64_t v = gtid; v < n; v += gsize) slot(0)[v] = slot(1)[v] = w.visited[v] = 0ull;
    if (gtid < 3) w.ntouched[gtid] = 0;
    if (gtid < 4) w.count[gtid] = RoundCount{};
    grid.sync();
  }
  MsbfsSums sum;
  if (fresh && blockIdx.x == 0 && threadIdx.x < 32) {  // the sources: a vertex may hold several
    bool act[kStep] = {};
    int d[kStep] = {}, deg[kStep] = {};
    u64 size = 0, edges = 0;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int l = threadIdx.x + 32 * u;
      if (l < w.k) {
        d[u] = w.sources[l];
        atomicOr(w.visited + d[u], 1ull << l);
        act[u] = atomicOr(slot(0) + d[u], 1ull << l) == 0ull;
        const int od = __ldg(g.out.off + d[u] + 1) - __ldg(g.out.off + d[u]);
        if (act[u]) deg[u] = od;
        size += act[u];
        edges += (unsigned)deg[u];
        sum.reached += 1;
        sum.outdeg += (unsigned)od;
      }
    }
    round_append(act, d, deg, w.q[0], w.count);
    size = warp_sum(size);
    edges = warp_sum(edges);
    if (threadIdx.x == 0) {
      w.count->size = size;
      w.count->edges = edges;
    }
  }
  grid.sync();
  PM_ROUND_STATS(st, gtid, from);
  bool have_queue = !from.have_bits;  // and visited holds every bit so far
  bool more = false;
  int32_t flushed = from.flushed;  // levels below this have their depths written
  int32_t level = from.level;
  for (;; ++level) {
    RoundCount *cur = w.count + (level - 1) % 3, *nxt = w.count + level % 3;
    RoundCount f = round_read(cur);
    more = f.size != 0 && level - from.level == kRoundsPerLaunch;
    if (f.size == 0 || more) break;
    const bool dense = (long long)(f.size + f.edges) >= threshold;
    const RoundQueue &q = w.q[(level - 1) & 1], &qn = w.q[level & 1];
    const u64 *front = slot(level - 1);
    u64 *next = slot(level);
    if (gtid == 0) {
      st.rounds++;
      st.dense_rounds += dense;
      w.count[(level + 1) % 3] = RoundCount{};
      w.ntouched[(level + 1) % 3] = 0;
    }
    if (level + 1 - flushed == w.slots) {  // the next level's slot still holds unwritten words
      msbfs_depths(w, n, flushed, level - flushed, flushed == 0);
      flushed = level;
    }
    sum.size = sum.edges = 0;
    u64 *zero = slot(level + 1);
    for (int64_t v = gtid; v < n; v += gsize) zero[v] = 0ull;
    if (dense) {
      msbfs_pull(g, w, front, next, full, !have_queue, sum);
    } else {
      if (!have_queue) {  // after a dense level: the vertices with a word
        for (int64_t base = (int64_t)blockIdx.x * kRoundThreads * kStep; base < n;
             base += (int64_t)gridDim.x * kRoundThreads * kStep) {
          bool act[kStep];
          int v[kStep], deg[kStep];
#pragma unroll
          for (int u = 0; u < kStep; ++u) {
            const int64_t x = base + u * kRoundThreads + threadIdx.x;
            v[u] = (int)min(x, n - 1);
            const u64 f = x < n ? front[v[u]] : 0ull;
            act[u] = f != 0ull;
            if (act[u]) w.visited[v[u]] |= f;
          }
#pragma unroll
          for (int u = 0; u < kStep; ++u)
            deg[u] = act[u] ? __ldg(g.out.off + v[u] + 1) - __ldg(g.out.off + v[u]) : 0;
          round_append_block(act, v, deg, q, cur);
        }
        grid.sync();
        f = round_read(cur);
      }
      unsigned *nt = w.ntouched + level % 3;
      round_push(
          g, q, f.rows, f.pieces, [&](int s) { return s; },
          [&](const int (&s)[kStep], const EdgePos (&)[kStep], const int (&d)[kStep], const bool (&ok)[kStep]) {
            bool act[kStep];
            int deg[kStep];
            u64 x[kStep];
#pragma unroll
            for (int u = 0; u < kStep; ++u) x[u] = ok[u] ? front[s[u]] & ~w.visited[d[u]] : 0ull;
#pragma unroll
            for (int u = 0; u < kStep; ++u) {
              // bits already there need no atomic (next only gains bits)
              const u64 seen = x[u] ? *((volatile u64 *)next + d[u]) : 0ull;
              act[u] = (x[u] & ~seen) != 0ull && atomicOr(next + d[u], x[u]) == 0ull;
            }
#pragma unroll
            for (int u = 0; u < kStep; ++u) {
              deg[u] = act[u] ? __ldg(g.out.off + d[u] + 1) - __ldg(g.out.off + d[u]) : 0;
              sum.size += act[u];
              sum.edges += (unsigned)deg[u];
            }
            int total;
            const int pos = warp_excl_scan(act[0] + act[1] + act[2] + act[3], &total);
            if (total) {
              unsigned at = 0;
              if (lane_id() == 0) at = atomicAdd(nt, (unsigned)total);
              at = __shfl_sync(0xffffffffu, at, 0) + pos;
#pragma unroll
              for (int u = 0; u < kStep; ++u)
                if (act[u]) w.touched[at++] = d[u];
              round_append(act, d, deg, qn, nxt);
            }
          });
      grid.sync();
      const unsigned touched = *(volatile unsigned *)nt;
      for (unsigned i = (unsigned)gtid; i < touched; i += (unsigned)gsize) {
        const int v = w.touched[i];
        const u64 bits = next[v];
        w.visited[v] |= bits;
        const unsigned deg = (unsigned)(__ldg(g.out.off + v + 1) - __ldg(g.out.off + v)), c = (unsigned)__popcll(bits);
        sum.reached += c;
        sum.outdeg += (u64)c * deg;
      }
    }
    have_queue = !dense;
    round_count_add(sum.size, sum.edges, nxt);
    grid.sync();
  }
  // the last levels' depths (level - 1 held the last words)
  if (!more) msbfs_depths(w, n, flushed, level - flushed, flushed == 0);
  RoundCount *total = w.count + 3;
  round_count_add(sum.reached, sum.outdeg, total);
  grid.sync();
  if (gtid == 0) {
    st.reached = (int64_t)((volatile RoundCount *)total)->size;
    st.edges_visited = (int64_t)((volatile RoundCount *)total)->edges;
    *w.end = RoundsEnd{st, level, more, !have_queue, flushed};
  }
}

void run_msbfs(pm_graph *g, const int32_t *d_sources, int k, int32_t *d_depth, int64_t threshold,
               pm_traversal_stats *st) {
  Engine &E = g->E;
  const int64_t n = g->n;
  MsbfsWork w{};
  // About 1 GiB of ring at most, 3 slots at least (the front, the level being
  // built, and the next one, cleared ahead): what a call with little memory
  // left falls back to.
  const int least = 3;
  w.slots = (int)std::max<int64_t>(least, std::min<int64_t>(kSlots, (int64_t(1) << 30) / (8 * n)));
  const size_t pieces = round_pieces(g->m);
  int2 *pc = nullptr;
  const RowOrder *order = nullptr;
  for (;;) {
    try {
      w.ring = (u64 *)g->scratch_buf(0, (size_t)n * 8 * w.slots);
      w.visited = (u64 *)g->scratch_buf(2, (size_t)n * 8);
      pc = (int2 *)g->scratch_buf(1, 2 * pieces * sizeof(int2));
      w.count = (RoundCount *)g->scratch_buf(30, 4 * sizeof(RoundCount) + 16);
      order = find_row_order(g, false);
      if (order || w.slots == least) break;
    } catch (const Failure &f) {
      if (f.status != PM_ERR_OOM || w.slots == least) throw;
    }
    g->scratch[0].reset();
    w.slots = least;
  }
  for (int i = 0; i < 2; ++i) {
    w.q[i].rows = g->subset(i).queue;
    w.q[i].pieces = pc + i * pieces;
  }
  w.touched = E.defer;
  w.ntouched = (unsigned *)(w.count + 4);
  w.np = w.rc = w.rh = w.rm = 0;
  w.short_rows = ~0u;  // without memory for the order: every row
  if (order) {
    w.order = order->order.as<int32_t>();
    w.long_pieces = order->pieces.as<int2>();
    w.np = order->npieces;
    w.rc = order->cuts[0];
    w.rh = order->cuts[1];
    w.rm = order->cuts[2];
    w.short_rows = kSortShort;
  }
  w.sources = d_sources;
  w.k = k;
  w.depth = d_depth;
  w.end = (RoundsEnd *)E.h_cnt;
  static const int per_sm = round_occupancy(k_msbfs);
  E.prof.begin("bfs_multi", E.stream);
  const pm_traversal_stats s = run_rounds(E, [&](const RoundsEnd &from) {
    PM_LAUNCH_COOP(k_msbfs, round_grid(E, per_sm), kRoundThreads, E.stream, E.g, w, from, threshold);
    E.prof.end(E.stream);
  });
  E.prof.set_passes((int)s.rounds);
  if (st) *st = s;
}

}  // namespace pm
