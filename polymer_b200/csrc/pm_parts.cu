// pm_parts.cu -- PageRank on every part of a disjoint union (Polymer's
// semantics, PR_F / PR_Vertex_F / PR_Vertex_Reset, numa-PageRank.C:64-148, n =
// the part's own vertex count), all parts in ONE persistent launch.
// Thread-block clusters of kPartCluster CTAs take parts from a work queue,
// largest first; the CTAs of a cluster split the part's vertices and separate
// the iterations with the cluster barrier (barrier.cluster, a hardware
// barrier: no flag is polled).  The frontier rides in the contribution's sign
// as in PageRank on one graph.
//
// Layout (built on the first call after the parts were set).  The vertices of
// a part get consecutive positions, longest in-degree first, and every 32
// positions are a slice stored column by column, so that the lanes of a warp
// read their ids in whole lines and have (nearly) the same number of edges.
// What bounds it: the gathers of the part's contributions (up to 400 KB: L1
// and L2).  In vertex order a warp ran as long as its longest row -- twice the
// mean of a random graph -- and each lane read its own ids: 256 Erdos-Renyi
// parts, 5.1 M vertices, 41 M edges, 20 iterations: 4.13 ms -> 2.71 ms.
#include <algorithm>
#include <functional>
#include <queue>

#include <cooperative_groups.h>

#include <cub/cub.cuh>

#include "pm_graph.cuh"

namespace cg = cooperative_groups;

namespace pm {

constexpr int kPartCluster = 8;
constexpr int kPartThreads = 512;
// CTAs per SM of the sorted kernel: more parts at once share an SM's L1 (256
// Erdos-Renyi parts: 3.05 ms with one, 2.72 with two, 2.88 with three, 3.3
// with four).
constexpr int kPartCtas = 2;

struct PartsView {
  const int64_t *vbase, *pbase;  // first vertex / first position of a part
  const int32_t *order;          // position -> vertex, -1 where a part is padded to whole slices
  const int32_t *deg, *odeg;     // in- and out-degree by position
  const int32_t *soff;           // first slot of a slice
  const int32_t *ids;            // positions of the sources
};

#define GRID_STRIDE(i, count)                                                       \
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (count);     \
       i += (int64_t)gridDim.x * blockDim.x)

// Sort key: the part, then the in-degree descending.  Degrees from kDegTop on
// share a class (their slices are measured, not assumed), which keeps the key
// in 32 bits and the sort to three passes.
constexpr int kDegBits = 12, kDegTop = (1 << kDegBits) - 1;
__global__ void k_parts_keys(const int32_t *off, const int64_t *vbase, int count, int64_t n, uint32_t *key,
                             int32_t *val) {
  GRID_STRIDE(v, n) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (vbase[mid] <= v) lo = mid; else hi = mid - 1;
    }
    key[v] = ((uint32_t)lo << kDegBits) | (uint32_t)(kDegTop - min(off[v + 1] - off[v], kDegTop));
    val[v] = (int32_t)v;
  }
}

// Rank r of the sorted order lies in the part its key names, at the part's
// own offset: its position is pbase + (r - vbase).
__global__ void k_parts_order(const uint32_t *key, const int32_t *val, const int64_t *vbase, const int64_t *pbase,
                              int64_t n, const int32_t *in_off, const int32_t *out_off, int32_t *order, int32_t *deg,
                              int32_t *odeg, int32_t *pos) {
  GRID_STRIDE(r, n) {
    const uint32_t part = key[r] >> kDegBits;
    const int32_t v = val[r];
    const int64_t p = pbase[part] + (r - vbase[part]);
    order[p] = v;
    deg[p] = in_off[v + 1] - in_off[v];
    odeg[p] = out_off[v + 1] - out_off[v];
    pos[v] = (int32_t)p;
  }
}

// Slots of a slice: 32 times its longest row (a warp per slice); *longest: the
// longest of all (the word starts at zero).
__global__ void k_parts_slices(const int32_t *deg, int64_t slices, int64_t *len, int32_t *all) {
  GRID_STRIDE(p, 32 * (slices + 1)) {
    const int64_t s = p >> 5;
    const int longest = __reduce_max_sync(0xffffffffu, s < slices ? deg[p] : 0);
    if ((p & 31) == 0) {
      len[s] = 32 * (int64_t)longest;
      if (longest > *(volatile int32_t *)all) atomicMax(all, longest);
    }
  }
}
__global__ void k_parts_narrow(const int64_t *in, int64_t count, int32_t *out) {
  GRID_STRIDE(i, count) out[i] = (int32_t)in[i];
}

__global__ void k_parts_fill(GraphView g, PartsView a, int64_t npos, const int32_t *__restrict__ pos, int32_t *ids) {
  constexpr int U = 4;
  GRID_STRIDE(p, npos) {
    const int32_t v = a.order[p];
    if (v < 0) continue;
    const int32_t *src = g.in.idx + g.in.off[v];
    int32_t *to = ids + a.soff[p >> 5] + (p & 31);
    const int d = a.deg[p];
    for (int k = 0; k < d; k += U) {
      int x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = __ldg(src + min(k + u, d - 1));
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = __ldg(pos + x[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k + u < d) to[32 * (k + u)] = x[u];
    }
  }
}

// Parts in flight at once: clusters of the sorted and of the vertex-order kernel.
static int parts_wave(const Engine &E, bool sorted);

// The layout keeps half as many parts in flight, for L1's sake, and takes less
// time for each; which form ends a union first depends on how many parts there
// are, how large and how unlike.  The time of an iteration on a part of n
// vertices and e edges, in us: what a cluster takes whatever the part (barrier,
// launch of the loads), per edge (more when the device is full of parts), per
// vertex, and per edge of the longest row, which is one lane's.  Fitted to 124
// unions of 1 to 10000 parts of 50 to 100000 vertices (rings, Erdos-Renyi, in-
// degrees skewed mildly and strongly, sizes alike and up to a factor of 20
// apart); the form it picks is at most 9 % slower than the other one on any of
// them, and the choice is worth up to a factor of two either way (in us, vertex
// order against the layout: 73 parts of 4000 to 64000 vertices 736 / 361, 48 of
// 500 to 7000 141 / 113, 8 of 100000 1160 / 806, 5 rings of 8000 83 / 76; 2000
// of 500 1976 / 2719, 400 rings of 100 271 / 409, 133 of 860 to 1700 147 / 189).
struct PartCost {
  double part, edge, full, vertex, longest;
};
constexpr PartCost kVertexOrder{1.5, 4.2e-5, 1.1e-4, 1.6e-4, 0.042};
constexpr PartCost kByPosition{1.3, 2.3e-5, 2.3e-5, 1.6e-4, 0.032};

// The time of an iteration over all parts, sizes largest first, `wave` at once,
// each taken as the kernels take it: by the first cluster that is free.
static double parts_time(const PartCost &c, const std::vector<int64_t> &sizes, double edges_per_vertex, int longest,
                         int wave) {
  const double full = c.full * std::min(1.0, (double)sizes.size() / wave);
  std::priority_queue<double, std::vector<double>, std::greater<double>> ends;  // of each cluster's parts so far
  double rest = 0.0;  // small parts past the first few thousand level the clusters out
  for (size_t i = 0; i < sizes.size(); ++i) {
    const double n = (double)sizes[i], t = c.part + (c.edge + full) * edges_per_vertex * n + c.vertex * n + c.longest * longest;
    if ((int)ends.size() < wave) {
      ends.push(t);
    } else if (i < 4096) {
      const double first = ends.top();
      ends.pop();
      ends.push(first + t);
    } else {
      rest += t;
    }
  }
  double last = 0.0;
  for (; !ends.empty(); ends.pop()) last = ends.top();
  return last + rest / wave;
}

// Large parts without a long row always gain: from kPartEdges edges on average,
// no row above a kPartRow-th of that (100 Erdos-Renyi parts of 30000 vertices,
// 180000 edges, 1600 / 1142; with rows up to 218 2113 / 1667).
constexpr int64_t kPartEdges = 131072, kPartRow = 512;

static bool parts_layout_pays(const pm_graph *g, int longest) {
  const int64_t count = (int64_t)g->parts.size() - 1, mean = g->m / count;
  if (mean >= kPartEdges && longest <= mean / kPartRow) return true;
  std::vector<int64_t> sizes(count);
  for (int64_t p = 0; p < count; ++p) sizes[p] = g->parts[p + 1] - g->parts[p];
  std::sort(sizes.begin(), sizes.end(), std::greater<int64_t>());
  const double epv = (double)g->m / (double)g->n;
  return parts_time(kByPosition, sizes, epv, longest, parts_wave(g->E, true)) <=
         parts_time(kVertexOrder, sizes, epv, longest, parts_wave(g->E, false));
}

size_t parts_layout_bytes(const pm_graph *g) {
  const size_t count = g->parts.size(), npos = (size_t)g->n + 32 * count;
  // a row's padding is at most its own length in each of the slice's 31 others
  return 4 * ((size_t)g->m + 32 * npos) + 48 * npos + (4u << 20);
}

// Slots of the layout per edge, beside a short part's slices: a row far longer
// than the rest of its slice reads ids that share no line with another row's
// (60 stars of 50000 vertices 60 ms in vertex order, 182 in slots; parts whose
// slots come to up to seven times their edges are faster all the same while they
// are few: 5 of 8000 vertices with rows up to 3849 2977 / 2426 us).
constexpr int kPartPadding = 8;

// The layout, or false when these parts run faster in vertex order
// (k_pagerank_parts), its slots would not fit int32 or be mostly padding, or
// there is no memory for it.
static bool ensure_parts_layout(pm_graph *g) {
  PartsLayout &L = g->parts_layout;
  if (g->lean) return false;
  if (L.state != 0) return L.state > 0;
  Engine &E = g->E;
  cudaStream_t st = E.stream;
  const int64_t n = g->n, m = g->m;
  const int count = (int)g->parts.size() - 1;
  std::vector<int64_t> pbase(count + 1, 0);
  for (int p = 0; p < count; ++p) pbase[p + 1] = pbase[p] + (g->parts[p + 1] - g->parts[p] + 31) / 32 * 32;
  const int64_t npos = pbase[count], slices = npos / 32;
  // without the longest row, which is known once the rows are sorted
  if (npos >= (1ll << 31) - 64 || count > 1 << 20 || !parts_layout_pays(g, 0)) {
    L.state = -1;
    return false;
  }
  if (L.need > 0 && dev_available() < L.need) return false;  // as in ensure_sorted
  try {
    OptionalAlloc optional;
    int pbits = 1;
    while ((1ll << pbits) < count) ++pbits;  // at most 20
    DevBuf dp((size_t)(count + 1) * 8), order((size_t)npos * 4), deg((size_t)npos * 4), odeg((size_t)npos * 4),
        soff((size_t)(slices + 1) * 4), pos((size_t)n * 4);
    PM_CUDA(cudaMemcpyAsync(dp.p, pbase.data(), (count + 1) * 8, cudaMemcpyHostToDevice, st));
    PM_CUDA(cudaMemsetAsync(order.p, 0xff, (size_t)npos * 4, st));
    PM_CUDA(cudaMemsetAsync(deg.p, 0, (size_t)npos * 4, st));
    PM_CUDA(cudaMemsetAsync(odeg.p, 0, (size_t)npos * 4, st));
    {
      DevBuf k0((size_t)n * 4), k1((size_t)n * 4), v0((size_t)n * 4), v1((size_t)n * 4);
      PM_LAUNCH(k_parts_keys, E.grid_for(n, 256, 16), 256, 0, st, E.g.in.off, g->parts_vbase.as<int64_t>(), count, n,
                k0.as<uint32_t>(), v0.as<int32_t>());
      size_t tmp = 0;
      PM_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, k0.as<uint32_t>(), k1.as<uint32_t>(), v0.as<int32_t>(),
                                              v1.as<int32_t>(), (int)n, 0, kDegBits + pbits, st));
      DevBuf tb(std::max<size_t>(tmp, 16));
      PM_CUDA(cub::DeviceRadixSort::SortPairs(tb.p, tmp, k0.as<uint32_t>(), k1.as<uint32_t>(), v0.as<int32_t>(),
                                              v1.as<int32_t>(), (int)n, 0, kDegBits + pbits, st));
      PM_LAUNCH(k_parts_order, E.grid_for(n, 256, 16), 256, 0, st, k1.as<uint32_t>(), v1.as<int32_t>(),
                g->parts_vbase.as<int64_t>(), dp.as<int64_t>(), n, E.g.in.off, E.g.out.off, order.as<int32_t>(),
                deg.as<int32_t>(), odeg.as<int32_t>(), pos.as<int32_t>());
    }
    int64_t slots = 0;
    int32_t longest = 0;
    {
      DevBuf all(4);
      PM_CUDA(cudaMemsetAsync(all.p, 0, 4, st));
      DevBuf len((size_t)(slices + 1) * 8), sum((size_t)(slices + 1) * 8);
      PM_LAUNCH(k_parts_slices, E.grid_for(32 * (slices + 1), 256, 16), 256, 0, st, deg.as<int32_t>(), slices, len.as<int64_t>(),
                all.as<int32_t>());
      size_t tmp = 0;
      PM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, len.as<int64_t>(), sum.as<int64_t>(), (int)(slices + 1), st));
      DevBuf tb(std::max<size_t>(tmp, 16));
      PM_CUDA(cub::DeviceScan::ExclusiveSum(tb.p, tmp, len.as<int64_t>(), sum.as<int64_t>(), (int)(slices + 1), st));
      PM_LAUNCH(k_parts_narrow, E.grid_for(slices + 1, 256, 16), 256, 0, st, sum.as<int64_t>(), slices + 1,
                soff.as<int32_t>());
      PM_CUDA(cudaMemcpyAsync(&slots, sum.as<int64_t>() + slices, 8, cudaMemcpyDeviceToHost, st));
      PM_CUDA(cudaMemcpyAsync(&longest, all.p, 4, cudaMemcpyDeviceToHost, st));
      PM_CUDA(cudaStreamSynchronize(st));
    }
    if (slots >= (1ll << 31) - 64 || slots > kPartPadding * m + 1024ll * count || !parts_layout_pays(g, longest)) {
      L.state = -1;
      return false;
    }
    DevBuf ids((size_t)std::max<int64_t>(slots, 1) * 4);
    PartsView a{g->parts_vbase.as<int64_t>(), dp.as<int64_t>(), order.as<int32_t>(), deg.as<int32_t>(),
                odeg.as<int32_t>(), soff.as<int32_t>(), ids.as<int32_t>()};
    PM_LAUNCH(k_parts_fill, E.grid_for(npos, 256, 16), 256, 0, st, E.g, a, npos, pos.as<int32_t>(), ids.as<int32_t>());
    L.pbase = std::move(dp);
    L.order = std::move(order);
    L.deg = std::move(deg);
    L.odeg = std::move(odeg);
    L.soff = std::move(soff);
    L.ids = std::move(ids);
    L.npos = npos;
    L.need = 0;
    L.state = 1;
  } catch (const Failure &f) {
    if (f.status != PM_ERR_OOM) throw;
    L.need = parts_layout_bytes(g);
    return false;
  }
  return true;
}

// The parts over the layout.  The frontier only shrinks (see run_pagerank_sorted):
// a vertex that leaves it in pass t ends with `added` after an even number of
// later passes, with 0 after an odd one, and is written then.
__global__ void __cluster_dims__(kPartCluster, 1, 1) __launch_bounds__(kPartThreads, kPartCtas)
    k_pagerank_parts_sorted(PartsView a, const int32_t *__restrict__ queue_order, int count, int iters, float damping,
                            float *c0, float *c1, float *out, Counters *queue) {
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ int s_part;
  const int rank = (int)cluster.block_rank();
  const int64_t stride = (int64_t)kPartCluster * kPartThreads;
  for (;;) {
    if (rank == 0 && threadIdx.x == 0) s_part = (int)atomicAdd(&queue->aux, 1ull);
    cluster.sync();
    const int part = *cluster.map_shared_rank(&s_part, 0);
    cluster.sync();  // every CTA has read the ticket before the next one is drawn
    if (part >= count) break;
    const int q = __ldg(queue_order + part);
    const int64_t size = __ldg(a.vbase + q + 1) - __ldg(a.vbase + q);
    const int64_t p0 = __ldg(a.pbase + q), p1 = __ldg(a.pbase + q + 1);  // whole slices
    const float r0 = 1.0f / (float)size, added = (1.0f - damping) * r0;
    const int64_t first = p0 + (int64_t)rank * kPartThreads + threadIdx.x;
    for (int64_t p = first; p < p1; p += stride) {
      const int od = __ldg(a.odeg + p), v = __ldg(a.order + p);
      c0[p] = od > 0 ? r0 / (float)od : 0.0f;
      if (iters == 0 && v >= 0) out[v] = r0;
    }
    cluster.sync();
    float *cc = c0, *cn = c1;
    for (int it = 0; it < iters; ++it) {
      for (int64_t p = first; p < p1; p += stride) {
        const int od = __ldg(a.odeg + p);
        const int32_t *ids = a.ids + __ldg(a.soff + (p >> 5)) + (p & 31);
        const float own = cc[p];
        const int d = signbit(own) ? 0 : __ldg(a.deg + p);
        float acc = -0.0f;
        constexpr int U = 4;
        for (int k = 0; k < d; k += U) {
          int s[U];
          float x[U];
#pragma unroll
          for (int u = 0; u < U; ++u) s[u] = k + u < d ? __ldg(ids + 32 * (k + u)) : -1;
#pragma unroll
          for (int u = 0; u < U; ++u) x[u] = s[u] >= 0 ? cc[s[u]] : -0.0f;
          acc += (x[0] + x[1]) + (x[2] + x[3]);
        }
        if (signbit(own)) {  // outside the frontier
          cn[p] = -0.0f;
          continue;
        }
        const bool hit = !signbit(acc);
        const float nb = damping * (0.0f + acc) + added;
        cn[p] = hit ? (od > 0 ? nb / (float)od : 0.0f) : -0.0f;
        if (!hit || it == iters - 1) {
          const int v = __ldg(a.order + p);
          if (v >= 0) out[v] = hit ? nb : (iters - 1 - it) % 2 == 0 ? added : 0.0f;
        }
      }
      cluster.sync();
      float *t = cc;
      cc = cn;
      cn = t;
    }
  }
}

// The parts in vertex order: one thread per vertex sums its in-edges.
__global__ void __cluster_dims__(kPartCluster, 1, 1) __launch_bounds__(kPartThreads)
    k_pagerank_parts(GraphView g, const int64_t *__restrict__ vbase, const int32_t *__restrict__ order,
                     int count, int iters, float damping, float *pc, float *pn, float *c0, float *c1,
                     float *out, Counters *queue) {
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ int s_part;
  const int rank = (int)cluster.block_rank();
  const int64_t stride = (int64_t)kPartCluster * kPartThreads;
  for (;;) {
    if (rank == 0 && threadIdx.x == 0) s_part = (int)atomicAdd(&queue->aux, 1ull);
    cluster.sync();
    const int part = *cluster.map_shared_rank(&s_part, 0);
    cluster.sync();  // every CTA has read the ticket before the next one is drawn
    if (part >= count) break;
    const int p = __ldg(order + part);
    const int64_t v0 = __ldg(vbase + p), v1 = __ldg(vbase + p + 1);
    const float p0 = 1.0f / (float)(v1 - v0);
    const float added = (1.0f - damping) * p0;
    const int64_t first = v0 + (int64_t)rank * kPartThreads + threadIdx.x;
    for (int64_t v = first; v < v1; v += stride) {
      const int deg = __ldg(g.out.off + v + 1) - __ldg(g.out.off + v);
      pc[v] = p0;
      pn[v] = 0.0f;
      c0[v] = deg > 0 ? p0 / (float)deg : 0.0f;
    }
    cluster.sync();
    float *A = pc, *B = pn, *cc = c0, *cn = c1;
    for (int it = 0; it < iters; ++it) {
      for (int64_t v = first; v < v1; v += stride) {
        const EdgePos e0 = __ldg(g.in.off + v), e1 = __ldg(g.in.off + v + 1);
        float acc = -0.0f;
        EdgePos e = e0;
        for (; e + 3 < e1; e += 4) {
          const int s0 = __ldg(g.in.idx + e), s1 = __ldg(g.in.idx + e + 1);
          const int s2 = __ldg(g.in.idx + e + 2), s3 = __ldg(g.in.idx + e + 3);
          acc += (cc[s0] + cc[s1]) + (cc[s2] + cc[s3]);
        }
        for (; e < e1; ++e) acc += cc[__ldg(g.in.idx + e)];
        const bool in_f = !signbit(cc[v]);
        const bool hit = !signbit(acc);
        float nb = B[v] + acc;
        if (in_f) {
          nb = damping * nb + added;
          A[v] = 0.0f;
        }
        B[v] = nb;
        const int deg = __ldg(g.out.off + v + 1) - __ldg(g.out.off + v);
        cn[v] = hit ? (deg > 0 ? nb / (float)deg : 0.0f) : -0.0f;
      }
      cluster.sync();
      float *t = A; A = B; B = t;
      t = cc; cc = cn; cn = t;
    }
    for (int64_t v = first; v < v1; v += stride) out[v] = A[v];
    cluster.sync();
  }
}

// Thread-block clusters of a parts kernel that fit on the device at once.
static int part_clusters(const void *kernel) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kPartCluster * 64);
  cfg.blockDim = dim3(kPartThreads);
  int r = 0;
  PM_CUDA(cudaOccupancyMaxActiveClusters(&r, kernel, &cfg));
  return std::max(r, 1);
}
static int parts_wave(const Engine &E, bool sorted) {
  static const int fit_sorted = part_clusters((const void *)k_pagerank_parts_sorted);
  static const int fit_vertex = part_clusters((const void *)k_pagerank_parts);
  return sorted ? std::max(1, std::min(fit_sorted, E.num_sms * kPartCtas / kPartCluster)) : fit_vertex;
}

void run_pagerank_parts(pm_graph *g, int iters, double damping, float *d_out) {
  Engine &E = g->E;
  const int64_t n = g->n;
  const int count = (int)g->parts.size() - 1;
  // outside [0, 1] a rank may turn negative: the sign of a contribution is then
  // no longer the frontier alone, and a vertex can come back into it
  const bool sorted = damping >= 0.0 && damping <= 1.0 && ensure_parts_layout(g);
  PM_CUDA(cudaMemsetAsync(E.d_cnt, 0, sizeof(Counters), E.stream));
  if (sorted) {
    const PartsLayout &L = g->parts_layout;
    const PartsView a{g->parts_vbase.as<int64_t>(), L.pbase.as<int64_t>(), L.order.as<int32_t>(), L.deg.as<int32_t>(),
                      L.odeg.as<int32_t>(), L.soff.as<int32_t>(), L.ids.as<int32_t>()};
    float *c0 = (float *)g->scratch_buf(2, (size_t)L.npos * 4);
    float *c1 = (float *)g->scratch_buf(3, (size_t)L.npos * 4);
    E.prof.begin("pagerank_parts", E.stream);
    PM_LAUNCH(k_pagerank_parts_sorted, kPartCluster * std::min(parts_wave(E, true), count), kPartThreads, 0, E.stream, a, g->parts_order.as<int32_t>(), count, iters, (float)damping, c0, c1, d_out, E.d_cnt);
    E.prof.end(E.stream);
    return;
  }
  float *pc = (float *)g->scratch_buf(0, (size_t)n * 4);
  float *pn = (float *)g->scratch_buf(1, (size_t)n * 4);
  float *c0 = (float *)g->scratch_buf(2, (size_t)n * 4);
  float *c1 = (float *)g->scratch_buf(3, (size_t)n * 4);
  E.prof.begin("pagerank_parts", E.stream);
  PM_LAUNCH(k_pagerank_parts, kPartCluster * std::min(parts_wave(E, false), count), kPartThreads, 0, E.stream, E.g,
            g->parts_vbase.as<int64_t>(), g->parts_order.as<int32_t>(), count, iters, (float)damping, pc, pn, c0, c1,
            d_out, E.d_cnt);
  E.prof.end(E.stream);
}

}  // namespace pm
