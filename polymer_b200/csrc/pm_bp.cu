// pm_bp.cu -- belief propagation, 2 states (numa-BP.C:89-140 BP_F /
// BP_Vertex_Reset, edgeMapDenseBPNoRep 179-230, loop 280-316), on whole
// graphs.  (Partition handles run the pull of pm_apps.cu.)
//
// With one psi for every edge, the message of an edge s->d depends on d
// alone, so an iteration multiplies d's product by belief_d ^ k_d, where k_d
// counts d's in-edges whose source is in the frontier F.  F starts as every
// vertex and the next F is {d : k_d > 0}, so by induction F only shrinks:
// k_d starts at the in-degree, and a vertex that leaves F lowers its
// out-neighbours' counts once and never comes back.  One call therefore
// needs no pass over the edges per iteration: the counts follow from peeling
// the vertices without in-edges, level by level (each edge is touched at most
// once per call, from a source that left F), and once a level is empty the
// counts are final and the remaining iterations are arithmetic on each
// vertex's own two values, run in registers.
//
// What bounds it: the arithmetic (one exp, three logs per state update; the
// active vertices of a tile are compacted so that its warps run full) and one
// read of the offsets, counts and priors plus one write of the results.
// Ten iterations in FP32 on the directed R-MAT with 2^24 vertices and 263 M
// edges: 9.10 ms as ten pull passes over the CSC -> 1.03-1.16 ms here.
#include <cooperative_groups.h>

#include "pm_bp.cuh"
#include "pm_graph.cuh"

namespace cg = cooperative_groups;

namespace pm {

constexpr int kBpThreads = 256;
constexpr int kBpTile = 1024;      // vertices whose active ones are compacted together
constexpr int kBpCounts = 4;       // iterations whose counts are kept at a time
constexpr int kBpBigRow = 4096;    // out-degree from which a peeled row is shared by the grid

// Workspaces of one call.
struct BpWork {
  int32_t *k[kBpCounts];  // counts of iterations t0, t0+1, ...
  int32_t *kp;            // counts of iteration t0 - 1 (membership of F at t0)
  int32_t *queue, *big;   // peeled vertices, level after level: short rows, long rows
  unsigned *tail;         // [0] entries in queue, [1] in big
};

// v left F: its out-edges are to be peeled (one reservation per group of
// lanes that arrive together; one atomic per vertex on one word cost 1 ms).
__device__ __forceinline__ void bp_leave(const GraphView &g, const BpWork &w, int v) {
  const int deg = __ldg(g.out.off + v + 1) - __ldg(g.out.off + v);
  if (deg == 0) return;
  if (deg >= kBpBigRow) {
    w.big[atomicAdd(w.tail + 1, 1u)] = v;
    return;
  }
  const cg::coalesced_group c = cg::coalesced_threads();
  unsigned base = 0;
  if (c.thread_rank() == 0) base = atomicAdd(w.tail, c.size());
  w.queue[c.shfl(base, 0) + c.thread_rank()] = v;
}

// The queued vertices [q0, q1) and [b0, b1) have left F: their out-edges no
// longer count.  A vertex whose count reaches zero here leaves next.
__device__ __forceinline__ void bp_peel(const GraphView &g, const BpWork &w, int32_t *k, unsigned q0, unsigned q1,
                                        unsigned b0, unsigned b1) {
  const int lane = lane_id();
  const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x, gsize = gridDim.x * blockDim.x;
  for (unsigned i = b0; i < b1; ++i) {
    const int v = w.big[i];
    const int64_t e1 = __ldg(g.out.off + v + 1);
    for (int64_t e = (int64_t)__ldg(g.out.off + v) + gtid; e < e1; e += gsize) {
      const int d = checked_id(g, __ldg(g.out.idx + e));
      if (atomicSub(k + d, 1) == 1) bp_leave(g, w, d);
    }
  }
  // a warp takes 32 queued vertices (mostly short rows) and lays their edges
  // out flat over its lanes
  for (unsigned base = q0 + (gtid >> 5) * 32; base < q1; base += gsize) {
    int o = 0, deg = 0;
    if (base + lane < q1) {
      const int v = w.queue[base + lane];
      o = __ldg(g.out.off + v);
      deg = __ldg(g.out.off + v + 1) - o;
    }
    int total;
    const int pos = warp_excl_scan(deg, &total);
    for (int c = 0; c < total; c += 32) {
      const int q = c + lane;
      int j = 0;  // last vertex whose first flat edge is <= q
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, pos, j + step) <= q) j += step;
      const int e = __shfl_sync(0xffffffffu, o, j) + (q - __shfl_sync(0xffffffffu, pos, j));
      if (q < total) {
        const int d = checked_id(g, __ldg(g.out.idx + e));
        if (atomicSub(k + d, 1) == 1) bp_leave(g, w, d);
      }
      __syncwarp();
    }
  }
}

// Starts the counts of an iteration: dst (and dst2, when given) = src.  The
// arrays are 16-byte aligned and hold n rounded up to 4.
__device__ __forceinline__ void bp_copy(const int32_t *src, int32_t *dst, int32_t *dst2, int64_t n) {
  const int64_t quads = (n + 3) / 4, gsize = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < quads; i += gsize) {
    const int4 x = reinterpret_cast<const int4 *>(src)[i];
    reinterpret_cast<int4 *>(dst)[i] = x;
    if (dst2) reinterpret_cast<int4 *>(dst2)[i] = x;
  }
}

// Iterations [t0, t0 + nb) of every vertex: iteration t0 + j uses the counts
// k[min(j, last)].  A vertex outside F at t0 keeps its two values (nothing
// reaches it any more); the others run in registers.  sa / sb hold the
// products of even / odd iterations across batches (unused when the call is
// one batch); the batch that ends the call writes out.
template <class T>
__device__ __forceinline__ void bp_batch(const GraphView &g, const BpWork &w, const BpPsi<T> &psi,
                                         const typename Vec2<T>::type *__restrict__ prior, int t0, int nb, int last,
                                         bool final, typename Vec2<T>::type *sa, typename Vec2<T>::type *sb,
                                         typename Vec2<T>::type *out, int32_t *s_list, int *s_count) {
  using V = typename Vec2<T>::type;
  V *const lc0 = t0 & 1 ? sb : sa, *const ln0 = t0 & 1 ? sa : sb;            // before the batch
  V *const lc1 = (t0 + nb) & 1 ? sb : sa, *const ln1 = (t0 + nb) & 1 ? sa : sb;  // after it
  const int lane = lane_id();
  for (int64_t base = (int64_t)blockIdx.x * kBpTile; base < g.n; base += (int64_t)gridDim.x * kBpTile) {
    if (threadIdx.x == 0) *s_count = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kBpTile / kBpThreads; ++i) {
      const int64_t v = base + i * kBpThreads + threadIdx.x;
      // at t0 = 0 every vertex is in F, but one without in-edges gets nothing
      const bool act = v < g.n && (t0 == 0 ? w.k[0][v] : w.kp[v]) > 0;
      if (v < g.n && !act) {
        if (final)
          out[v] = t0 == 0 ? V{T(0), T(0)} : lc1[v];
        else if (t0 == 0)
          sa[v] = sb[v] = V{T(0), T(0)};
      }
      const unsigned bal = __ballot_sync(0xffffffffu, act);
      int pos = 0;
      if (lane == 0 && bal) pos = atomicAdd(s_count, __popc(bal));
      pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(bal & ((1u << lane) - 1u));
      if (act) s_list[pos] = (int32_t)v;
    }
    __syncthreads();
    const int count = *s_count;
    for (int i = threadIdx.x; i < count; i += kBpThreads) {
      const int v = s_list[i];
      int kk[kBpCounts];
#pragma unroll
      for (int j = 0; j < kBpCounts; ++j) kk[j] = j <= last ? w.k[j][v] : 0;
      const V pr = prior[v];
      V a = V{T(0), T(0)}, b = a;
      if (t0 > 0) {
        a = lc0[v];
        b = ln0[v];
      }
      // While k > 0 the vertex stays in F: its next product starts from 1 and
      // takes this iteration's messages.  The iteration in which k reaches
      // zero leaves 1; from then on the two values only take turns.
      int j = 0, k = kk[0];
      for (; j < last && j < nb && k > 0; ++j) {
        b = a;
        a = bp_message(psi, pr, a, k);
        k = 0;  // the next iteration's count
#pragma unroll
        for (int c = 1; c < kBpCounts; ++c)
          if (j + 1 == c) k = kk[c];
      }
      if (k > 0)
        for (; j < nb; ++j) {
          b = a;
          a = bp_message(psi, pr, a, k);
        }
      if (j < nb) {
        b = a;
        a = V{T(0), T(0)};
        if ((nb - j - 1) & 1) {
          const V t = a;
          a = b;
          b = t;
        }
      }
      if (final) {
        out[v] = a;
      } else {
        lc1[v] = a;
        ln1[v] = b;
      }
    }
    __syncthreads();  // the list is free again
  }
}

// The whole call in one cooperative launch (grid barriers between levels).
template <class T>
__global__ void __launch_bounds__(kBpThreads, sizeof(T) == 4 ? 6 : 3) k_bp(GraphView g, BpWork w, BpPsi<T> psi,
                                                   const typename Vec2<T>::type *__restrict__ prior, int iters,
                                                   typename Vec2<T>::type *sa, typename Vec2<T>::type *sb,
                                                   typename Vec2<T>::type *out) {
  __shared__ int32_t s_list[kBpTile];
  __shared__ int s_count;
  cg::grid_group grid = cg::this_grid();
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (int64_t)gridDim.x * blockDim.x;
  const volatile unsigned *tail = w.tail;
  for (int64_t v0 = gtid; v0 < g.n; v0 += 4 * gsize) {  // four vertices' offsets in flight
    int d[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t v = min(v0 + i * gsize, (int64_t)g.n - 1);
      d[i] = __ldg(g.in.off + v + 1) - __ldg(g.in.off + v);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t v = v0 + i * gsize;
      if (v >= g.n) break;
      w.k[0][v] = d[i];
      if (d[i] == 0) bp_leave(g, w, (int)v);
    }
  }
  grid.sync();
  unsigned q0 = 0, b0 = 0;  // levels below these have been peeled
  for (int t0 = 0; t0 < iters;) {
    int last = 0;
    bool settled = false;  // no vertex left F in the newest level: the counts stay
    for (;;) {
      const unsigned q1 = tail[0], b1 = tail[1];
      settled = q1 == q0 && b1 == b0;
      if (settled || last + 1 == kBpCounts || t0 + last + 1 >= iters) break;
      bp_copy(w.k[last], w.k[last + 1], nullptr, g.n);
      grid.sync();  // the copy is complete, and every thread has read the tails
      bp_peel(g, w, w.k[last + 1], q0, q1, b0, b1);
      grid.sync();
      q0 = q1;
      b0 = b1;
      ++last;
    }
    const int nb = settled ? iters - t0 : last + 1;
    bp_batch<T>(g, w, psi, prior, t0, nb, last, t0 + nb == iters, sa, sb, out, s_list, &s_count);
    t0 += nb;
    if (t0 >= iters) break;
    // the next batch starts one level further on
    const unsigned q1 = tail[0], b1 = tail[1];
    grid.sync();
    bp_copy(w.k[kBpCounts - 1], w.k[0], w.kp, g.n);
    grid.sync();
    bp_peel(g, w, w.k[0], q0, q1, b0, b1);
    grid.sync();
    q0 = q1;
    b0 = b1;
  }
}

template <class T>
void run_bp_counts(pm_graph *g, const T *d_prior, const T *psi, int iters, T *d_out) {
  using V = typename Vec2<T>::type;
  Engine &E = g->E;
  const int64_t n = g->n;
  if (iters == 0) {
    PM_CUDA(cudaMemsetAsync(d_out, 0, (size_t)n * sizeof(V), E.stream));
    return;
  }
  V *sa = (V *)g->scratch_buf(0, (size_t)n * sizeof(V));
  V *sb = (V *)g->scratch_buf(1, (size_t)n * sizeof(V));
  // the frontier queues and the deferred-row list are idle here (n + 1 ids each,
  // allocated in multiples of 512 bytes)
  BpWork w;
  const size_t n4 = (size_t)(n + 3) / 4 * 4;
  int32_t *extra = (int32_t *)g->scratch_buf(2, 3 * n4 * sizeof(int32_t));
  w.k[0] = g->subset(0).queue;
  w.k[1] = g->subset(1).queue;
  w.k[2] = extra;
  w.k[3] = extra + n4;
  w.kp = extra + 2 * n4;
  w.queue = E.defer;
  w.big = (int32_t *)g->scratch_buf(3, (size_t)(g->m / kBpBigRow + 1) * 4 + 16);
  w.tail = (unsigned *)g->scratch_buf(4, 16);
  PM_CUDA(cudaMemsetAsync(w.tail, 0, 8, E.stream));
  static const int per_sm = [] {
    int r = 0;
    PM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_bp<T>, kBpThreads, 0));
    return std::max(r, 1);
  }();
  const int grid = E.grid_for(n, kBpThreads, per_sm);
  const BpPsi<T> p{psi[0], psi[1], psi[2], psi[3]};
  const V *prior = (const V *)d_prior;
  V *out = (V *)d_out;
  E.prof.begin("bp", E.stream, iters);
  PM_LAUNCH_COOP((k_bp<T>), grid, kBpThreads, E.stream, E.g, w, p, prior, iters, sa, sb, out);
  E.prof.end(E.stream);
}

template void run_bp_counts<float>(pm_graph *, const float *, const float *, int, float *);
template void run_bp_counts<double>(pm_graph *, const double *, const double *, int, double *);

}  // namespace pm
