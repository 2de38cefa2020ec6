// pm_sorted.cuh -- pull sums over a degree-sorted copy of one adjacency, for
// the applications that add up a gathered value per in-edge (PageRank, SpMV,
// the weighted fixed points and their adjoints).
//
// Layout (built on a handle's first such call, kept with it).  Rows are
// sorted by degree, longest first; every vertex has a position in that order
// and the application's vectors live in position order, so that the values
// most edges gather sit together (an L1 line of hubs serves many edges).
// Four kinds of rows, each with the loads that suit it:
//   positions [0, rc)   >= kSortCta edges: a CTA per piece of `piece` edges;
//                       rows of several pieces are folded in piece order by
//                       the last piece to finish
//   positions [rc, rh)  >= kSortLong edges: a warp per row, lane-strided
//   positions [rh, rm)  >= kSortShort edges: kSubLanes lanes per row
//   positions [rm, rl)  the rest: 32 rows a slice, stored column by column
//                       (slot k of the slice's 32 rows side by side), so a
//                       lane per row reads ids in whole lines; consecutive
//                       rows have (nearly) the same degree: no padding
//   positions [rl, n)   no edges: their values are constants, set by the
//                       application outside the passes
// Every warp's work is bounded (kSortCta edges), so a graph of any size ends
// without a long warp, and an edge costs an id load, a gather and an add.
//
// What bounds it: the rate at which an SM can issue scattered gathers that
// miss its L1 (about 270 G/s on this GPU) or hit it (720 G/s).  The pull over
// the CSC in vertex order (k_pull_reduce) spends about 100 warp instructions
// per 32 edges on locating rows and folding straddling ones, and one warp on
// each batch of 32 rows, which for R-MAT's first 32 rows is 170 windows in a
// row: 60 us whatever the graph's size.  Before -> now: PageRank FP32, 20
// passes of a 2^24-vertex, 263 M-edge R-MAT 23.3 -> 16.1 ms (a pass sums at
// 330 G edges/s); SpMV, 10 passes of it 12.8 -> 9.1 ms; PageRank FP64, 10
// passes of 2^16 vertices and 1 M edges 606 -> 94 us; a weighted fixed point,
// its adjoint and one SpMV backward on 2^20 vertices and 16.8 M edges
// 20.5 -> 6.9 ms.
// The cuts (128 and 32 edges): 512 / 32 sums a 2^24-vertex R-MAT in 760 us,
// 128 / 32 in 746 us, 128 / 16 in 769 us; 8 lanes per middle row beat a warp
// (178 against 234 us) and a lane per short row beat 4 (102 against 177 us).
// A shared-memory copy of the hottest 16 K to 56 K values was not faster
// (768 to 1425 us: it takes the room from L1), nor were sources sorted within
// a row (3 %, for two more sorts of all edges at build time).
#pragma once
#include "pm_graph.cuh"

namespace pm {

constexpr int kSortCta = 1024;
constexpr int kSortLong = 128;
constexpr int kSortShort = 32;
constexpr int kSubLanes = 8;
constexpr int kSortThreads = 256;
constexpr int kAuxSlots = 1024;  // spread FP64 sums of a pass (one atomic per block)

struct SortedView {
  int32_t n = 0, rc = 0, rh = 0, rm = 0, rl = 0;
  int32_t np = 0, piece = 0;        // CTA pieces, edges of one
  const int32_t *off = nullptr;     // [0, rm]: first slot of a row; [rm + s]: first slot of slice s
  const int32_t *ids = nullptr;     // positions of the sources
  const float *w = nullptr;
  const uint8_t *deg = nullptr;     // degree of row rm + i
  const int4 *pieces = nullptr;     // {first slot, end slot, row, the row's first piece or -1 when alone}
  const int32_t *pfirst = nullptr;  // row -> its first piece (rc + 1 entries)
  const int32_t *order = nullptr;   // position -> vertex
  const int32_t *odeg = nullptr;    // out-degree by position
  void *partials = nullptr;         // np accumulators of 8 bytes
  int32_t *done = nullptr;          // finished pieces of a row (zero between passes)
  __host__ __device__ int64_t sub_warps() const { return ((int64_t)(rm - rh) * kSubLanes + 31) / 32; }
  __host__ __device__ int64_t slices() const { return ((int64_t)(rl - rm) + 31) / 32; }
  // the grid of a pass: np CTAs for pieces, then kSortThreads / 32 warps a CTA
  __host__ __device__ int64_t warps() const { return (int64_t)(rh - rc) + sub_warps() + slices(); }
  int64_t blocks() const { return np + (warps() + kSortThreads / 32 - 1) / (kSortThreads / 32); }
};

// The sum of f.edge over slots e, e + STRIDE, ... below e1: four id loads, then
// four gathers in flight, their values added in pairs (a quarter of the
// dependent additions, and of their rounding); the remainder is one predicated
// step.
template <bool W, int STRIDE, class F>
__device__ __forceinline__ typename F::Acc sorted_sum(const SortedView &a, const F &f, int e, int e1) {
  using Acc = typename F::Acc;
  constexpr int U = 4;
  Acc acc = f.identity();
  int s[U];
  float w[U];
  for (; e + (U - 1) * STRIDE < e1; e += U * STRIDE) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      s[u] = __ldcs(a.ids + e + u * STRIDE);
      if constexpr (W) w[u] = __ldcs(a.w + e + u * STRIDE);
    }
    Acc v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = f.edge(s[u], W ? w[u] : 0.0f);
    acc = f.combine(acc, f.combine(f.combine(v[0], v[1]), f.combine(v[2], v[3])));
  }
  if (e < e1) {
#pragma unroll
    for (int u = 0; u < U - 1; ++u) {
      const bool in = e + u * STRIDE < e1;
      s[u] = in ? __ldcs(a.ids + e + u * STRIDE) : -1;
      if constexpr (W) w[u] = in ? __ldcs(a.w + e + u * STRIDE) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U - 1; ++u)
      if (s[u] >= 0) acc = f.combine(acc, f.edge(s[u], W ? w[u] : 0.0f));
  }
  return acc;
}

// The warp's sum, in a fixed order, on lane 0.
template <class F>
__device__ __forceinline__ typename F::Acc sorted_warp_fold(const F &f, typename F::Acc v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v = f.combine(v, shfl_down(v, d));
  return v;
}

// Whether a functor adds FP64 values in commit() (residuals, norms).
template <class F, class = void>
struct HasAux : std::false_type {};
template <class F>
struct HasAux<F, std::enable_if_t<F::kAux>> : std::true_type {};

// One pass: f.commit(position, sum, f.pre(position), aux) for every row with edges.  stop, when
// given and set, makes the launch return at once (a fixed point that has
// converged while later passes were already queued).
template <class F, bool W>
__global__ void __launch_bounds__(kSortThreads, sizeof(typename F::Acc) == 4 ? 8 : 6)
    k_sorted_pull(SortedView a, F f, double2 *aux, const int *stop) {
  using Acc = typename F::Acc;
  if (stop && *stop) return;
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int64_t t = ((int64_t)blockIdx.x - a.np) * (kSortThreads / 32) + wid;
  double2 my_aux = make_double2(0.0, 0.0);
  const int64_t rows = a.rh - a.rc, subs = a.sub_warps();
  // f.pre(r): what commit reads of the row besides its sum
  if (t < 0) {
    __shared__ Acc s_part[kSortThreads / 32];
    const int4 pc = __ldg(a.pieces + blockIdx.x);
    const Acc w = sorted_warp_fold(f, sorted_sum<W, kSortThreads>(a, f, pc.x + threadIdx.x, pc.y));
    if (lane == 0) s_part[wid] = w;
    __syncthreads();
    if (wid == 0) {
      Acc v = sorted_warp_fold(f, lane < kSortThreads / 32 ? s_part[lane] : f.identity());
      bool mine = true;
      if (pc.w >= 0) {  // one of several pieces: the last to finish folds them
        Acc *part = reinterpret_cast<Acc *>(a.partials);
        const int count = __ldg(a.pfirst + pc.z + 1) - pc.w;
        int last = 0;
        if (lane == 0) {
          part[blockIdx.x] = v;
          __threadfence();
          last = atomicAdd(a.done + pc.z, 1) == count - 1;
        }
        mine = __shfl_sync(0xffffffffu, last, 0) != 0;
        if (mine) {
          __threadfence();  // the other pieces' partials, written before they were counted
          v = f.identity();
          for (int k = lane; k < count; k += 32) v = f.combine(v, __ldcg(part + pc.w + k));
          v = sorted_warp_fold(f, v);
          if (lane == 0) a.done[pc.z] = 0;
        }
      }
      if (mine && lane == 0) f.commit(pc.z, v, f.pre(pc.z), my_aux);
    }
  } else if (t < rows) {
    const int r = a.rc + (int)t;
    const auto pre = f.pre(r);
    const Acc v = sorted_warp_fold(f, sorted_sum<W, 32>(a, f, __ldg(a.off + r) + lane, __ldg(a.off + r + 1)));
    if (lane == 0) f.commit(r, v, pre, my_aux);
  } else if (t < rows + subs) {
    const int r = a.rh + (int)((t - rows) * (32 / kSubLanes)) + lane / kSubLanes;
    const auto pre = f.pre(min(r, a.rm - 1));
    Acc v = f.identity();
    if (r < a.rm) v = sorted_sum<W, kSubLanes>(a, f, __ldg(a.off + r) + lane % kSubLanes, __ldg(a.off + r + 1));
#pragma unroll
    for (int d = kSubLanes / 2; d > 0; d >>= 1) v = f.combine(v, shfl_down(v, d));
    if (r < a.rm && lane % kSubLanes == 0) f.commit(r, v, pre, my_aux);
  } else if (t < rows + subs + a.slices()) {
    const int64_t s = t - rows - subs;
    const int64_t r = a.rm + s * 32 + lane;
    if (r < a.rl) {
      const auto pre = f.pre((int)r);
      const int e0 = __ldg(a.off + a.rm + s) + lane;
      const Acc v = sorted_sum<W, 32>(a, f, e0, e0 + 32 * (int)__ldg(a.deg + (r - a.rm)));
      f.commit((int)r, v, pre, my_aux);
    }
  }
  if constexpr (HasAux<F>::value) {
    if (aux) {
      __shared__ double2 s_aux[kSortThreads / 32];
      my_aux.x = warp_sum(my_aux.x);
      my_aux.y = warp_sum(my_aux.y);
      if (lane == 0) s_aux[threadIdx.x >> 5] = my_aux;
      __syncthreads();
      if (threadIdx.x == 0) {
        double2 sum = s_aux[0];
        for (int i = 1; i < kSortThreads / 32; ++i) {
          sum.x += s_aux[i].x;
          sum.y += s_aux[i].y;
        }
        double2 *slot = aux + blockIdx.x % kAuxSlots;
        if (sum.x != 0.0) atomicAdd(&slot->x, sum.x);
        if (sum.y != 0.0) atomicAdd(&slot->y, sum.y);
      }
    }
  }
}

// The degree-sorted copy of g's in-adjacency (or out-adjacency when csr),
// with the float weights when weighted; built on first use.  Null when the
// handle is a partition, the edge slots would not fit int32, or there is no
// memory for the copy: the caller then takes the pull over the CSC.
const SortedView *ensure_sorted(pm_graph *g, bool csr, bool weighted, SortedView &view);

// The rows of g's in-adjacency (or out-adjacency when csr) by degree.
const RowOrder &ensure_row_order(pm_graph *g, bool csr);
// The same, or null when there is no memory for it: the caller then takes the
// rows in vertex order.
const RowOrder *find_row_order(pm_graph *g, bool csr);

// y[p] = x[order[p]]: a vector in position order.
template <class T>
__global__ void k_to_positions(const T *__restrict__ x, const int32_t *__restrict__ order, int64_t n,
                               T *__restrict__ y) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) y[p] = __ldg(x + __ldcs(order + p));
}
// y[order[p]] = x[p]: back to vertex order.
template <class T>
__global__ void k_to_vertices(const T *__restrict__ x, const int32_t *__restrict__ order, int64_t n,
                              T *__restrict__ y) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) y[__ldcs(order + p)] = __ldcs(x + p);
}
template <class T>
__global__ void k_fill_range(T *x, int64_t lo, int64_t hi, T v) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = lo + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += stride) x[i] = v;
}
template <class T>
void launch_to_positions(Engine &E, const SortedView &a, const T *x, T *y) {
  PM_LAUNCH((k_to_positions<T>), E.grid_for(a.n, 256, 16), 256, 0, E.stream, x, a.order, (int64_t)a.n, y);
}
template <class T>
void launch_to_vertices(Engine &E, const SortedView &a, const T *x, T *y) {
  PM_LAUNCH((k_to_vertices<T>), E.grid_for(a.n, 256, 16), 256, 0, E.stream, x, a.order, (int64_t)a.n, y);
}
// x[rl .. n) = v: the rows without edges.
template <class T>
void launch_fill_tail(Engine &E, const SortedView &a, T *x, T v) {
  if (a.n > a.rl)
    PM_LAUNCH((k_fill_range<T>), E.grid_for(a.n - a.rl, 256, 16), 256, 0, E.stream, x, (int64_t)a.rl, (int64_t)a.n, v);
}

template <bool W, class F>
void launch_sorted_pull(Engine &E, const SortedView &a, F f, double2 *aux = nullptr, const int *stop = nullptr) {
  static_assert(sizeof(typename F::Acc) <= 8, "accumulator larger than the partials slot");
  const int64_t blocks = a.blocks();
  if (blocks > 0) PM_LAUNCH((k_sorted_pull<F, W>), (unsigned)blocks, kSortThreads, 0, E.stream, a, f, aux, stop);
}

// Progress of a fixed-point iteration, kept on the device: the passes done,
// whether the last one met the tolerance, its relative L1 change.
struct FixState {
  int iters, stop;
  double rel;
};
// Folds a pass's spread sums (and clears them): the change sum|x' - x|, plus
// tail_first in the first pass, over the norm sum|x'| plus tail_norm (or
// *d_tail_norm) -- what the rows without edges add.
__global__ void k_fix_end(double2 *aux, double tail_first, double tail_norm, const double *d_tail_norm, double tol,
                          FixState *st);

}  // namespace pm
