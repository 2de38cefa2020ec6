// pm_sorted.cu -- the degree-sorted copy of an adjacency (pm_sorted.cuh) and
// PageRank and SpMV over it.
#include <algorithm>
#include <mutex>
#include <vector>

#include <cub/cub.cuh>

#include "pm_sorted.cuh"

namespace pm {

// ---------------------------------------------------------------------------
// Building the copy.
// ---------------------------------------------------------------------------
#define GRID_STRIDE(i, count)                                                       \
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (count);     \
       i += (int64_t)gridDim.x * blockDim.x)

__global__ void k_sort_keys(const int32_t *off, int64_t n, int32_t *deg, int32_t *v) {
  GRID_STRIDE(i, n) {
    deg[i] = off[i + 1] - off[i];
    v[i] = (int32_t)i;
  }
}

// cuts[k] = number of rows with at least {kSortCta, kSortLong, kSortShort, 1} edges
// (deg is descending).
__global__ void k_sort_cuts(const int32_t *deg, int64_t n, int32_t *cuts) {
  const int least = threadIdx.x == 0 ? kSortCta : threadIdx.x == 1 ? kSortLong : threadIdx.x == 2 ? kSortShort : 1;
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (deg[mid] >= least) lo = mid + 1; else hi = mid;
  }
  cuts[threadIdx.x] = (int32_t)lo;
}

// pos = the inverse of order; odeg = out-degrees by position; len = slots of
// row r < rm, then of slice s (32 times its first, longest row); pieces of
// row r < rc.  len has rm + slices + 1 entries, pieces rc + 1.
__global__ void k_sort_tables(const int32_t *order, const int32_t *src_off, const int32_t *out_off, int64_t n,
                              int32_t rc, int32_t rm, int32_t rl, int32_t piece, int32_t *pos, int32_t *odeg,
                              int32_t *len, int32_t *pieces, uint8_t *bdeg) {
  GRID_STRIDE(p, n) {
    const int32_t v = order[p], d = src_off[v + 1] - src_off[v];
    pos[v] = (int32_t)p;
    odeg[p] = out_off[v + 1] - out_off[v];
    if (p < rm) len[p] = d;
    if (p >= rm && p < rl) {
      bdeg[p - rm] = (uint8_t)d;
      if (((p - rm) & 31) == 0) len[rm + (p - rm) / 32] = 32 * d;
    }
    if (p < rc) pieces[p] = edge_pieces(d, piece);
  }
}

__global__ void k_sort_pieces(const int32_t *pfirst, const int32_t *off, int32_t rc, int32_t piece, int4 *pieces) {
  GRID_STRIDE(r, rc) {
    const int32_t k0 = pfirst[r], k1 = pfirst[r + 1];
    EdgePos e = off[r];
    for (int32_t k = k0; k < k1; ++k, e += piece)
      pieces[k] = make_int4((int)e, (int)edge_end(e, piece, off[r + 1]), (int32_t)r, k1 - k0 > 1 ? k0 : -1);
  }
}

// Slot of the copy <- slot of the adjacency: the warps of a pass, copying.
// IDS: the sources' positions; otherwise their weights.
template <bool IDS>
__global__ void __launch_bounds__(kSortThreads) k_sort_fill(GraphView g, SortedView a, const int32_t *__restrict__ src_off,
                                                   const int32_t *__restrict__ src_idx,
                                                   const float *__restrict__ src_w, const int32_t *__restrict__ pos,
                                                   int32_t *__restrict__ ids, float *__restrict__ w) {
  const int lane = lane_id();
  const int64_t t = ((int64_t)blockIdx.x - a.np) * (kSortThreads / 32) + (threadIdx.x >> 5);
  const int64_t rows = a.rh - a.rc, subs = a.sub_warps();
  // `cnt` slots from `from` (consecutive) to `to` (to_step apart), this lane
  // taking every step-th from k on: four loads in flight
  auto copy = [&](int64_t to, int64_t from, int k, int cnt, int step, int to_step) {
    constexpr int U = 4;
    for (; k < cnt; k += U * step) {
      int x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int q = min(k + u * step, cnt - 1);
        if constexpr (IDS)
          x[u] = checked_id(g, __ldg(src_idx + from + q));
        else
          x[u] = __float_as_int(__ldg(src_w + from + q));
      }
      if constexpr (IDS) {
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = __ldg(pos + x[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k + u * step < cnt) {
          const int64_t q = to + (int64_t)(k + u * step) * to_step;
          if constexpr (IDS)
            ids[q] = x[u];
          else
            w[q] = __int_as_float(x[u]);
        }
    }
  };
  if (t < 0) {
    const int4 pc = a.pieces[blockIdx.x];
    const int from = src_off[a.order[pc.z]] + (pc.x - a.off[pc.z]);
    copy(pc.x, from, threadIdx.x, pc.y - pc.x, kSortThreads, 1);
  } else if (t < rows) {
    const int r = a.rc + (int)t;
    copy(a.off[r], src_off[a.order[r]], lane, a.off[r + 1] - a.off[r], 32, 1);
  } else if (t < rows + subs) {
    const int r = a.rh + (int)((t - rows) * (32 / kSubLanes)) + lane / kSubLanes;
    if (r < a.rm) copy(a.off[r], src_off[a.order[r]], lane % kSubLanes, a.off[r + 1] - a.off[r], kSubLanes, 1);
  } else if (t < rows + subs + a.slices()) {
    const int64_t s = t - rows - subs, r = a.rm + s * 32 + lane;
    if (r < a.rl) copy((int64_t)a.off[a.rm + s] + lane, src_off[a.order[r]], 0, a.deg[r - a.rm], 1, 32);
  }
}

// Edges of a CTA's piece.  Folding a row's pieces costs a fence and an atomic
// each, so large graphs take long pieces (20 passes of a 263 M-edge R-MAT:
// 20.7 ms with pieces of 1024, 17.7 with 2048, 16.5 with 8192, 16.1 with
// 16384); small graphs cut their hubs finer so that the pass does not end on
// one CTA (a 1 M-edge graph's passes are equal within 4 % from 1024 to 16384).
static int32_t piece_edges(int64_t m) {
  int32_t p = 2048;
  while (p < 16384 && (int64_t)p * 256 < m) p *= 2;
  return p;
}

static void exclusive_sum(const int32_t *in, int32_t *out, int64_t count, cudaStream_t st) {
  size_t tmp = 0;
  PM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, in, out, (int)count, st));
  DevBuf tb(std::max<size_t>(tmp, 16));
  PM_CUDA(cub::DeviceScan::ExclusiveSum(tb.p, tmp, in, out, (int)count, st));
}

// {vertex, first edge} of each kOrderPiece-edge piece of the rows [0, rc).
__global__ void k_order_pieces(const int32_t *order, const int32_t *src_off, const int32_t *first, int32_t rc,
                               int2 *pieces) {
  GRID_STRIDE(r, rc) {
    const int32_t v = order[r];
    EdgePos e = src_off[v];
    for (int32_t k = first[r]; k < first[r + 1]; ++k, e += kOrderPiece) pieces[k] = make_int2(v, (int)e);
  }
}
__global__ void k_order_counts(const int32_t *deg, int32_t rc, int32_t *count) {
  GRID_STRIDE(r, rc + 1) count[r] = r < rc ? edge_pieces(deg[r], kOrderPiece) : 0;
}

const RowOrder &ensure_row_order(pm_graph *g, bool csr) {
  RowOrder &o = csr ? g->order_out : g->order_in;
  if (o.order.p) return o;
  Engine &E = g->E;
  cudaStream_t st = E.stream;
  const Adj &src = csr ? E.g.out : E.g.in;
  const int64_t n = g->n;
  int bits = 1;
  while (bits < 31 && (1ll << bits) <= g->m) ++bits;
  DevBuf order((size_t)n * 4), key((size_t)n * 4), deg((size_t)n * 4), val((size_t)n * 4), cuts(16);
  PM_LAUNCH(k_sort_keys, E.grid_for(n, 256, 16), 256, 0, st, src.off, n, key.as<int32_t>(), val.as<int32_t>());
  size_t tmp = 0;
  PM_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, key.as<int32_t>(), deg.as<int32_t>(),
                                                    val.as<int32_t>(), order.as<int32_t>(), (int)n, 0, bits, st));
  DevBuf tb(std::max<size_t>(tmp, 16));
  PM_CUDA(cub::DeviceRadixSort::SortPairsDescending(tb.p, tmp, key.as<int32_t>(), deg.as<int32_t>(),
                                                    val.as<int32_t>(), order.as<int32_t>(), (int)n, 0, bits, st));
  PM_LAUNCH(k_sort_cuts, 1, 4, 0, st, deg.as<int32_t>(), n, cuts.as<int32_t>());
  int32_t h[4];
  PM_CUDA(cudaMemcpyAsync(h, cuts.p, sizeof h, cudaMemcpyDeviceToHost, st));
  PM_CUDA(cudaStreamSynchronize(st));
  const int32_t rc = h[0];
  int32_t np = 0;
  if (rc > 0) {
    DevBuf count((size_t)(rc + 1) * 4), first((size_t)(rc + 1) * 4);
    PM_LAUNCH(k_order_counts, E.grid_for(rc + 1, 256, 16), 256, 0, st, deg.as<int32_t>(), rc, count.as<int32_t>());
    exclusive_sum(count.as<int32_t>(), first.as<int32_t>(), rc + 1, st);
    PM_CUDA(cudaMemcpyAsync(&np, first.as<int32_t>() + rc, 4, cudaMemcpyDeviceToHost, st));
    PM_CUDA(cudaStreamSynchronize(st));
    o.pieces.alloc((size_t)np * sizeof(int2));
    PM_LAUNCH(k_order_pieces, E.grid_for(rc, 256, 16), 256, 0, st, order.as<int32_t>(), src.off, first.as<int32_t>(),
              rc, o.pieces.as<int2>());
  }
  std::copy(h, h + 4, o.cuts);
  o.npieces = np;
  o.order = std::move(order);
  return o;
}

const RowOrder *find_row_order(pm_graph *g, bool csr) {
  try {
    return &ensure_row_order(g, csr);
  } catch (const Failure &f) {
    if (f.status != PM_ERR_OOM) throw;
    return nullptr;
  }
}

// Bytes that building (the missing parts of) a copy takes at most: the slots, the
// tables, and while it is built the sort of the degrees.
static size_t copy_bytes(const pm_graph *g, bool csr, bool built, bool weighted) {
  const size_t slots = 4 * (size_t)(g->m + 2048), n = (size_t)g->n;
  const bool ordered = (csr ? g->order_out : g->order_in).order.p != nullptr;
  return (weighted ? slots : 0) + (built ? 0 : slots + (ordered ? 20 : 44) * n) + (4u << 20);
}

static void build_sorted(pm_graph *g, bool csr, SortedAdj &b) {
  Engine &E = g->E;
  cudaStream_t st = E.stream;
  const Adj &src = csr ? E.g.out : E.g.in;
  const int64_t n = g->n, m = g->m;
  const RowOrder &o = ensure_row_order(g, csr);
  SortedView v;
  v.n = (int32_t)n;
  v.piece = piece_edges(m);
  v.rc = o.cuts[0];
  v.rh = o.cuts[1];
  v.rm = o.cuts[2];
  v.rl = o.cuts[3];
  v.order = o.order.as<int32_t>();
  DevBuf odeg((size_t)n * 4), pos((size_t)n * 4);
  const int grid = E.grid_for(n, 256, 16);
  const int64_t rows = v.rm + v.slices();  // entries of off before its end
  DevBuf off((size_t)(rows + 1) * 4), len((size_t)(rows + 1) * 4), pieces((size_t)(v.rc + 1) * 4),
      pfirst((size_t)(v.rc + 1) * 4), bdeg((size_t)std::max(v.rl - v.rm, 1));
  PM_CUDA(cudaMemsetAsync(len.as<int32_t>() + rows, 0, 4, st));
  PM_CUDA(cudaMemsetAsync(pieces.as<int32_t>() + v.rc, 0, 4, st));
  PM_LAUNCH(k_sort_tables, grid, 256, 0, st, v.order, src.off, E.g.out.off, n, v.rc, v.rm,
            v.rl, v.piece, pos.as<int32_t>(), odeg.as<int32_t>(), len.as<int32_t>(), pieces.as<int32_t>(),
            bdeg.as<uint8_t>());
  exclusive_sum(len.as<int32_t>(), off.as<int32_t>(), rows + 1, st);
  exclusive_sum(pieces.as<int32_t>(), pfirst.as<int32_t>(), v.rc + 1, st);
  int32_t np = 0, slots = 0;
  PM_CUDA(cudaMemcpyAsync(&np, pfirst.as<int32_t>() + v.rc, 4, cudaMemcpyDeviceToHost, st));
  PM_CUDA(cudaMemcpyAsync(&slots, off.as<int32_t>() + rows, 4, cudaMemcpyDeviceToHost, st));
  PM_CUDA(cudaStreamSynchronize(st));
  v.np = np;
  DevBuf ids((size_t)std::max(slots, 1) * 4), ptab((size_t)std::max(np, 1) * 16),
      partials((size_t)std::max(np, 1) * 8), done((size_t)std::max(v.rc, 1) * 4);
  PM_CUDA(cudaMemsetAsync(done.p, 0, (size_t)std::max(v.rc, 1) * 4, st));
  v.off = off.as<int32_t>();
  v.odeg = odeg.as<int32_t>();
  v.deg = bdeg.as<uint8_t>();
  v.pieces = ptab.as<int4>();
  v.pfirst = pfirst.as<int32_t>();
  v.ids = ids.as<int32_t>();
  v.partials = partials.p;
  v.done = done.as<int32_t>();
  if (v.rc > 0)
    PM_LAUNCH(k_sort_pieces, E.grid_for(v.rc, 256, 16), 256, 0, st, v.pfirst, v.off, v.rc, v.piece, ptab.as<int4>());
  const int64_t blocks = v.blocks();
  if (blocks > 0)
    PM_LAUNCH((k_sort_fill<true>), (unsigned)blocks, kSortThreads, 0, st, E.g, v, src.off, src.idx, nullptr,
              pos.as<int32_t>(), ids.as<int32_t>(), nullptr);
  b.odeg = std::move(odeg);
  b.off = std::move(off);
  b.ids = std::move(ids);
  b.deg = std::move(bdeg);
  b.pieces = std::move(ptab);
  b.pfirst = std::move(pfirst);
  b.partials = std::move(partials);
  b.done = std::move(done);
  b.slots = slots;
  b.view = std::make_shared<SortedView>(v);
}

const SortedView *ensure_sorted(pm_graph *g, bool csr, bool weighted, SortedView &view) {
  // slices pad by at most 32 * kSortShort slots in all, and round up once
  if (g->is_part || g->lean || g->m > (1ll << 31) - 8192) return nullptr;
  SortedAdj &b = csr ? g->sorted_out : g->sorted_in;
  Engine &E = g->E;
  const bool have = b.view && (!weighted || b.w.p);
  // a build that found no room is not repeated (its sorts and passes, and the
  // block cache emptied for nothing) until there is
  if (!have && b.need > 0 && dev_available() < b.need) return nullptr;
  try {
    OptionalAlloc optional;
    if (!b.view) build_sorted(g, csr, b);
    if (weighted && !b.w.p) {
      const DevBuf &w = csr ? g->w_f32_out : g->w_f32_in;
      if (!w.p) fail(PM_ERR_INVALID_ARG, "graph has no float weights");
      DevBuf sw((size_t)std::max<int64_t>(b.slots, 1) * 4);
      const SortedView &v = *b.view;
      const int64_t blocks = v.blocks();
      if (blocks > 0)
        PM_LAUNCH((k_sort_fill<false>), (unsigned)blocks, kSortThreads, 0, E.stream, E.g, v, csr ? E.g.out.off : E.g.in.off,
                  nullptr, w.as<float>(), nullptr, nullptr, sw.as<float>());
      b.w = std::move(sw);
    }
  } catch (const Failure &f) {
    if (f.status != PM_ERR_OOM) throw;
    b.need = copy_bytes(g, csr, b.view != nullptr, weighted);
    return nullptr;
  }
  b.need = 0;
  view = *b.view;
  view.w = weighted ? b.w.as<float>() : nullptr;
  return &view;
}

static bool has_copies(const pm_graph *g) {
  return g->sorted_in.odeg.p || g->sorted_out.odeg.p || g->parts_layout.state > 0;
}
static void give_back(pm_graph *g) {
  g->E.release_graphs();
  for (bool csr : {false, true}) {
    SortedAdj &b = csr ? g->sorted_out : g->sorted_in;
    if (!b.view) continue;
    const bool weighted = b.w.p != nullptr;
    b = SortedAdj{};
    b.need = copy_bytes(g, csr, false, weighted);
  }
  if (g->parts_layout.state > 0) {
    g->parts_layout = PartsLayout{};
    g->parts_layout.need = parts_layout_bytes(g);
  }
}

bool drop_copies(pm_graph *g) {
  if (!has_copies(g)) return false;
  PM_CUDA(cudaStreamSynchronize(g->E.stream));
  give_back(g);
  return true;
}

// Every handle of the process.  The list's lock is held while one is looked at,
// so that none is destroyed meanwhile; a handle's own lock, so that no call
// starts on it.
namespace {
struct Handles {
  std::mutex mu;
  std::vector<pm_graph *> list;
};
Handles &handles() {
  static Handles *h = new Handles();  // never destroyed: handles may outlive static teardown order
  return *h;
}
}  // namespace

void register_graph(pm_graph *g) {
  std::lock_guard<std::mutex> lk(handles().mu);
  handles().list.push_back(g);
}
void unregister_graph(pm_graph *g) {
  Handles &h = handles();
  std::lock_guard<std::mutex> lk(h.mu);
  h.list.erase(std::remove(h.list.begin(), h.list.end(), g), h.list.end());
}

bool reclaim_copies(int device) {
  std::lock_guard<std::mutex> lk(handles().mu);
  // freed with no stream named: a taker waits for the device first
  AllocScope unknown(AllocCtx{});
  bool any = false;
  for (pm_graph *g : handles().list) {
    if (g->device != device) continue;
    std::unique_lock<std::mutex> own(g->use_mu, std::try_to_lock);
    if (!own || g->users > 0 || !has_copies(g)) continue;
    give_back(g);
    any = true;
  }
  return any;
}

__global__ void __launch_bounds__(kAuxSlots) k_fix_end(double2 *aux, double tail_first, double tail_norm,
                                                       const double *d_tail_norm, double tol, FixState *st) {
  __shared__ double2 s[kAuxSlots / 32];
  if (st->stop) return;
  const int t = threadIdx.x;
  double2 v = aux[t];
  aux[t] = make_double2(0.0, 0.0);
  v.x = warp_sum(v.x);
  v.y = warp_sum(v.y);
  if ((t & 31) == 0) s[t >> 5] = v;
  __syncthreads();
  if (t == 0) {
    double y = d_tail_norm ? *d_tail_norm : tail_norm;
    // a row without edges keeps its value: no change, or inf - inf = NaN
    double x = (st->iters == 0 ? tail_first : 0.0) + (y - y);
    for (int i = 0; i < kAuxSlots / 32; ++i) {
      x += s[i].x;
      y += s[i].y;
    }
    st->rel = y > 0 ? x / y : 0.0;
    st->iters += 1;
    st->stop = st->rel <= tol;
  }
}

// *dst = the pass's spread sum plus tail; the slots are cleared.
__global__ void __launch_bounds__(kAuxSlots) k_sum_aux(double2 *aux, double tail, double *dst) {
  __shared__ double s[kAuxSlots / 32];
  const int t = threadIdx.x;
  const double v = warp_sum(aux[t].x);
  aux[t] = make_double2(0.0, 0.0);
  if ((t & 31) == 0) s[t >> 5] = v;
  __syncthreads();
  if (t == 0) {
    double x = tail;
    for (int i = 0; i < kAuxSlots / 32; ++i) x += s[i];
    *dst = x;
  }
}

// ---------------------------------------------------------------------------
// PageRank (numa-PageRank.C:64-148, loop 273-335; the semantics PR_F states).
// The frontier starts as every vertex and only shrinks: a vertex that gets no
// push leaves it and nothing reaches it again.  So for a frontier vertex the
// stale vector is 0 (its entry was zeroed a pass ago) and the new rank is
// damping * sum + added; a vertex that leaves at pass t holds `added` in the
// vector of that pass and 0 in the other, for good: its result is known then.
// A pass therefore reads the contributions and out-degrees and writes the
// next contributions; ranks are written when they are final (or every pass,
// when the residuals are asked for).
// ---------------------------------------------------------------------------
template <class T, bool RESID>
struct PRS_F {
  const T *c_cur;
  T *c_next;
  T *p;
  const int32_t *odeg;
  T damping, added, gone;  // gone: the result of a vertex that leaves in this pass
  bool last;
  using Acc = T;
  static constexpr bool kAux = RESID;
  __device__ __forceinline__ Acc identity() const { return T(-0.0); }
  __device__ __forceinline__ Acc edge(int s, float) const { return __ldg(c_cur + s); }
  __device__ __forceinline__ Acc combine(Acc a, Acc b) const { return a + b; }
  struct Row {
    T c;
    int deg;
  };
  __device__ __forceinline__ Row pre(int r) const { return Row{__ldg(c_cur + r), __ldg(odeg + r)}; }
  __device__ __forceinline__ void commit(int r, Acc acc, Row row, double2 &resid) const {
    const bool hit = !signbit(acc);
    if (signbit(row.c)) {  // outside the frontier: its two vectors take turns
      c_next[r] = T(-0.0);
      if constexpr (RESID) resid.x += (double)added;
      return;
    }
    const T nb = damping * (T(0) + acc) + added;
    if constexpr (RESID) resid.x += fabs((double)nb - (double)p[r]);
    c_next[r] = hit ? (row.deg > 0 ? nb / T(row.deg) : T(0)) : T(-0.0);
    if (RESID || last || !hit) p[r] = hit ? nb : gone;
  }
};

template <class T>
__global__ void k_prs_init(T *c, T *c_other, T *p, const int32_t *__restrict__ odeg, int64_t n, int64_t rl,
                           T tail_rank) {
  const T p0 = T(1) / T(n);
  GRID_STRIDE(r, n) {
    const int deg = odeg[r];
    c[r] = deg > 0 ? p0 / T(deg) : T(0);
    if (r < rl) {
      p[r] = p0;
    } else {  // no in-edges: leaves in the first pass
      c_other[r] = T(-0.0);
      p[r] = tail_rank;
    }
  }
}

template <class T>
bool run_pagerank_sorted(pm_graph *g, int iters, double damping, T *d_out, double *d_resid) {
  Engine &E = g->E;
  SortedView a;
  // outside [0, 1] a rank may turn negative: the sign of a contribution is then
  // no longer the frontier alone, and a vertex can come back into it
  if (!(damping >= 0.0 && damping <= 1.0) || !ensure_sorted(g, false, false, a)) return false;
  const int64_t n = g->n;
  T *c0 = (T *)g->scratch_buf(0, (size_t)n * sizeof(T));
  T *c1 = (T *)g->scratch_buf(1, (size_t)n * sizeof(T));
  T *p = (T *)g->scratch_buf(2, (size_t)n * sizeof(T));
  double2 *aux = nullptr;
  if (d_resid) {
    aux = (double2 *)g->scratch_buf(3, kAuxSlots * sizeof(double2));
    PM_CUDA(cudaMemsetAsync(aux, 0, kAuxSlots * sizeof(double2), E.stream));
  }
  const T dmp = (T)damping, added = (T)((1.0 - damping) * (1.0 / (double)n)), p0 = T(1) / T(n);
  // a vertex that leaves at pass t: added after an even number of later passes
  auto gone = [&](int t) { return (iters - 1 - t) % 2 == 0 ? added : T(0); };
  PM_LAUNCH((k_prs_init<T>), E.grid_for(n, 256, 16), 256, 0, E.stream, c0, c1, p, a.odeg, n, (int64_t)a.rl,
            iters > 0 ? gone(0) : p0);
  E.run_loop(loop_key("pagerank_sorted", (int)sizeof(T), iters, damping, c0, c1, p, aux, d_resid), [&] {
    T *x = c0, *y = c1;
    for (int it = 0; it < iters; ++it) {
      E.prof.begin("pagerank", E.stream);
      if (d_resid)
        launch_sorted_pull<false>(E, a, PRS_F<T, true>{x, y, p, a.odeg, dmp, added, gone(it), it == iters - 1}, aux);
      else
        launch_sorted_pull<false>(E, a, PRS_F<T, false>{x, y, p, a.odeg, dmp, added, gone(it), it == iters - 1});
      E.prof.end(E.stream);
      // from the second pass on the vertices without in-edges push nothing
      if (it == 0) launch_fill_tail(E, a, x, T(-0.0));
      if (d_resid) {
        const double each = it == 0 ? fabs((double)added - (double)p0) : (double)added;
        PM_LAUNCH(k_sum_aux, 1, kAuxSlots, 0, E.stream, aux, each * (double)(n - a.rl), d_resid + it);
      }
      std::swap(x, y);
    }
  });
  launch_to_vertices(E, a, p, d_out);
  return true;
}

// ---------------------------------------------------------------------------
// SpMV (numa-SPMV.C:56-110, loop 168-193): y = A_w^T x, then x = y.
// ---------------------------------------------------------------------------
template <class T, bool NORM>
struct SPMVS_F {
  const T *x;
  T *y;
  using Acc = T;
  static constexpr bool kAux = NORM;
  __device__ __forceinline__ Acc identity() const { return T(-0.0); }
  __device__ __forceinline__ Acc edge(int s, float w) const { return T(w) * __ldg(x + s); }
  __device__ __forceinline__ Acc combine(Acc a, Acc b) const { return a + b; }
  __device__ __forceinline__ int pre(int) const { return 0; }
  __device__ __forceinline__ void commit(int r, Acc acc, int, double2 &norm) const {
    const T v = acc + T(0);
    y[r] = v;
    if constexpr (NORM) norm.x += fabs((double)v);
  }
};

template <class T>
bool run_spmv_sorted(pm_graph *g, const T *d_x0, int iters, T *d_y, double *d_norm) {
  Engine &E = g->E;
  SortedView a;
  if (!ensure_sorted(g, false, true, a)) return false;
  const int64_t n = g->n;
  T *x = (T *)g->scratch_buf(0, (size_t)n * sizeof(T));
  T *y = (T *)g->scratch_buf(1, (size_t)n * sizeof(T));
  double2 *aux = nullptr;
  if (d_norm) {
    aux = (double2 *)g->scratch_buf(3, kAuxSlots * sizeof(double2));
    PM_CUDA(cudaMemsetAsync(aux, 0, kAuxSlots * sizeof(double2), E.stream));
  }
  launch_to_positions(E, a, d_x0, x);
  launch_fill_tail(E, a, y, T(0));
  E.run_loop(loop_key("spmv_sorted", (int)sizeof(T), iters, x, y, (const void *)a.w, aux, d_norm), [&] {
    T *s = x, *t = y;
    for (int it = 0; it < iters; ++it) {
      E.prof.begin("spmv", E.stream);
      if (d_norm)
        launch_sorted_pull<true>(E, a, SPMVS_F<T, true>{s, t}, aux);
      else
        launch_sorted_pull<true>(E, a, SPMVS_F<T, false>{s, t});
      E.prof.end(E.stream);
      if (it == 0) launch_fill_tail(E, a, s, T(0));  // rows without in-edges
      if (d_norm) PM_LAUNCH(k_sum_aux, 1, kAuxSlots, 0, E.stream, aux, 0.0, d_norm + it);
      std::swap(s, t);
    }
  });
  launch_to_vertices(E, a, iters % 2 ? y : x, d_y);
  return true;
}

template bool run_pagerank_sorted<float>(pm_graph *, int, double, float *, double *);
template bool run_pagerank_sorted<double>(pm_graph *, int, double, double *, double *);
template bool run_spmv_sorted<float>(pm_graph *, const float *, int, float *, double *);
template bool run_spmv_sorted<double>(pm_graph *, const double *, int, double *, double *);

}  // namespace pm
