// pm_ppr.cu -- personalised PageRank for up to 32 seeds in one SpMM-shaped
// pull per iteration (PR_F's push p[s]/outdeg(s) and PR_Vertex_F's damping,
// numa-PageRank.C:87-90, 125-137, applied to all vectors at once, teleport to
// each vector's seed).  The contribution matrix C (COLS floats a row, C[u][j]
// = x_j[u] / outdeg(u); COLS the seeds rounded up to 8, 16 or 32) is gathered
// one row per in-edge, COLS / 4 lanes holding four columns each.
//
// The matrices live in the positions of the degree-sorted copy
// (pm_sorted.cuh): a pass reads offsets, out-degrees and ids and writes the
// next matrix in order, and the rows most edges gather lie together.  Rows of
// 1024 edges or more are cut into pieces of a CTA each, rows of 128 or more
// take a warp, of 32 or more COLS / 4 lanes, and the shorter ones -- most rows,
// a third of the edges -- as much, out of slices, where the rows of a warp have
// (nearly) the same length and one id load covers 32 edges of them.  Rows
// without in-edges never change after the first iteration.
//
// What bounds it: the row gathers -- of 34 GB a pass 12.5 GB come from DRAM, the
// rest from the L2 and L1 -- and the number of warps to wait for them.
// Directed 2^24-vertex, 263 M-edge R-MAT, 32 seeds, 20 iterations: 108 ms with
// a warp per row in vertex order and a lane per column, 73.9 ms with rows by
// degree but the matrices in vertex order (k_ppr_pull; 72.1 with packed
// additions and no test per gather), 65 to 68 ms here; 16 seeds 54.9 -> 42.9 ms,
// 8 seeds 40.3 -> 28.9 ms.
#include "pm_sorted.cuh"

namespace pm {

using u64 = unsigned long long;

constexpr int kPprCols = 32;

// Four columns as two packed pairs: Blackwell adds a pair in one instruction.
struct Quad {
  u64 lo, hi;
};
__device__ __forceinline__ u64 pair_add(u64 a, u64 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ void add4(Quad &a, const Quad &b) {
  a.lo = pair_add(a.lo, b.lo);
  a.hi = pair_add(a.hi, b.hi);
}
__device__ __forceinline__ Quad ldg4(const float *p) {
  const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(p));
  return Quad{v.x, v.y};
}
__device__ __forceinline__ float4 unpack4(const Quad &a) {
  return make_float4(__uint_as_float((unsigned)a.lo), __uint_as_float((unsigned)(a.lo >> 32)),
                     __uint_as_float((unsigned)a.hi), __uint_as_float((unsigned)(a.hi >> 32)));
}
template <int COLS>
__device__ __forceinline__ Quad xor_add4(Quad a) {  // over the groups of COLS / 4 lanes of a warp
#pragma unroll
  for (int d = COLS / 4; d < 32; d <<= 1)
    add4(a, Quad{__shfl_xor_sync(0xffffffffu, a.lo, d), __shfl_xor_sync(0xffffffffu, a.hi, d)});
  return a;
}

// This lane group's sum of the rows named by idx[e], idx[e + step], ... below
// e1 (the lane's four columns): kPprStep row gathers in flight per group.
// Past e1 a group adds row `zero`, which holds zeros: no test and no select
// per gather.  All lanes of the warp call it; groups may have different rows
// and lengths.
constexpr int kPprStep = 4;
template <int COLS>
__device__ __forceinline__ Quad ppr_sum(const int32_t *__restrict__ idx, EdgePos e, EdgePos e1, int step,
                                        const float *__restrict__ c, int zero) {
  constexpr int L = COLS / 4, U = kPprStep;      // lanes per row; gathers per step
  constexpr int B = L > U ? L : U, I = B / L;    // edges and id loads per batch
  const int sub = lane_id() % L;
  const float *col = c + 4 * sub;
  Quad acc{0, 0};
  for (; __any_sync(0xffffffffu, e < e1); e += B * step) {
    int id[I];
#pragma unroll
    for (int i = 0; i < I; ++i) {
      const EdgePos x = e + (i * L + sub) * step;
      id[i] = x < e1 ? __ldcs(idx + x) : zero;
    }
#pragma unroll
    for (int b = 0; b < B; b += U) {
      if (b > 0 && !__any_sync(0xffffffffu, e + b * step < e1)) break;
      Quad v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = ldg4(col + (int64_t)__shfl_sync(0xffffffffu, id[(b + u) / L], (b + u) % L, L) * COLS);
      // in pairs: a quarter of the roundings of the running sum
#pragma unroll
      for (int d = 1; d < U; d *= 2)
#pragma unroll
        for (int u = 0; u < U; u += 2 * d) add4(v[u], v[u + d]);
      add4(acc, v[0]);
    }
  }
  return acc;
}

// ---------------------------------------------------------------------------
// In vertex order, for handles without a sorted copy (more edges than its
// slots can name, or no room): rows with more than g.heavy_deg in-edges are
// summed by chunk CTAs first, the rest in order of in-degree, a warp each for
// the longest, COLS / 4 lanes each for the others.
// ---------------------------------------------------------------------------
template <int COLS>
__global__ void __launch_bounds__(256) k_ppr_heavy(GraphView g, const float *__restrict__ c,
                                                   float *__restrict__ partials) {
  constexpr int L = COLS / 4;
  __shared__ Quad s_part[8][L];
  const int ch = blockIdx.x;
  if (ch >= g.in.nchunks) return;
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int r = __ldg(g.in.hrow + ch);
  const int k = ch - __ldg(g.in.hfirst + r);
  const int row_end = __ldg(g.in.off + r + 1);
  const int e0 = __ldg(g.in.off + r) + k * kChunkEdges, e1 = min(row_end - e0, kChunkEdges) + e0;
  const Quad sum = xor_add4<COLS>(ppr_sum<COLS>(g.in.idx, (EdgePos)e0 + threadIdx.x / L, e1, 256 / L, c, g.n));
  if (lane < L) s_part[wid][lane] = sum;
  __syncthreads();
  if (wid == 0 && lane < L) {
    Quad t = s_part[0][lane];
    for (int w = 1; w < 8; ++w) add4(t, s_part[w][lane]);
    reinterpret_cast<float4 *>(partials)[(int64_t)ch * L + lane] = unpack4(t);
  }
}

// Row v's new value and contribution: this lane's four columns.
template <int COLS>
__device__ __forceinline__ void ppr_commit(const GraphView &g, int v, const float4 &acc, const int4 &seed, float damping,
                                           float *__restrict__ c_next, float *__restrict__ y_out, int k_out) {
  const int sub = lane_id() % (COLS / 4);
  const int od = __ldg(g.out.off + v + 1) - __ldg(g.out.off + v);
  const float jump = 1.0f - damping;
  float4 y;
  y.x = damping * acc.x + (v == seed.x ? jump : 0.0f);
  y.y = damping * acc.y + (v == seed.y ? jump : 0.0f);
  y.z = damping * acc.z + (v == seed.z ? jump : 0.0f);
  y.w = damping * acc.w + (v == seed.w ? jump : 0.0f);
  if (y_out) {
    float *out = y_out + (int64_t)v * k_out + 4 * sub;
    if (4 * sub < k_out) out[0] = y.x;
    if (4 * sub + 1 < k_out) out[1] = y.y;
    if (4 * sub + 2 < k_out) out[2] = y.z;
    if (4 * sub + 3 < k_out) out[3] = y.w;
  }
  const float f = (float)od;
  const float4 cn = od > 0 ? make_float4(y.x / f, y.y / f, y.z / f, y.w / f) : make_float4(0.f, 0.f, 0.f, 0.f);
  *reinterpret_cast<float4 *>(c_next + (int64_t)v * COLS + 4 * sub) = cn;
}
// The seeds of this lane's columns (-1 past the last).
template <int COLS>
__device__ __forceinline__ int4 ppr_seeds(const int32_t *__restrict__ seeds, int k) {
  const int j = 4 * (lane_id() % (COLS / 4));
  return make_int4(j < k ? __ldg(seeds + j) : -1, j + 1 < k ? __ldg(seeds + j + 1) : -1,
                   j + 2 < k ? __ldg(seeds + j + 2) : -1, j + 3 < k ? __ldg(seeds + j + 3) : -1);
}

// order: vertices by in-degree (null: by id); [0, rh) have kSortLong in-edges or more and
// take a warp each, [rh, rl) a group of lanes each.
template <int COLS>
__global__ void __launch_bounds__(256, COLS == 32 ? 8 : 6) k_ppr_pull(GraphView g, const int32_t *__restrict__ order, int rh, int rl,
                                                     const float *__restrict__ c_cur, float *__restrict__ c_next,
                                                     float *__restrict__ y_out, int k_out,
                                                     const float *__restrict__ partials,
                                                     const int32_t *__restrict__ seeds, float damping) {
  constexpr int L = COLS / 4;
  const int lane = lane_id(), group = lane / L;
  const int64_t t = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int4 seed = ppr_seeds<COLS>(seeds, k_out);
  if (t < rh) {
    const int v = order ? __ldg(order + t) : (int)t;
    const int o = __ldg(g.in.off + v), o1 = __ldg(g.in.off + v + 1);
    Quad acc{0, 0};
    if (o1 - o > g.heavy_deg) {
      const int first = __ldg(g.in.hfirst + v), nch = edge_pieces(o1 - o, kChunkEdges);
      for (int q = 0; q < nch; ++q)
        add4(acc, ldg4(partials + ((int64_t)(first + q) * L + lane % L) * 4));
    } else {
      acc = xor_add4<COLS>(ppr_sum<COLS>(g.in.idx, (EdgePos)o + group, o1, 32 / L, c_cur, g.n));
    }
    if (lane < L) ppr_commit<COLS>(g, v, unpack4(acc), seed, damping, c_next, y_out, k_out);
  } else {
    const int64_t r = rh + (t - rh) * (32 / L) + group;
    int v = 0, o = 0, o1 = 0;
    bool heavy = false;
    if (r < rl) {
      v = __ldg(order + r);
      o = __ldg(g.in.off + v);
      o1 = __ldg(g.in.off + v + 1);
      heavy = o1 - o > g.heavy_deg;  // a cut-off below kSortLong
    }
    Quad acc = ppr_sum<COLS>(g.in.idx, heavy ? o1 : o, o1, 1, c_cur, g.n);
    if (heavy) acc = ldg4(partials + ((int64_t)__ldg(g.in.hfirst + v) * L + lane % L) * 4);
    if (r < rl) ppr_commit<COLS>(g, v, unpack4(acc), seed, damping, c_next, y_out, k_out);
  }
}

// The vertices without in-edges (order[rl .. n)): their rows of the second
// matrix and of the result, which no iteration changes.
template <int COLS>
__global__ void __launch_bounds__(256) k_ppr_tail(GraphView g, const int32_t *__restrict__ order, int rl,
                                                  float *__restrict__ c, float *__restrict__ y_out, int k_out,
                                                  const int32_t *__restrict__ seeds, float damping) {
  constexpr int L = COLS / 4;
  const int4 seed = ppr_seeds<COLS>(seeds, k_out);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x / L;
  for (int64_t r = rl + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / L; r < g.n; r += stride)
    ppr_commit<COLS>(g, __ldg(order + r), make_float4(0.f, 0.f, 0.f, 0.f), seed, damping, c, y_out, k_out);
}

// C0[v][j] = x / outdeg(v) for the seeds v = seeds[j]; with tail only those
// without in-edges.
__global__ void k_ppr_seed(const int32_t *seeds, int k, GraphView g, float *c, int cols, float x, bool tail,
                           float *y0, int k_out) {
  const int j = threadIdx.x;
  if (j >= k) return;
  const int v = seeds[j];
  if (tail && g.in.off[v + 1] > g.in.off[v]) return;
  const int od = g.out.off[v + 1] - g.out.off[v];
  c[(int64_t)v * cols + j] = od > 0 ? x / (float)od : 0.f;
  if (y0) y0[(int64_t)v * k_out + j] = x;
}

// ---------------------------------------------------------------------------
// Over the degree-sorted copy.
// ---------------------------------------------------------------------------
// Position r's new value and contribution: this lane's four columns.  at: the
// seeds' positions, looked at only when some (the same for the whole warp)
// says that one of them may be r.  OUT: the last pass, which writes the result.
template <int COLS, bool OUT>
__device__ __forceinline__ void ppr_commit_at(const SortedView &a, int r, const Quad &sum, bool some,
                                              const int32_t *__restrict__ at, float damping,
                                              float *__restrict__ c_next, float *__restrict__ y_out, int k) {
  const int sub = lane_id() % (COLS / 4);
  const float4 acc = unpack4(sum);
  float4 y = make_float4(damping * acc.x + 0.0f, damping * acc.y + 0.0f, damping * acc.z + 0.0f, damping * acc.w + 0.0f);
  if (some) {
    const int4 seed = ppr_seeds<COLS>(at, k);
    const float jump = 1.0f - damping;
    if (r == seed.x) y.x = damping * acc.x + jump;
    if (r == seed.y) y.y = damping * acc.y + jump;
    if (r == seed.z) y.z = damping * acc.z + jump;
    if (r == seed.w) y.w = damping * acc.w + jump;
  }
  if constexpr (OUT) {
    float *out = y_out + (int64_t)__ldg(a.order + r) * k + 4 * sub;
    if (4 * sub < k) out[0] = y.x;
    if (4 * sub + 1 < k) out[1] = y.y;
    if (4 * sub + 2 < k) out[2] = y.z;
    if (4 * sub + 3 < k) out[3] = y.w;
  } else {
    const int od = __ldg(a.odeg + r);
    const float f = (float)od;
    const float4 cn = od > 0 ? make_float4(y.x / f, y.y / f, y.z / f, y.w / f) : make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4 *>(c_next + (int64_t)r * COLS + 4 * sub) = cn;
  }
}

// Rows of a slice a warp takes (kPer per group of lanes), and the gathers a
// lane has in flight there.
template <int COLS>
struct PprSlice {
  static constexpr int kPer = 1;
  static constexpr int kRows = kPer * 128 / COLS;
  static constexpr int kFlight = 2;
};
template <int COLS>
struct PprPlan {  // warps by kind of row
  int64_t rows, subs, slices;
  __host__ __device__ explicit PprPlan(const SortedView &a)
      : rows(a.rh - a.rc), subs(((int64_t)(a.rm - a.rh) * (COLS / 4) + 31) / 32),
        slices(a.slices() * (32 / PprSlice<COLS>::kRows)) {}
  int64_t blocks(const SortedView &a) const { return a.np + (rows + subs + slices + 7) / 8; }
};

// CTAs per SM: 32 seeds on 2^24 vertices, 263 M edges, 20 iterations take
// 82.9 ms with four (four rows of a slice per group, eight gathers in flight),
// 72.9 with five (two rows), 65.6 with six (two rows, four in flight), 65.1
// with seven (one row, four) and 64.9 with eight (one row, two).
constexpr int kPprCtas = 8;
template <int COLS, bool OUT>
__global__ void __launch_bounds__(256, kPprCtas)
    k_ppr_sorted(SortedView a, const float *__restrict__ c, float *__restrict__ c_next, float *__restrict__ y_out,
                 int k, float *part, const int32_t *__restrict__ at, float damping) {
  constexpr int L = COLS / 4, G = 32 / L;  // lanes per row, rows a warp gathers at once
  const int lane = lane_id(), wid = threadIdx.x >> 5, sub = lane % L, group = lane / L;
  const PprPlan<COLS> plan(a);
  const int64_t t = ((int64_t)blockIdx.x - a.np) * 8 + wid;
  const int32_t my_seed = lane < k ? __ldg(at + lane) : -1;
  // whether a seed lies in [first, first + count), by the whole warp
  auto seed_in = [&](int64_t first, int count) {
    return __any_sync(0xffffffffu, my_seed >= first && my_seed < first + count) != 0;
  };
  if (t < 0) {
    __shared__ Quad s_part[8][L];
    const int4 pc = __ldg(a.pieces + blockIdx.x);
    const Quad sum = xor_add4<COLS>(ppr_sum<COLS>(a.ids, pc.x + (int)threadIdx.x / L, pc.y, 256 / L, c, a.n));
    if (lane < L) s_part[wid][lane] = sum;
    __syncthreads();
    if (wid != 0) return;
    Quad v = s_part[0][sub];
    for (int w = 1; w < 8; ++w) add4(v, s_part[w][sub]);
    if (pc.w >= 0) {  // one of several pieces: the last to finish folds them
      const int count = __ldg(a.pfirst + pc.z + 1) - pc.w;
      if (lane < L) {
        *reinterpret_cast<float4 *>(part + (int64_t)blockIdx.x * COLS + 4 * lane) = unpack4(v);
        __threadfence();
      }
      __syncwarp();
      int last = 0;
      if (lane == 0) last = atomicAdd(a.done + pc.z, 1) == count - 1;
      if (!__shfl_sync(0xffffffffu, last, 0)) return;
      __threadfence();  // the other pieces' sums, written before they were counted
      v = Quad{0, 0};
      for (int q = group; q < count; q += G) {
        const ulonglong2 x = __ldcg(reinterpret_cast<const ulonglong2 *>(part + (int64_t)(pc.w + q) * COLS + 4 * sub));
        add4(v, Quad{x.x, x.y});
      }
      v = xor_add4<COLS>(v);
      if (lane == 0) a.done[pc.z] = 0;
    }
    const bool some = seed_in(pc.z, 1);
    if (lane < L) ppr_commit_at<COLS, OUT>(a, pc.z, v, some, at, damping, c_next, y_out, k);
  } else if (t < plan.rows) {
    const int r = a.rc + (int)t;
    const Quad v = xor_add4<COLS>(ppr_sum<COLS>(a.ids, __ldg(a.off + r) + group, __ldg(a.off + r + 1), G, c, a.n));
    const bool some = seed_in(r, 1);
    if (lane < L) ppr_commit_at<COLS, OUT>(a, r, v, some, at, damping, c_next, y_out, k);
  } else if (t < plan.rows + plan.subs) {
    const int64_t r = a.rh + (t - plan.rows) * G + group;
    const bool in = r < a.rm;
    const Quad v = ppr_sum<COLS>(a.ids, in ? __ldg(a.off + r) : 0, in ? __ldg(a.off + r + 1) : 0, 1, c, a.n);
    const bool some = seed_in(r - group, G);
    if (in) ppr_commit_at<COLS, OUT>(a, (int)r, v, some, at, damping, c_next, y_out, k);
  } else if (t < plan.rows + plan.subs + plan.slices) {
    using P = PprSlice<COLS>;
    constexpr int R = P::kRows, J = P::kPer, S = 32 / R;     // S: slots an id load covers
    constexpr int K = P::kFlight / J, I = K > S ? K / S : 1;  // slots a step gathers, id loads per batch
    const int64_t q = t - plan.rows - plan.subs, s = q / S;
    const int in_slice = (int)(q % S) * R;
    const int64_t base = a.rm + 32 * s + in_slice;
    if (base >= a.rl) return;
    const int64_t mine = base + lane % R;  // the row whose ids this lane loads
    const int d = mine < a.rl ? (int)__ldg(a.deg + (mine - a.rm)) : 0;
    const int longest = __shfl_sync(0xffffffffu, d, 0);
    const int32_t *ids = a.ids + __ldg(a.off + a.rm + s) + in_slice + lane % R;
    const float *col = c + 4 * sub;
    Quad acc[J];
#pragma unroll
    for (int j = 0; j < J; ++j) acc[j] = Quad{0, 0};
    for (int k0 = 0; k0 < longest; k0 += S * I) {
      int id[I];
#pragma unroll
      for (int i = 0; i < I; ++i) {
        const int slot = k0 + i * S + lane / R;
        id[i] = slot < d ? __ldcs(ids + 32 * slot) : a.n;  // past the row: zeros
      }
#pragma unroll
      for (int b = 0; b < S * I; b += K) {
        if (b > 0 && k0 + b >= longest) break;  // the same for the whole warp
        Quad v[K][J];
#pragma unroll
        for (int u = 0; u < K; ++u)
#pragma unroll
          for (int j = 0; j < J; ++j)
            v[u][j] = ldg4(col + (int64_t)__shfl_sync(0xffffffffu, id[(b + u) / S], (b + u) % S * R + j * G + group) * COLS);
#pragma unroll
        for (int j = 0; j < J; ++j) {
#pragma unroll
          for (int u = 1; u < K; ++u) add4(v[0][j], v[u][j]);
          add4(acc[j], v[0][j]);
        }
      }
    }
    const bool some = seed_in(base, R);
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int64_t r = base + j * G + group;
      if (r < a.rl) ppr_commit_at<COLS, OUT>(a, (int)r, acc[j], some, at, damping, c_next, y_out, k);
    }
  }
}

// The positions of the seeds, at[j] for seed j.
__global__ void __launch_bounds__(256) k_ppr_positions(const int32_t *__restrict__ order, int64_t n,
                                                       const int32_t *__restrict__ seeds, int k, int32_t *at) {
  __shared__ int32_t s_seed[32];
  if (threadIdx.x < k) s_seed[threadIdx.x] = __ldg(seeds + threadIdx.x);
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
    const int32_t v = __ldcs(order + r);
    for (int j = 0; j < k; ++j)
      if (v == s_seed[j]) at[j] = (int32_t)r;
  }
}

// C[at[j]][j] = x / outdeg for the seeds; with tail only those without in-edges.
__global__ void k_ppr_seed_at(SortedView a, const int32_t *at, int k, float *c, int cols, float x, bool tail) {
  const int j = threadIdx.x;
  if (j >= k || (tail && at[j] < a.rl)) return;
  const int od = a.odeg[at[j]];
  c[(int64_t)at[j] * cols + j] = od > 0 ? x / (float)od : 0.f;
}

// The results of the vertices without in-edges: 1 - damping at their seeds.
template <int COLS>
__global__ void __launch_bounds__(256) k_ppr_tail_at(SortedView a, const int32_t *__restrict__ at, int k, float jump,
                                                     float *__restrict__ y) {
  constexpr int L = COLS / 4;
  const int4 seed = ppr_seeds<COLS>(at, k);
  const int sub = lane_id() % L;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x / L;
  for (int64_t r = a.rl + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / L; r < a.n; r += stride) {
    float *out = y + (int64_t)__ldg(a.order + r) * k + 4 * sub;
    if (4 * sub < k) out[0] = r == seed.x ? jump : 0.0f;
    if (4 * sub + 1 < k) out[1] = r == seed.y ? jump : 0.0f;
    if (4 * sub + 2 < k) out[2] = r == seed.z ? jump : 0.0f;
    if (4 * sub + 3 < k) out[3] = r == seed.w ? jump : 0.0f;
  }
}

// False (nothing launched): no sorted copy, or a damping that is not finite
// (whose products with the zero rows are NaN, not 0).
template <int COLS>
static bool run_ppr_sorted(pm_graph *g, const int32_t *d_seeds, int k, int iters, double damping, float *d_out) {
  Engine &E = g->E;
  SortedView a;
  const float dmp = (float)damping;
  if (iters == 0 || !std::isfinite(dmp) || !ensure_sorted(g, false, false, a)) return false;
  const int64_t n = g->n, row = COLS * 4;
  // row n of both holds zeros (ppr_sum)
  char *c0 = (char *)g->scratch_buf(0, (size_t)((n + 1) * row)), *c1 = (char *)g->scratch_buf(1, (size_t)((n + 1) * row));
  float *part = (float *)g->scratch_buf(2, (size_t)std::max(a.np, 1) * row);
  int32_t *at = (int32_t *)g->scratch_buf(4, 32 * 4);
  PM_CUDA(cudaMemsetAsync(c0, 0, (size_t)((n + 1) * row), E.stream));
  PM_CUDA(cudaMemsetAsync(c1 + a.rl * row, 0, (size_t)((n + 1 - a.rl) * row), E.stream));
  PM_LAUNCH(k_ppr_positions, E.grid_for(n, 256, 16), 256, 0, E.stream, a.order, n, d_seeds, k, at);
  PM_LAUNCH(k_ppr_seed_at, 1, 32, 0, E.stream, a, at, k, (float *)c0, COLS, 1.0f, false);
  if (a.rl < n) {
    PM_LAUNCH(k_ppr_seed_at, 1, 32, 0, E.stream, a, at, k, (float *)c1, COLS, 1.0f - dmp, true);
    PM_LAUNCH((k_ppr_tail_at<COLS>), E.grid_for((n - a.rl) * (COLS / 4), 256, 8), 256, 0, E.stream, a, at, k,
              1.0f - dmp, d_out);
  }
  const int64_t blocks = PprPlan<COLS>(a).blocks(a);
  E.run_loop(loop_key("ppr_sorted", iters, k, damping, c0, c1, part, at, d_out), [&] {
    float *x = (float *)c0, *y = (float *)c1;
    for (int it = 0; it < iters; ++it) {
      E.prof.begin("ppr", E.stream);
      if (blocks > 0 && it < iters - 1)
        PM_LAUNCH((k_ppr_sorted<COLS, false>), (unsigned)blocks, 256, 0, E.stream, a, x, y, d_out, k, part, at, dmp);
      else if (blocks > 0)
        PM_LAUNCH((k_ppr_sorted<COLS, true>), (unsigned)blocks, 256, 0, E.stream, a, x, y, d_out, k, part, at, dmp);
      // the seeds without in-edges settle in the first matrix, too
      if (it == 0 && a.rl < n) PM_LAUNCH(k_ppr_seed_at, 1, 32, 0, E.stream, a, at, k, x, COLS, 1.0f - dmp, true);
      E.prof.end(E.stream);
      std::swap(x, y);
    }
  });
  return true;
}

template <int COLS>
static void run_ppr_cols(pm_graph *g, const int32_t *d_seeds, int k, int iters, double damping, float *d_out) {
  if (run_ppr_sorted<COLS>(g, d_seeds, k, iters, damping, d_out)) return;
  Engine &E = g->E;
  const int64_t n = g->n;
  // without memory for the order, a warp per row in vertex order
  const RowOrder *o = find_row_order(g, false);
  const int32_t *order = o ? o->order.as<int32_t>() : nullptr;
  const int rh = o ? o->cuts[1] : (int)n, rl = o ? o->cuts[3] : (int)n;
  // row n of both holds zeros (ppr_sum)
  float *c0 = (float *)g->scratch_buf(0, (size_t)(n + 1) * COLS * 4);
  float *c1 = (float *)g->scratch_buf(1, (size_t)(n + 1) * COLS * 4);
  float *part = (float *)g->scratch_buf(2, (size_t)std::max(E.g.in.nchunks, 1) * COLS * 4);
  const float dmp = (float)damping;
  PM_CUDA(cudaMemsetAsync(c0, 0, (size_t)(n + 1) * COLS * 4, E.stream));
  PM_CUDA(cudaMemsetAsync(c1 + n * COLS, 0, COLS * 4, E.stream));
  if (iters == 0) PM_CUDA(cudaMemsetAsync(d_out, 0, (size_t)n * k * 4, E.stream));
  PM_LAUNCH(k_ppr_seed, 1, 32, 0, E.stream, d_seeds, k, E.g, c0, COLS, 1.0f, false, iters == 0 ? d_out : nullptr, k);
  if (iters > 0 && rl < n)
    PM_LAUNCH((k_ppr_tail<COLS>), E.grid_for((n - rl) * (COLS / 4), 256, 8), 256, 0, E.stream, E.g, order, rl, c1,
              d_out, k, d_seeds, dmp);
  const int64_t warps = rh + ((int64_t)(rl - rh) * (COLS / 4) + 31) / 32;
  E.run_loop(loop_key("ppr", iters, k, damping, c0, c1, part, (const void *)d_seeds, d_out, (const void *)order), [&] {
    float *a = c0, *b = c1;
    for (int it = 0; it < iters; ++it) {
      E.prof.begin("ppr", E.stream);
      if (E.g.in.nchunks > 0)
        PM_LAUNCH((k_ppr_heavy<COLS>), E.g.in.nchunks, 256, 0, E.stream, E.g, a, part);
      if (warps > 0)
        PM_LAUNCH((k_ppr_pull<COLS>), (unsigned)((warps + 7) / 8), 256, 0, E.stream, E.g, order, rh, rl, a, b,
                  it == iters - 1 ? d_out : nullptr, k, part, d_seeds, dmp);
      // the seeds without in-edges settle in the first matrix, too
      if (it == 0) PM_LAUNCH(k_ppr_seed, 1, 32, 0, E.stream, d_seeds, k, E.g, a, COLS, 1.0f - dmp, true, nullptr, k);
      E.prof.end(E.stream);
      std::swap(a, b);
    }
  });
}

void run_ppr(pm_graph *g, const int32_t *d_seeds, int k, int iters, double damping, float *d_out) {
  if (k <= 8)
    run_ppr_cols<8>(g, d_seeds, k, iters, damping, d_out);
  else if (k <= 16)
    run_ppr_cols<16>(g, d_seeds, k, iters, damping, d_out);
  else
    run_ppr_cols<kPprCols>(g, d_seeds, k, iters, damping, d_out);
}

}  // namespace pm
