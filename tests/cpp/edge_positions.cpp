// Walks rows that end at or near the last edge position a handle can hold the
// way the kernels do (include/pm/pm_edges.cuh), with 64-bit arithmetic beside
// it: every edge of the row must be met exactly once and nothing outside it.
// Prints the number of walks; exits 1 with a message at the first mistake.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "pm_edges.cuh"

using namespace pm;

static void fail(const char *what, int64_t end, int64_t len, int64_t x) {
  std::printf("%s: row of %lld edges ending at %lld, %lld\n", what, (long long)len, (long long)end, (long long)x);
  std::exit(1);
}

struct Row {
  int64_t first, end;
  std::vector<int> seen;
  Row(int64_t f, int64_t e) : first(f), end(e), seen((size_t)(e - f), 0) {}
  void meet(const char *what, EdgePos e) {
    if ((int64_t)e < first || (int64_t)e >= end) fail(what, end, end - first, (int64_t)e);
    seen[(size_t)(e - first)]++;
  }
  void done(const char *what) {
    for (size_t i = 0; i < seen.size(); ++i)
      if (seen[i] != 1) fail(what, end, end - first, (int64_t)i);
  }
};

int main() {
  const int64_t top = (1ll << 31) - 2;  // the largest m
  long walks = 0;
  for (int64_t end : {top, top - 1, top - 2, top - 3, top - 31, top - 255, top - 2047, (int64_t)100000})
    for (int64_t len : {1, 2, 3, 4, 5, 31, 32, 33, 127, 255, 256, 257, 1023, 2049, 16383, 16384, 16385, 40000}) {
      const EdgePos first = (EdgePos)(end - len), row_end = (EdgePos)end;
      // strided walks: lanes `width` apart, U positions each per step (round_push 32 x 4, bfs_pull's warp
      // scan 32 x 4, msbfs 512 x 4, 32 x 4, 8 x 4 and 1 x 4, ppr_sum 32 x 8 and 64 x 8, bf_multi_relax 8 and 32)
      for (int width : {1, 8, 32, 64, 128, 256, 512})
        for (int U : {1, 4, 8}) {
          Row r(end - len, end);
          for (int lane = 0; lane < width; ++lane)
            for (EdgePos e = first + lane; e < row_end; e += (EdgePos)(U * width))
              for (int u = 0; u < U; ++u)
                if (e + u * width < row_end) r.meet("strided walk", e + u * width);
          r.done("strided walk");
          ++walks;
        }
      // pieces, each taken in shares (round_push) or whole (msbfs, bf_multi)
      for (int piece : {256, 512, 16384})
        for (int parts : {1, 2, 8}) {
          Row r(end - len, end);
          const int n = edge_pieces((int32_t)len, piece);
          if (n != (len + piece - 1) / piece) fail("edge_pieces", end, len, n);
          for (int k = 0; k < n; ++k)
            for (int part = 0; part < parts; ++part) {
              const EdgeSpan s = edge_share(first, row_end, (EdgePos)(k * piece), part, piece / parts);
              if (s.begin > s.end || (int64_t)s.end > end) fail("edge_share", end, len, k);
              for (EdgePos b = s.begin; b < s.end; b += 128)
                for (int lane = 0; lane < 128; ++lane)
                  if (b + lane < s.end) r.meet("edge_share", b + lane);
            }
          r.done("edge_share");
          ++walks;
          Row q(end - len, end);
          for (int k = 0; k < n; ++k) {
            const EdgePos e0 = first + (EdgePos)(k * piece), e1 = edge_end(e0, piece, row_end);
            if ((int64_t)e1 != std::min<int64_t>((int64_t)e0 + piece, end)) fail("edge_end", end, len, (int64_t)e1);
            for (EdgePos e = e0; e < e1; ++e) q.meet("edge_end", e);
          }
          q.done("edge_end");
        }
      // two, then kStep, then kPullScan edges at a time (bfs_pull, k_dense_pull)
      Row r(end - len, end);
      EdgePos e = first;
      for (EdgePos step : {2u, 4u, 32u}) {
        const EdgePos lim = edge_end(e, step, row_end);
        for (; e < lim; ++e) r.meet("scan", e);
      }
      for (; e < row_end; ++e) r.meet("scan", e);
      r.done("scan");
    }
  // a row of all edges, and one that starts at the end
  if (edge_pieces((int32_t)top, 4096) != 524288 || edge_pieces((int32_t)top, 256) != 8388608 || edge_pieces(0, 256) != 0)
    fail("edge_pieces", top, top, 0);
  if (edge_end((EdgePos)top, 2, (EdgePos)top) != (EdgePos)top) fail("edge_end", top, 0, 0);
  std::printf("%ld\n", walks);
}
