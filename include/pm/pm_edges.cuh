// pm_edges.cuh -- arithmetic on edge positions, for host and device.
//
// A handle holds up to 2^31 - 2 edges, so an edge position fits an int32 but a
// position plus a stride need not: kernels that step through a row carry
// positions as EdgePos, where a position plus anything a kernel adds to it
// (less than 2^31) is exact, and compare them there.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define PM_EDGE_FN __host__ __device__ __forceinline__
#else
#define PM_EDGE_FN inline
#endif

namespace pm {

using EdgePos = uint32_t;

struct EdgeSpan {
  EdgePos begin, end;  // begin <= end
};

// The end of at most len edges from e on in a row that ends at row_end.
PM_EDGE_FN EdgePos edge_end(EdgePos e, EdgePos len, EdgePos row_end) {
  const EdgePos end = e + len;
  return end < row_end ? end : row_end;
}

// Share `part` of part_len edges of the piece that starts `at` edges into the
// row [first, row_end); empty past the row's end.
PM_EDGE_FN EdgeSpan edge_share(EdgePos first, EdgePos row_end, EdgePos at, EdgePos part, EdgePos part_len) {
  EdgePos begin = first + at + part * part_len;
  if (begin > row_end) begin = row_end;
  return EdgeSpan{begin, edge_end(begin, part_len, row_end)};
}

// Pieces of piece edges that a row of deg edges is cut into.
PM_EDGE_FN int32_t edge_pieces(int32_t deg, int32_t piece) { return deg / piece + (deg % piece != 0); }

}  // namespace pm
