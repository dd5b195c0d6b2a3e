// Equal parts of a launch's edges, of which uvu_edge.cuh says when and how they are cut: what a team has, and where its rows end.
// Integer arithmetic that compiles for the host as well, where a test can see every index into the row table.
#pragma once

#ifdef __CUDACC__
#define LUNA_PARTS_INLINE __host__ __device__ __forceinline__
#else
#define LUNA_PARTS_INLINE inline
#endif

namespace luna {
namespace edgek {

// A team's part of a launch: its edges [pos, end), the rows [n, n_hi) that they are of, and whether the first of these rows began
// in an earlier team's part (joined) and the last one goes on in the next team's (open).  A part without rows may have n at the
// number of rows, whose entry is the row table's last.
struct TeamPart {
  int n, n_hi, pos, end;
  int cta_pos, cta_edges;  // the CTA's edges
  int joined, open;
  // the row that the next team goes on with, or -1
  LUNA_PARTS_INLINE int open_row() const { return open ? n_hi - 1 : -1; }
  // whether the first row began earlier and ends here
  LUNA_PARTS_INLINE bool closes() const { return joined && n != open_row(); }
};
LUNA_PARTS_INLINE int part_begin(int cta_pos, int cta_edges, int team, int teams) {
  return cta_pos + static_cast<int>(static_cast<unsigned>(cta_edges) * static_cast<unsigned>(team) / static_cast<unsigned>(teams));
}
// Where, up to `end`, the edges of row n end, the first of rows [n, n_hi); without rows, `end`: the table need not have an entry
// behind n's.
template <typename Rows>
LUNA_PARTS_INLINE int first_row_end(const Rows& rowptr, int n, int n_hi, int end) {
  if (n >= n_hi) return end;
  const int row_end = rowptr[n + 1];
  return row_end < end ? row_end : end;
}

}  // namespace edgek
}  // namespace luna
