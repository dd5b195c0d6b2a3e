// Common parts of the edge kernels: the convolution's forward and first derivatives for path lists that are complete
// over three sets of degrees, with everything about the list compiled in.
//
// A shape is three sets of degrees (x, edge attributes, out) as bit masks.  Its list is every (l1, l2, l3) from the
// sets that satisfies the triangle rule and has an even degree sum, in that order, which is also the order of the
// weight blocks.  The list of compiled shapes is closed (kEdgeShapeMasks); the number of channels is not compiled in.
//
// Teams.  A team of one or more warps of a CTA walks the edges of a row (a destination in the forward, a source in the
// backward kernel); warp t of a team of n owns channels [t, t + 1) * ch / n of every block, and a lane owns CPL of them
// (lanes beyond the warp's channels repeat the last lane's addresses and contribute zeros).
// One lane of the team stages an edge's rows - the whole weight row, the whole gathered node row - with one bulk copy
// each, whatever the number of warps: DRAM sees requests of full rows.
//
// Slices.  Blocks too wide for a team (more than eight warps, or rows that do not fit twice in shared memory) are cut into
// slices of 32 * CPL channels, blockIdx.y their number: a one-warp team walks the rows of its slice, whose pieces, one per
// path and per degree, the lanes copy side by side.  Each slice has its tile counters and its part of dL/dy; the parts are
// summed in order by a second kernel.
//
// Three ways of handing out rows.  Large launches: a team takes tiles of consecutive rows from a counter.  Small launches, in
// which a few tiles per team would leave the chip waiting for the last ones: every CTA has an equal stretch of the edges, up
// to whole rows, and every team of it an equal part of that, whatever the rows; a row that several teams share is summed
// at the end, in the teams' order, through shared memory.  The forward of very few rows: `group` teams of a CTA share a row, each
// a contiguous part of its edges, and the parts are summed in a fixed order through shared memory.  No sum depends
// on which team was first.  A row's sum is one over its own edges, in their order, where tiles are handed out (two edges at a time:
// that of the first, third, ... and that of the others); in a group it is cut by the row's length and `group`; in equal parts it is
// cut where a team's part ends, so by the lengths of other rows too.  So a piece of a graph gives the same rows to the bit where
// both launches hand out tiles, or both share rows in groups of one size (edge_split), and else to rounding.
#pragma once

#include <atomic>

#include "uvu_fast.cuh"
#include "uvu_packets.cuh"
#include "uvu_parts.cuh"

namespace luna {
namespace edgek {

using namespace fastk;

constexpr int kEdgeMaxStages = 4;
constexpr int kEdgeMaxSlices = kTileCounterWords / 2;
constexpr int64_t kPartEdges = 256;          // of a team, at most
constexpr int64_t kPartGathered = 24 << 20;  // bytes
constexpr int64_t kEarlyWeights = 128 << 20;  // bytes, of launches that write dL/dw and start early
constexpr int kEdgeMaxCoefs = 10;  // paths with a degree of zero

// ---- shapes ---------------------------------------------------------------------------------------------------------
constexpr int top_degree(int mask) { return mask >= 8 ? 3 : (mask >= 4 ? 2 : (mask >= 2 ? 1 : 0)); }
template <int MX_, int MY_, int MO_>
struct Shape {
  static constexpr int MX = MX_, MY = MY_, MO = MO_;
  static constexpr bool has(int mask, int l) { return ((mask >> l) & 1) != 0; }
  // components of the degrees below l
  static constexpr int below(int mask, int l) {
    int n = 0;
    for (int a = 0; a < l; ++a)
      if (has(mask, a)) n += 2 * a + 1;
    return n;
  }
  static constexpr int XD = below(MX, 4), YD = below(MY, 4), OD = below(MO, 4);
  static constexpr int xoff(int l) { return below(MX, l); }
  static constexpr int yoff(int l) { return below(MY, l); }
  static constexpr int ooff(int l) { return below(MO, l); }
  static constexpr bool ok(int l1, int l2, int l3) {
    const int lo = l1 > l2 ? l1 - l2 : l2 - l1;
    return has(MX, l1) && has(MY, l2) && has(MO, l3) && l3 >= lo && l3 <= l1 + l2 && (l1 + l2 + l3) % 2 == 0;
  }
  // position of a path's weight block; past-the-end arguments give the number of paths
  static constexpr int rank(int a, int b, int c) {
    int r = 0;
    for (int l1 = 0; l1 < 4; ++l1)
      for (int l2 = 0; l2 < 4; ++l2)
        for (int l3 = 0; l3 < 4; ++l3) {
          if (l1 == a && l2 == b && l3 == c) return r;
          if (ok(l1, l2, l3)) ++r;
        }
    return r;
  }
  static constexpr int paths = rank(-1, -1, -1);
  // A path with a degree of zero couples component by component with one coefficient (edge_diagonal): it has no matrix and
  // no terms.  Position of its coefficient; past-the-end arguments give their number.
  static constexpr bool diagonal(int l1, int l2, int l3) { return l1 == 0 || l2 == 0 || l3 == 0; }
  static constexpr int coff(int a, int b, int c) {
    int n = 0;
    for (int l3 = 0; l3 < 4; ++l3)
      for (int l1 = 0; l1 < 4; ++l1)
        for (int l2 = 0; l2 < 4; ++l2) {
          if (l1 == a && l2 == b && l3 == c) return n;
          if (ok(l1, l2, l3) && diagonal(l1, l2, l3)) ++n;
        }
    return n;
  }
  // the edge's attributes as they are, behind the matrices: every degree at a multiple of four
  static constexpr int ypos(int l) { return l == 3 ? 16 : 4 * l; }
  static constexpr int y_elems = ypos(top_degree(MY)) + 4 * ((2 * top_degree(MY) + 4) / 4);
  // first entry of a path in an edge's coupling-matrix buffer: the entries that some edge attribute reaches, in (i, k)
  // order, paths in (l3, l1, l2) order, every path padded to a multiple of four
  static constexpr int moff(int a, int b, int c) {
    int m = 0;
    for (int l3 = 0; l3 < 4; ++l3)
      for (int l1 = 0; l1 < 4; ++l1)
        for (int l2 = 0; l2 < 4; ++l2) {
          if (!ok(l1, l2, l3)) continue;
          if (l1 == a && l2 == b && l3 == c) return m;
          m += diagonal(l1, l2, l3) ? 0 : (cg_pair_count(l1, l2, l3) + 3) / 4 * 4;
        }
    return m;
  }
  static constexpr int m_total = moff(-1, -1, -1);
  static constexpr int m_rounds = (m_total + 31) / 32;
  static constexpr int m_elems = m_rounds * 32 + y_elems;
  // first coupling term of a path in the term list: (l3, l1, l2) order, every path's terms padded to a multiple of four
  static constexpr int toff(int a, int b, int c) {
    int t = 0;
    for (int l3 = 0; l3 < 4; ++l3)
      for (int l1 = 0; l1 < 4; ++l1)
        for (int l2 = 0; l2 < 4; ++l2) {
          if (!ok(l1, l2, l3)) continue;
          if (l1 == a && l2 == b && l3 == c) return t;
          t += diagonal(l1, l2, l3) ? 0 : (cg_count(l1, l2, l3) + 3) / 4 * 4;
        }
    return t;
  }
  static constexpr int terms = toff(-1, -1, -1);
  static constexpr int LO = top_degree(MO);
};

// The shape with the roles of x and out exchanged; the weight blocks stay where they are.
template <typename S>
struct Transposed : Shape<S::MO, S::MY, S::MX> {
  static constexpr int rank(int a, int b, int c) { return S::rank(c, b, a); }
};

// The compiled shapes: layers with edge harmonics to degree l = 1, 2 or 3 whose features are scalars before (first layers),
// scalars after (last layers) or to degree l on both sides, features to degree 2 that become degree 3, and the single
// vector-vector-scalar coupling.  Every other list, complete or not, runs the table kernels, and one thread per output element
// if its channels are no multiple of 32; among them layers whose features stop below the harmonics.  300 MB of weights, FP32,
// forward / backward: (1, 2, 2) with 64 channels 0.18 / 0.55 ms and with 48 channels 1.16 / 3.97, (1, 3, 3) 0.18 / 0.65 and
// 1.69 / 5.55; beside them (2, 2, 2), compiled, 0.08 / 0.19 and 0.11 / 0.26.
constexpr int kEdgeShapes = 11;
constexpr int kEdgeShapeMasks[kEdgeShapes][3] = {{1, 3, 3},  {1, 7, 7},   {1, 15, 15}, {3, 3, 3},   {7, 7, 7}, {15, 15, 15},
                                                 {7, 15, 15}, {3, 3, 1},  {7, 7, 1},   {15, 15, 1}, {2, 2, 1}};
// Shapes whose kernels are compiled for slices too.  The others have no wide layers in use; theirs run the table kernels.
constexpr bool edge_sliced(int id) { return id >= 3 && id <= 6; }
template <int ID>
using ShapeOf = Shape<kEdgeShapeMasks[ID][0], kEdgeShapeMasks[ID][1], kEdgeShapeMasks[ID][2]>;
// What a launch computes, as far as the choice of its layout goes: one gradient is dL/dy or dL/dw alone, sums are dL/dx, alone or
// with dL/dw.
enum class EdgeUse { kForward, kOneGradient, kSums, kOutputAndWeights, kAllGradients };

// ---- launch arguments, type-erased ------------------------------------------------------------------------------------
struct EdgeForwardArgs {
  const void *x, *y, *w;
  void* out;
  bool accumulate;
};
struct EdgeBackwardArgs {
  const void *x, *y, *w, *g;
  void *gx, *gy, *gw;
  bool acc_x, acc_y, acc_w;
  void* scratch;  // for the slices' parts of gy
  int64_t scratch_bytes;
  void* out;  // with gw alone: the output as well, if not null
};
// The kernels of one (element type, channels per lane, shape), compiled in a file of their own.
template <typename T, int CPL, int ID>
struct EdgeKernels {
  static int forward(const luna_uvu_plan* plan, const DeviceTables& dt, const luna_graph* graph,
                     const EdgeLanes& lanes, const EdgeForwardArgs& a, cudaStream_t stream);
  static int backward(const luna_uvu_plan* plan, const DeviceTables& dt, const luna_graph* graph,
                      const EdgeLanes& lanes, const EdgeBackwardArgs& a, cudaStream_t stream);
  static bool joins_output();  // whether output and gw come in one launch
  // shared memory of a block of the forward kernel, or of the backward kernel of all gradients
  static size_t smem_bytes(const luna_uvu_plan* plan, const EdgeLanes& lanes, bool backward, int max_smem);
};

// ---- how a launch is laid out -----------------------------------------------------------------------------------------
struct EdgeLaunch {
  int warps = 0;   // per CTA
  int stages = 0;  // per team
  int split = 0;   // backward: g in one slot per degree instead of in the stages
  size_t bytes = 0;
  int team_elems = 0;  // of shared memory
};
// Rows shared by `group` teams, or else equal parts of the edges, or else tiles of rows.
struct EdgeSplit {
  int group = 1;
  bool parts = false;
  int64_t blocks = 1;
  int64_t tile_rows = 1;
};

// CTAs that a slice may take: as many as make whole waves of all slices' CTAs, one per SM, with at most 5 % of the SMs idle.
// With a CTA per SM and slice, a CTA's part of a small graph is too short for what it costs to start: degrees (1, 1, 1),
// 27 slices, 22,000 edges, forward / backward 0.37 / 0.78 ms, and 0.23 / 0.55 like this.
inline int slice_ctas(int sm_count, int slices) {
  int best = 1;
  double best_use = 0.0;
  for (int waves = 1; waves <= 4; ++waves) {
    const int ctas = sm_count * waves / slices;
    const double use = static_cast<double>(ctas) * slices / (static_cast<double>(sm_count) * waves);
    if (ctas >= 1 && use > best_use) {
      best = ctas;
      best_use = use;
    }
    if (best_use >= 0.95) break;
  }
  return best;
}

constexpr int kNamedBarriers = 15;  // of a CTA, beside the one of __syncthreads

// Parts of the edges are even to about a row per CTA; what they lose is order: a CTA's rows are its own, so the rows that all
// CTAs gather at a time are spread over the whole graph.  So: as long as a team's part is short, and while the node rows that
// are gathered (`gathered` bytes) stay in L2 whoever reads them.  Groups (`may_group`): while a CTA has three rows
// or fewer, too few for even parts.  The group is a matter of the kernel and of the edges per row, so pieces of such a graph that
// have as many edges per row give the same sums.  Rows and edges
// shared as before (groups of up to eight teams, then tiles) and in parts, forward / all gradients: (2, 2, 2), 64 channels,
// 2,083 nodes of 41 edges 80 / 160 -> 78 / 148 us, 4,000 of 30 98 / 201 -> 90 / 180; 48 channels, 10,001 of 52 290 / 777 -> 258 /
// 711; 32 channels, 4,003 of 52 100 / 202 -> 88 / 176.  With 442 edges a team (64 channels, 20,000 nodes) the two are even, and
// with 64 MB of gathered rows ((3, 3, 3), 128 channels, 8,000 nodes) parts lose: forward 0.98 -> 1.27 ms.
inline bool few_rows(int64_t rows, int ctas) { return rows <= 3 * static_cast<int64_t>(ctas); }
inline bool shares_rows(int64_t rows, int64_t edges, int ctas) { return few_rows(rows, ctas) && edges >= 4 * rows; }
inline EdgeSplit edge_split(int64_t rows, int64_t edges, int sm_count, int teams, int team_warps, int64_t wanted_tile,
                            int at_once, int64_t gathered, bool may_group) {
  EdgeSplit s;
  const int64_t all = static_cast<int64_t>(sm_count) * teams;
  const double degree = static_cast<double>(edges) / static_cast<double>(std::max<int64_t>(rows, 1));
  const bool few = may_group && few_rows(rows, sm_count);
  if (may_group && shares_rows(rows, edges, sm_count)) {
    int want = 8;  // and at least two steps of a team in a part
    while (want > 1 && (want > teams || teams % want != 0 || degree < 2.0 * at_once * want)) want /= 2;
    if (want > 1 && team_warps > 1 && teams + teams / want > kNamedBarriers) want = 1;
    s.group = want;
  }
  if (s.group > 1 || (!few && edges <= kPartEdges * all && gathered <= kPartGathered && degree >= 4.0)) {
    s.parts = s.group == 1;
    s.blocks = std::max<int64_t>(1, std::min<int64_t>(sm_count, rows));
    return s;
  }
  const int64_t tile_edges = tile_edges_for(edges, all, wanted_tile);
  s.tile_rows = std::min<int64_t>(1 << 20, std::max<int64_t>(1, static_cast<int64_t>(tile_edges / std::max(degree, 1e-3) + 0.5)));
  const int64_t tiles = ceil_div(std::max<int64_t>(rows, 1), s.tile_rows);
  s.blocks = std::max<int64_t>(1, std::min<int64_t>(sm_count, ceil_div(tiles, teams)));
  return s;
}

// ---- coupling patterns --------------------------------------------------------------------------------------------------
// Terms of a pattern are sorted by (i, k, j).  The end of the row of term t0, and the position of term t's (i, k) among
// the pattern's distinct ones.
template <typename PT>
__host__ __device__ constexpr int edge_row_end(int t0) {
  int t = t0;
  while (t < PT::n && PT::t[t].i == PT::t[t0].i) ++t;
  return t;
}
template <typename PT>
__host__ __device__ constexpr bool edge_new_entry(int t) {
  return t == 0 || PT::t[t].i != PT::t[t - 1].i || PT::t[t].k != PT::t[t - 1].k;
}
template <typename PT>
__host__ __device__ constexpr bool edge_new_row(int t) {
  return t == 0 || PT::t[t].i != PT::t[t - 1].i;
}
template <typename PT>
__host__ __device__ constexpr int edge_entry(int t) {
  int e = -1;
  for (int q = 0; q <= t; ++q) e += edge_new_entry<PT>(q) ? 1 : 0;
  return e;
}

// ---- device helpers ---------------------------------------------------------------------------------------------------
// Where element `a` of a slice's row of blocks (the degrees of `mask`, `ch` channels each) lies in the whole row, whose
// blocks have `row_ch` channels and in which the slice begins with channel `first`.
template <typename S>
__device__ __forceinline__ int slice_element(int mask, int a, int ch, int row_ch, int first) {
  int at = a;
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    if (!S::has(mask, l)) continue;
    const int begin = S::below(mask, l), d = 2 * l + 1;
    if (a >= ch * begin && a < ch * (begin + d)) at = a + (row_ch - ch) * begin + first * d;
  }
  return at;
}
__device__ __forceinline__ void named_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Synchronises the warps of a team (its own barrier, unless it is one warp).
__device__ __forceinline__ void team_sync(int team_warps, int team_id) {
  if (team_warps == 1)
    __syncwarp();
  else
    named_barrier(1 + team_id, team_warps * 32);
}
// The first rows that begin at `bound` or after it, one search in each half of the warp, and where they begin.  A guess is
// looked up with its neighbours, 16 entries at a time, and mended by what they say; after three of those the interval is halved
// (rows of very uneven length).  Not inlined: the searches of all kernels would be a sixth of the library.
struct FoundRow {
  int row, begin;
};
static __device__ __noinline__ FoundRow part_rows(const int* rowptr, int rows, int bound, float guess, float rows_per_edge, int lane) {
  const int place = lane & 15, shift = lane & 16;
  int lo = 0, hi = rows;  // of the answer
  FoundRow found{rows, 0};
  bool done = false;
#pragma unroll 1
  for (int step = 0; __any_sync(0xffffffffu, !done); ++step) {
    const int wanted = step < 3 ? static_cast<int>(fminf(fmaxf(guess, 0.0f), static_cast<float>(rows))) : lo + (hi - lo) / 2;
    const int base = max(lo, min(wanted - 8, hi - 15));
    const int at = base + place, value = at <= hi ? rowptr[at] : 0x7fffffff;
    const int below = __popc((__ballot_sync(0xffffffffu, value < bound) >> shift) & 0xffffu);
    const int first = __shfl_sync(0xffffffffu, value, shift), last = __shfl_sync(0xffffffffu, value, shift + 15);
    const int here = __shfl_sync(0xffffffffu, value, shift + min(below, 15));
    if (done) continue;
    if (below < 16 && (below > 0 || base == lo)) {
      found = FoundRow{base + below, here};
      done = true;
    } else if (below == 16) {
      lo = base + 16;
      guess = static_cast<float>(lo) + static_cast<float>(bound - last) * rows_per_edge;
    } else {
      hi = base;
      guess = static_cast<float>(hi) + static_cast<float>(bound - first) * rows_per_edge;
    }
  }
  return found;
}
__device__ __forceinline__ TeamPart team_part(const int* __restrict__ rowptr, int64_t rows, int64_t edges, float rows_per_edge,
                                              int team, int teams, int lane) {
  TeamPart p;
  const int all = static_cast<int>(rows), first_half = lane < 16;
  // the CTA: the rows that begin in its stretch of the edges
  const int from = static_cast<int>(edges * blockIdx.x / gridDim.x), to = static_cast<int>(edges * (blockIdx.x + 1) / gridDim.x);
  const int bound = first_half ? from : to;
  FoundRow f = part_rows(rowptr, all, bound, static_cast<float>(bound) * rows_per_edge, rows_per_edge, lane);
  const int r0 = __shfl_sync(0xffffffffu, f.row, 0), p0 = __shfl_sync(0xffffffffu, f.begin, 0);
  int r1 = __shfl_sync(0xffffffffu, f.row, 16), p1 = __shfl_sync(0xffffffffu, f.begin, 16);
  if (blockIdx.x + 1 == gridDim.x) {  // rows without edges at the end
    r1 = all;
    p1 = static_cast<int>(edges);
  }
  p.cta_pos = p0;
  p.cta_edges = p1 - p0;
  p.pos = part_begin(p0, p.cta_edges, team, teams);
  p.end = part_begin(p0, p.cta_edges, team + 1, teams);
  const int mine = first_half ? p.pos : p.end;
  const float per_edge = static_cast<float>(r1 - r0) / static_cast<float>(max(p.cta_edges, 1));
  f = part_rows(rowptr, all, mine, static_cast<float>(r0) + static_cast<float>(mine - p0) * per_edge, per_edge, lane);
  p.n = __shfl_sync(0xffffffffu, f.row, 0);
  p.n_hi = __shfl_sync(0xffffffffu, f.row, 16);
  p.joined = p.pos < p.end && __shfl_sync(0xffffffffu, f.begin, 0) > p.pos;
  p.open = p.pos < p.end && __shfl_sync(0xffffffffu, f.begin, 16) > p.end;
  if (team + 1 == teams) {
    p.n_hi = r1;
    p.open = 0;
  }
  if (p.joined) --p.n;
  return p;
}
// The end of a launch in equal parts: rows that a team joined and ended get the earlier teams' sums, which lie `stride` elements
// apart in shared memory, in the teams' order; element a of row n is at element(n, a).  By all threads of the CTA, whose barriers
// are the first thing: what a row's elements cost is a trip to memory and back, so they all go at a time.  As the work of the
// joining team alone, one element of a lane after the other, it was up to half of a small launch.  64 channels: (2, 2, 2), all
// gradients of 4,800 edges 27 -> 19 us, of 20,000 41 -> 37, forward of 20,000 25 -> 19; (0, 3, 3), forward of 20,000 25 -> 13.
template <typename T, typename F>
__device__ __forceinline__ void merge_parts(TeamPart* kept, int teams, const int* __restrict__ rowptr, const T* parts, size_t stride,
                                            int elements, F&& element) {
  __syncthreads();
  if (threadIdx.x < 32) {
    const int team = static_cast<int>(threadIdx.x);
    TeamPart p{};
    if (team < teams) p = kept[team];
    const bool closes = team < teams && p.closes();
    unsigned earlier = 0u;  // the teams before this one, back to where the row begins, that have any of its edges
    if (closes) {
      const int row_begin = rowptr[p.n];
      for (int q = team - 1, end = p.pos; q >= 0; --q) {
        const int begin = part_begin(p.cta_pos, p.cta_edges, q, teams);
        if (begin < end) earlier |= 1u << q;
        if (begin <= row_begin) break;
        end = begin;
      }
    }
    const unsigned closing = __ballot_sync(0xffffffffu, closes);
    __syncwarp();
    if (closes) {  // the rows side by side
      TeamPart& to = kept[__popc(closing & ((1u << team) - 1u))];
      to.n = p.n;
      to.joined = static_cast<int>(earlier);
    }
    if (team == 0) kept[0].open = __popc(closing);
  }
  __syncthreads();
  const int total = kept[0].open * elements;
#pragma unroll 2
  for (int i = static_cast<int>(threadIdx.x); i < total; i += static_cast<int>(blockDim.x)) {
    const int row = i / elements, a = i - row * elements;
    T* const to = element(kept[row].n, a);
    T sum = *to;
    for (unsigned left = static_cast<unsigned>(kept[row].joined); left != 0u;) {
      T part[4];
      int count = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (left == 0u) break;
        part[k] = parts[(__ffs(static_cast<int>(left)) - 1) * stride + a];
        left &= left - 1u;
        ++count;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < count) sum += part[k];
    }
    *to = sum;
  }
}
// After one wait has run out the kernel keeps its control flow (other warps may be waiting for it at a barrier), writes
// nothing more to rely on, and stops spending time on waits.
constexpr uint32_t kWaitAfterFailure = 64;
__device__ __forceinline__ bool edge_wait(uint64_t* bar, uint32_t parity, bool alive) {
  const uint32_t limit = alive ? kWaitLimit : kWaitAfterFailure;
#pragma unroll 1
  for (uint32_t spin = 0; spin < limit; ++spin)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void bulk_reduce_add_s2g(float* dst, const float* src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_reduce_add_s2g(double* dst, const double* src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;" ::"l"(dst),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}
// Four consecutive entries of a 16-byte aligned table; every lane reads the same address.
template <typename T>
__device__ __forceinline__ void edge_load_four(const T* p, T* out) {
  constexpr int per = 16 / static_cast<int>(sizeof(T));
#pragma unroll
  for (int v = 0; v < 4 / per; ++v) {
    const Vec<T, per> t = reinterpret_cast<const Vec<T, per>*>(p)[v];
#pragma unroll
    for (int c = 0; c < per; ++c) out[v * per + c] = t.a[c];
  }
}

// The 2l + 1 attributes of degree l out of an edge's matrix buffer.
template <typename S, int l, typename T>
__device__ __forceinline__ void edge_attributes(const T* buffer, T* y) {
#pragma unroll
  for (int q = 0; q < (2 * l + 4) / 4; ++q) edge_load_four<T>(buffer + S::m_rounds * 32 + S::ypos(l) + 4 * q, y + 4 * q);
}

// A lane's channels.  Packet q of a lane holds PK::W consecutive channels, and the packets of the warp's lanes lie side
// by side: packet q of lane l starts at channel  own + q * W * lanes  with  own = first + W * l.
// Weights then arrive as ready-made packets, and the scalar loads that assemble the packets of a node row (channel-
// major, 2l + 1 components) meet two-way bank conflicts at most (with four consecutive channels per lane: four-way).
// Spread packets hold channels  own + (q * W + c) * lanes  with  own = first + l:  no conflicts, and a load for every weight.
// Pairs are spread (edge_spread) where an edge's gathered row has at least twice as many components as its weight row has paths:
// first layers backward, which gather g, and last layers forward, which gather x.  128 channels: (0, 3, 3), 1.05 M edges, all
// gradients 1,169 -> 1,090 us, dL/dx with dL/dw 1,002 -> 947; (3, 3, 0), 0.4 M edges, forward 272 -> 244; (2, 2, 0) 182 -> 165.
// Elsewhere the further loads of weights cost what the conflicts did: (2, 2, 2) and (2, 3, 3) within 2 %, (2, 2, 2) with 96
// channels, dL/dw 526 -> 567.
constexpr bool edge_spread(int gathered, int paths) { return gathered >= 2 * paths; }
template <typename T, int CPL, bool SPREAD>
struct EdgePacket : PkT<T, CPL, UsePairs<T, CPL>::value> {
  static constexpr bool spread = SPREAD || PkT<T, CPL, UsePairs<T, CPL>::value>::spread;
};
template <typename PK>
__device__ __forceinline__ int lane_channel(int q, int c, int lanes) {
  return PK::spread ? (q * PK::W + c) * lanes : q * PK::W * lanes + c;
}
template <typename PK>
__device__ __forceinline__ int lane_first(int lane) {
  return PK::spread ? lane : PK::W * lane;
}
template <typename PK, typename T>
__device__ __forceinline__ void lane_load(const T* p, int lanes, typename PK::V* out) {
#pragma unroll
  for (int q = 0; q < PK::NP; ++q) {
    if constexpr (PK::W == 2 && !PK::spread) {
      out[q].v = *reinterpret_cast<const unsigned long long*>(p + q * PK::W * lanes);
    } else {
      T vals[PK::W];
#pragma unroll
      for (int c = 0; c < PK::W; ++c) vals[c] = p[lane_channel<PK>(q, c, lanes)];
      out[q] = make_packet(vals, typename PK::V{});
    }
  }
}
template <typename PK, typename T>
__device__ __forceinline__ void lane_store(T* p, int lanes, const typename PK::V* in) {
#pragma unroll
  for (int q = 0; q < PK::NP; ++q) {
    if constexpr (PK::W == 2 && !PK::spread) {
      *reinterpret_cast<unsigned long long*>(p + q * PK::W * lanes) = in[q].v;
    } else {
      T vals[PK::W];
      split_packet(in[q], vals);
#pragma unroll
      for (int c = 0; c < PK::W; ++c) p[lane_channel<PK>(q, c, lanes)] = vals[c];
    }
  }
}
// Components of a node row's block of D components per channel -> packets [component][packet]; p: the block plus
// own * D, `lanes` as above.  Scalar loads on purpose: the two halves then land in the pair's registers, while halves
// taken from vector loads are put together again in front of every packed instruction that uses the pair (measured on
// the 128-channel degree-(2,3,3) backward: 18.9 ms against 11.4).
template <typename PK, typename T, int D>
__device__ __forceinline__ void lane_load_block(const T* p, int lanes, typename PK::V* out) {
  using V = typename PK::V;
#pragma unroll
  for (int q = 0; q < PK::NP; ++q)
#pragma unroll
    for (int i = 0; i < D; ++i) {
      T vals[PK::W];
#pragma unroll
      for (int c = 0; c < PK::W; ++c) vals[c] = p[lane_channel<PK>(q, c, lanes) * D + i];
      out[i * PK::NP + q] = make_packet(vals, V{});
    }
}
// Packets [component][packet] to such a block in memory, added to what is there if `add`.
template <typename PK, typename T, int D>
__device__ __forceinline__ void lane_store_block(T* p, int lanes, const typename PK::V* in, bool add) {
#pragma unroll
  for (int q = 0; q < PK::NP; ++q) {
    T row[PK::W * D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
      T vals[PK::W];
      split_packet(in[i * PK::NP + q], vals);
#pragma unroll
      for (int c = 0; c < PK::W; ++c) row[c * D + i] = vals[c];
    }
    constexpr int together = PK::spread ? 1 : PK::W;  // channels side by side
#pragma unroll
    for (int c = 0; c < PK::W; c += together) {
      T *to = p + lane_channel<PK>(q, c, lanes) * D, *from = row + c * D;
      if (add) {
        T old[together * D];
        load_vectors<T, together, D>(to, old);
#pragma unroll
        for (int a = 0; a < together * D; ++a) from[a] += old[a];
      }
      store_vectors<T, together, D>(to, from);
    }
  }
}

// The program that turns an edge's attributes, one per lane, into its coupling matrices: entry m is a_m y[ja] + b_m
// y[jb].  Entries are made in rounds of 32, one to a lane; `team_warps` warps that share the
// matrices take turns.  The forward's teams do, which leaves FP64, degrees (2, 3, 3), 128 channels room for four teams instead of
// three: 0.4 M edges 1.55 -> 1.40 ms.  The backward's warps have matrices of their own: shared ones cost it a barrier an edge, or
// the order of events (all gradients of the same case 4.31 -> 4.57).  An entry made of one attribute only takes kNoAttribute as its second, a lane
// that holds no attribute but zero: with any attribute in its place 0 times an infinite one would make the entry NaN.
constexpr int kNoAttribute = 31;
// Where lane j stores attribute j of the edge, behind the matrices.
template <typename S>
__device__ __forceinline__ int attribute_position(int j) {
  int at = 0;
#pragma unroll
  for (int l = 0; l < 4; ++l)
    if (S::has(S::MY, l) && j >= S::yoff(l)) at = S::m_rounds * 32 + S::ypos(l) + j - S::yoff(l);
  return at;
}
template <typename T, typename S>
struct MatrixProgram {
  static_assert(S::YD <= kNoAttribute, "one lane is left without an attribute");
  T a[S::m_rounds + 1], b[S::m_rounds + 1];
  unsigned j[(S::m_rounds + 2) / 2];  // two attribute indices of 8 bits per round
  int own;                            // where this lane's attribute goes
  __device__ __forceinline__ void load(const T* coefficients, const unsigned short* attributes, int lane, int member, int team_warps) {
    own = attribute_position<S>(lane);
#pragma unroll
    for (int r = 0; r < (S::m_rounds + 1) / 2; ++r) j[r] = 0u;
#pragma unroll
    for (int r = 0; r < S::m_rounds; ++r) {
      const int m = (r * team_warps + member) * 32 + lane;
      a[r] = m < S::m_total ? coefficients[m] : T(0);
      b[r] = m < S::m_total ? coefficients[S::m_total + m] : T(0);
      j[r / 2] |= (m < S::m_total ? static_cast<unsigned>(attributes[m]) : 0u) << (16 * (r % 2));
    }
  }
  __device__ __forceinline__ void run(T y, T* to, int lane, int member, int team_warps) const {
#pragma unroll
    for (int r = 0; r < S::m_rounds; ++r) {
      const int round = r * team_warps + member;
      if (round >= S::m_rounds) break;  // never with one warp
      const T ya = __shfl_sync(0xffffffffu, y, static_cast<int>((j[r / 2] >> (16 * (r % 2))) & 255u));
      const T yb = __shfl_sync(0xffffffffu, y, static_cast<int>((j[r / 2] >> (16 * (r % 2) + 8)) & 255u));
      to[round * 32 + lane] = fma(b[r], yb, a[r] * ya);
    }
    if (member == 0 && lane < S::YD) to[own] = y;
  }
};

// The same for two edges at a time, one to each half of the warp: place is the lane's in its half, y and the buffer are the
// half's.
template <typename T, typename S>
struct HalfMatrixProgram {
  static constexpr int rounds = 2 * S::m_rounds;
  T a[rounds + 1], b[rounds + 1];
  unsigned j[(rounds + 2) / 2];
  int own;
  __device__ __forceinline__ void load(const T* coefficients, const unsigned short* attributes, int place) {
    own = attribute_position<S>(place);
#pragma unroll
    for (int r = 0; r < (rounds + 1) / 2; ++r) j[r] = 0u;
#pragma unroll
    for (int r = 0; r < rounds; ++r) {
      const int m = r * 16 + place;
      a[r] = m < S::m_total ? coefficients[m] : T(0);
      b[r] = m < S::m_total ? coefficients[S::m_total + m] : T(0);
      j[r / 2] |= (m < S::m_total ? static_cast<unsigned>(attributes[m]) : 0u) << (16 * (r % 2));
    }
  }
  __device__ __forceinline__ void run(T y, T* to, int place) const {
#pragma unroll
    for (int r = 0; r < rounds; ++r) {
      const unsigned ja = (j[r / 2] >> (16 * (r % 2))) & 255u, jb = (j[r / 2] >> (16 * (r % 2) + 8)) & 255u;
      const T ya = __shfl_sync(0xffffffffu, y, static_cast<int>(ja & 15u), 16);
      T yb = __shfl_sync(0xffffffffu, y, static_cast<int>(jb & 15u), 16);
      if (S::YD == 16 && jb == kNoAttribute) yb = T(0);  // else the half's last lane holds no attribute
      to[r * 16 + place] = fma(b[r], yb, a[r] * ya);
    }
    if (place < S::YD) to[own] = y;
  }
};

// Warps per CTA by the registers a lane is going to need (an estimate from the state it keeps): the launch bound caps
// the registers at 65,536 / threads.  slack: by how much the estimate is too high.
__host__ __device__ constexpr int warps_for(int regs, int slack = 0) {
  return regs <= 60 ? 24 : (regs <= 120 + slack ? 16 : (regs <= 150 + slack ? 12 : 8));
}
// Of the backward kernels, whose estimate has room for coupling matrices in it: lists without any need less, dL/dy alone, which
// keeps neither gradients nor matrices, least.  Twelve warps and sixteen, 0.4 M edges: dL/dy alone, 128 channels, (3, 3, 0) 248 ->
// 215 us, FP64 (0, 3, 3), 64 channels 334 -> 281; dL/dx with dL/dw, (2, 2, 0), 128 channels, 0.8 M edges 640 -> 555; output with
// dL/dw, (0, 2, 2), 608 -> 537.  Above these limits it loses: all gradients of (2, 2, 0), 128 channels 716 -> 800.  So it does with two
// edges at a time, which have no slack: (2, 2, 0), 64 channels, 0.26 M edges, dL/dx with dL/dw 116 -> 193 us, FP64, 48 channels, 60,000
// edges 46 -> 54; and FP32 dL/dy alone with idle lanes (not `full`): (0, 3, 3), 80 channels, 600 and 15,000 edges +34 and +9 %.
template <typename T, typename S>
constexpr int slack_for(bool with_sums, bool full) {
  if (S::m_total != 0) return 0;
  return with_sums ? 10 : (full || sizeof(T) == 8 ? 35 : 0);
}

// Attributes a kernel needs set once per device, not on every launch.
struct KernelSetup {
  std::atomic<uint64_t> done{0};
  int once(const void* kernel, int max_smem) {
    int device = 0;
    LUNA_CUDA_CHECK(cudaGetDevice(&device));
    const uint64_t bit = 1ull << (device & 63);
    if (device < 64 && (done.load(std::memory_order_acquire) & bit)) return LUNA_OK;
    LUNA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    LUNA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (device < 64) done.fetch_or(bit, std::memory_order_release);
    return LUNA_OK;
  }
};

}  // namespace edgek
}  // namespace luna
