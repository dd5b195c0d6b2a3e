// Which plans the edge kernels serve, the tables they read, and the choice of the compiled instance.
#include "uvu_pair_bwd.cuh"

#include <cmath>
#include <utility>

namespace luna {
namespace edgek {

namespace {

template <typename T, int CPL, int... ID>
int registers_of(int shape, EdgeUse use, std::integer_sequence<int, ID...>) {
  int found = 0;
  ((found = shape == ID ? registers_of<T, CPL, ShapeOf<ID>>(use) : found), ...);
  return found;
}
int registers_of(const luna_uvu_plan* plan, int shape, EdgeUse use, int cpl) {
  constexpr std::make_integer_sequence<int, kEdgeShapes> all{};
  if (plan->dtype == LUNA_F64)
    return cpl == 3 ? registers_of<double, 3>(shape, use, all)
                    : (cpl == 2 ? registers_of<double, 2>(shape, use, all) : registers_of<double, 1>(shape, use, all));
  if (cpl >= 3) return cpl == 4 ? registers_of<float, 4>(shape, use, all) : registers_of<float, 3>(shape, use, all);
  return cpl == 2 ? registers_of<float, 2>(shape, use, all) : registers_of<float, 1>(shape, use, all);
}

template <typename T, int CPL, int... ID>
bool paired(int shape, EdgeUse use, std::integer_sequence<int, ID...>) {
  bool found = false;
  ((found = found || (shape == ID && edge_paired<T, CPL, ID>(use))), ...);
  return found;
}
bool paired(const luna_uvu_plan* plan, int shape, EdgeUse use, int cpl) {
  constexpr std::make_integer_sequence<int, kEdgeShapes> all{};
  if (plan->dtype == LUNA_F64)
    return cpl == 1 ? paired<double, 1>(shape, use, all)
                    : (cpl == 2 ? paired<double, 2>(shape, use, all) : cpl == 3 && paired<double, 3>(shape, use, all));
  if (cpl >= 3) return cpl == 4 ? paired<float, 4>(shape, use, all) : cpl == 3 && paired<float, 3>(shape, use, all);
  return cpl == 1 ? paired<float, 1>(shape, use, all) : cpl == 2 && paired<float, 2>(shape, use, all);
}

// Whether one edge at a time with three channels per lane is compiled.
template <typename T, int... ID>
bool three(int shape, EdgeUse use, std::integer_sequence<int, ID...>) {
  bool found = false;
  ((found = found || (shape == ID && edge_alone<T, 3, ID>(use))), ...);
  return found;
}
bool three(const luna_uvu_plan* plan, int shape, EdgeUse use) {
  constexpr std::make_integer_sequence<int, kEdgeShapes> all{};
  return plan->dtype == LUNA_F64 ? three<double>(shape, use, all) : three<float>(shape, use, all);
}

// Coupling-matrix entries of the shape.
template <int... ID>
int matrix_entries(int shape, std::integer_sequence<int, ID...>) {
  int found = 0;
  ((found = shape == ID ? ShapeOf<ID>::m_total : found), ...);
  return found;
}

// Channels per lane and warps per team, or slices for blocks that no team takes.  A warp's pass over an edge costs about one
// unit of fixed work plus one per channel of a lane, so 40 channels take one warp with two channels on 20 lanes, 96 one warp
// with three on all of them.  A kernel that spills counts half as much again: degrees (3, 3, 3) with the most channels
// per lane, all gradients, which then spills 176 (FP32) or 276 bytes and more.  300 MB of weights, FP64: 224 channels with one
// channel per lane 0.83 -> 0.54 ms; FP32: 128 channels 0.33 -> 0.27 with two (2.6 GB: 2.03 -> 1.54), 256 channels 0.39 -> 0.30.
// The forward with an estimate of more than 190 registers counts a third more: FP32 (3, 3, 3), 128 channels, two warps with two channels
// per lane instead of one with four, 0.2 M edges 620 -> 583 us, 24,000 edges 134 -> 115; 256 channels, 60,000 edges, 420 -> 398.  Not where
// two channels would leave lanes idle: 80 channels, 24 nodes 18.6 -> 25.7 us, 60,000 edges 158 -> 167; 160, five warps with one channel
// instead of two with four, 27 -> 61 and 292 -> 311.  (FP64 with 128 channels would lose by one per lane, 867 -> 972, and at a third more
// the choice stays at two.)
// Three channels per lane, where four or two left a quarter of the lanes idle.  96 channels, forward / all gradients / dL/dy / dL/dw,
// FP32: (2, 2, 2), 0.4 M edges 364 / 958 / 465 / 520 -> 323 / 759 / 426 / 434 us; (2, 3, 3), 0.4 M edges 653 / 1,611 / 852 / 922 ->
// 550 / 1,439 / 790 / 718; FP64, two warps with two and one with three: (2, 2, 2), 0.2 M edges 361 / 1,050 / 566 / 567 -> 332 /
// 763 / 426 / 450; (0, 1, 1), 0.4 M edges 217 / 580 / 408 / 348 -> 128 / 351 / 185 / 207.  It is not taken where its state is far above
// the registers (FP64, (3, 3, 3), all gradients of 0.12 M edges 1.96 -> 3.27 ms), for more than two warps, for slices, and for two FP32
// warps with long coupling matrices: 192 channels, forward / dL/dy (3, 3, 3) 408 / 523 -> 486 / 556 us, (2, 3, 3) 466 / 698 -> 495 /
// 758, but (0, 2, 2) 332 / 560 -> 246 / 398.  Nor for two FP64 warps of estimates above 220: 192 channels, 60,000 edges, (3, 3, 3), dL/dy /
// dL/dw 796 / 955 -> 843 / 1,022 us, (2, 3, 3), dL/dx with dL/dw 697 -> 760; below, (2, 3, 3), dL/dy / dL/dw 562 / 650 -> 523 / 559.
// ch / 16 channels on each of a half warp's 16 lanes, two edges at a time, where that is compiled (edge_paired).  48 channels, one edge
// on 24 lanes and two edges with three channels per lane, 0.8 M edges: (1, 1, 1) 192 / 576 / 340 / 393 -> 165 / 352 / 194 / 252; (0, 3, 3)
// 260 / 642 / 359 / 432 -> 187 / 463 / 252 / 287; (2, 2, 2), 0.52 M edges, 274 / 715 / 378 / 427 -> 260 / 683 / 301 / 301.
// The forward of few rows, whose teams share them (`few`), keeps the layout with the shorter way through an edge: its smallest graphs wait
// for that.  24 / 100 / 300 / 440 nodes of 30 edges, 48 channels on 24 lanes, one edge, and three per lane, two edges: (2, 2, 2)
// 7.0 / 8.0 / 13.9 / 16.4 and 7.6 / 8.6 / 10.8 / 12.2 us, (0, 3, 3) 5.4 / 6.0 / 10.2 / 11.2 and 6.5 / 7.2 / 8.1 / 8.4.  FP64 with coupling
// matrices, 96 channels, two warps with two channels per lane and one with three: (2, 2, 2) 15.6 / 20.2 / 26.6 / 31.9 and 17.3 / 22.5 /
// 26.5 / 30.7.
EdgeLanes choose_lanes(const luna_uvu_plan* plan, int shape, EdgeUse use, bool sliced, bool few = false) {
  const int ch = plan->edge.ch, elem = plan->dtype == LUNA_F64 ? 8 : 4;
  // one team with two stages must fit an SM's shared memory in either direction
  const size_t room = 200 * 1024, W = static_cast<size_t>(plan->W) * elem, X = static_cast<size_t>(plan->X) * elem,
               O = static_cast<size_t>(plan->O) * elem;
  const size_t rows = std::max(std::max(2 * W + O, 2 * (W + X)), std::max(X, O));
  EdgeLanes best;
  double best_cost = 0.0;
  for (int cpl = plan->dtype == LUNA_F64 ? 3 : 4; cpl >= 1; --cpl) {
    if (plan->tuning.lane_channels > 0 && cpl != plan->tuning.lane_channels) continue;
    const int parts = (ch + 32 * cpl - 1) / (32 * cpl);
    if (sliced ? ch % (32 * cpl) != 0 || parts > kEdgeMaxSlices
               : parts > capped_warps(plan->tuning, 8) || ch % (parts * cpl) != 0 || rows + parts * 8192 > room)
      continue;
    const int registers = registers_of(plan, shape, use, cpl);
    if (cpl == 3 && few && elem == 8 && matrix_entries(shape, std::make_integer_sequence<int, kEdgeShapes>{}) > 0) continue;
    if (cpl == 3 && (sliced || parts > 2 || !three(plan, shape, use) ||
                     (parts == 2 && (elem == 8 ? registers > 220 : matrix_entries(shape, std::make_integer_sequence<int, kEdgeShapes>{}) > 64))))
      continue;
    const double crowded = (use == EdgeUse::kAllGradients || cpl == 3) && registers > 255 ? 1.5
                           : use == EdgeUse::kForward && registers > 190 && (elem == 8 || ch % 64 == 0) ? 1.3
                                                                                                         : 1.0;
    const double cost = parts * (1 + cpl) * crowded;
    if (best.cpl != 0 && cost >= best_cost) continue;
    best_cost = cost;
    best = sliced ? EdgeLanes{cpl, 1, parts} : EdgeLanes{cpl, parts, 1};
  }
  const int half = ch / 16;
  if (!sliced && !(few && half == 3) && ch % 16 == 0 && (plan->tuning.lane_channels == 0 || plan->tuning.lane_channels == half) &&
      paired(plan, shape, use, half))
    return EdgeLanes{half, 1, 1, 2};
  return best;
}

// Exchanging x and out turns the pattern of a coupling into that of the exchanged degrees.
template <int L1, int L2, int L3>
constexpr bool pattern_transposes() {
  using P = CgPattern<L1, L2, L3>;
  using Q = CgPattern<L3, L2, L1>;
  if (P::n != Q::n) return false;
  for (int t = 0; t < P::n; ++t) {
    bool found = false;
    for (int u = 0; u < Q::n; ++u) found = found || (P::t[t].i == Q::t[u].k && P::t[t].j == Q::t[u].j && P::t[t].k == Q::t[u].i);
    if (!found) return false;
  }
  return true;
}
template <int... I>
constexpr bool patterns_transpose(std::integer_sequence<int, I...>) {
  return (pattern_transposes<I / 16, I / 4 % 4, I % 4>() && ...);
}
static_assert(patterns_transpose(std::make_integer_sequence<int, 64>{}),
              "rows by destination use the patterns of the exchanged degrees");

// The tables of shape R for the plan: R is the plan's shape, or that with x and out exchanged.  False if the plan's terms
// are not exactly the compiled-in patterns.
template <typename R>
bool fill_tables(luna_uvu_plan* plan, bool exchanged) {
  std::vector<double> term_c(R::terms, 0.0), prog_c(2 * R::m_total, 0.0);
  std::vector<unsigned short> prog_j(R::m_total, kNoAttribute | kNoAttribute << 8);
  std::vector<int> entry_terms(R::m_total, 0);
  std::vector<double> coef(R::coff(-1, -1, -1), 0.0);
  for (const PathRec& p : plan->paths) {
    const int l1 = (p.d1 - 1) / 2, l2 = (p.d2 - 1) / 2, l3 = (p.d3 - 1) / 2, a = exchanged ? l3 : l1, c = exchanged ? l1 : l3;
    const CgTerm* pattern = cg_pattern(a, l2, c);
    const bool diagonal = R::diagonal(a, l2, c);
    double* const one = &coef[diagonal ? R::coff(a, l2, c) : 0];
    const int n = cg_count(a, l2, c), toff = R::toff(a, l2, c), moff = R::moff(a, l2, c);
    std::vector<char> seen(n, 0);
    int found = 0;
    for (int k = 0; k < p.d3; ++k)
      for (int t = plan->rowptr_k[p.byk_ptr + k]; t < plan->rowptr_k[p.byk_ptr + k + 1]; ++t) {
        const auto& term = plan->terms_k[t];  // (a, b) = (i, j)
        const int row = exchanged ? k : term.a, column = exchanged ? term.a : k;
        int slot = -1;
        for (int u = 0; u < n; ++u)
          if (pattern[u].i == row && pattern[u].j == term.b && pattern[u].k == column) slot = u;
        if (slot < 0 || seen[slot]) return false;
        seen[slot] = 1;
        ++found;
        if (diagonal) {  // one coefficient, up to the rounding of the tensor
          if (found == 1) *one = term.c;
          if (std::abs(term.c - *one) > std::abs(*one) * (plan->dtype == LUNA_F64 ? 4e-15 : 5e-7)) return false;
          continue;
        }
        term_c[toff + slot] = term.c;
        int entry = moff - 1;  // the term's (i, k) among the pattern's distinct ones
        for (int u = 0; u <= slot; ++u)
          entry += u == 0 || pattern[u].i != pattern[u - 1].i || pattern[u].k != pattern[u - 1].k;
        const int which = entry_terms[entry]++;
        if (which > 1) return false;  // degrees up to 3 have at most two terms per entry
        prog_c[which * R::m_total + entry] = term.c;
        prog_j[entry] = static_cast<unsigned short>((prog_j[entry] & ~(255 << (8 * which))) | (p.y_off + term.b) << (8 * which));
      }
    if (found != n) return false;
  }
  plan->edge.term_c[exchanged] = term_c;
  plan->edge.prog_c[exchanged] = prog_c;
  plan->edge.prog_j[exchanged] = prog_j;
  plan->edge.coef[exchanged] = coef;
  return true;
}

template <typename S>
bool match_shape(luna_uvu_plan* plan) {
  const auto& paths = plan->paths;
  const int ch = paths[0].ch;
  if (static_cast<int>(paths.size()) != S::paths || plan->X != S::XD * ch || plan->O != S::OD * ch || plan->Y != S::YD ||
      plan->W != S::paths * ch)
    return false;
  for (const PathRec& p : paths) {
    const int l1 = (p.d1 - 1) / 2, l2 = (p.d2 - 1) / 2, l3 = (p.d3 - 1) / 2;
    if (p.ch != ch || p.w_stride != 1 || l1 > 3 || l2 > 3 || l3 > 3 || !S::ok(l1, l2, l3)) return false;
    if (p.x_off != ch * S::xoff(l1) || p.y_off != S::yoff(l2) || p.out_off != ch * S::ooff(l3) ||
        p.w_off != ch * S::rank(l1, l2, l3))
      return false;
  }
  if (!fill_tables<S>(plan, false) || !fill_tables<Transposed<S>>(plan, true)) return false;
  plan->edge.ch = ch;
  return true;
}

template <int ID>
int find_shape(luna_uvu_plan* plan) {
  if constexpr (ID < kEdgeShapes) {
    return match_shape<ShapeOf<ID>>(plan) ? ID : find_shape<ID + 1>(plan);
  } else {
    return -1;
  }
}

// Calls body with the compiled instance of a plan.
template <typename T, int CPL, int ID, typename F>
int with_shape(int shape, F&& body) {
  if constexpr (ID < kEdgeShapes) {
    if (shape == ID) return body(EdgeKernels<T, CPL, ID>{});
    return with_shape<T, CPL, ID + 1>(shape, body);
  } else {
    return fail(LUNA_ERR_UNSUPPORTED, "no edge kernel of shape %d", shape);
  }
}
template <typename F>
int with_instance(const luna_uvu_plan* plan, const EdgeLanes& lanes, F&& body) {
  const int shape = plan->edge.shape;
  if (plan->dtype == LUNA_F64)
    return lanes.cpl == 3 ? with_shape<double, 3, 0>(shape, body)
                          : (lanes.cpl == 2 ? with_shape<double, 2, 0>(shape, body) : with_shape<double, 1, 0>(shape, body));
  if (lanes.cpl == 4) return with_shape<float, 4, 0>(shape, body);
  if (lanes.cpl == 3) return with_shape<float, 3, 0>(shape, body);
  return lanes.cpl == 2 ? with_shape<float, 2, 0>(shape, body) : with_shape<float, 1, 0>(shape, body);
}

}  // namespace

// Slices pay against the table kernels: 300 MB of weights, 20 edges per node, forward / backward, degrees (2, 3, 3), FP32, 352
// channels 0.37 / 1.41 -> 0.18 / 0.46 ms, 1,024 channels 0.24 / 1.03 -> 0.12 / 0.26; (3, 3, 3), FP64, 288 channels
// 0.39 / 1.14 -> 0.18 / 0.47.
void analyse(luna_uvu_plan* plan) {
  plan->edge = EdgePlan{};
  if (plan->paths.empty() || plan->tuning.no_canon) return;
  const int elem = plan->dtype == LUNA_F64 ? 8 : 4;
  if (plan->paths[0].ch * elem % 16 != 0) return;  // bulk copies move whole 16-byte pieces
  const int shape = find_shape<0>(plan);
  if (shape < 0) return;
  const bool sliced = choose_lanes(plan, shape, EdgeUse::kForward, false).cpl == 0;
  if (sliced && !edge_sliced(shape)) return;
  plan->edge.lanes = choose_lanes(plan, shape, EdgeUse::kForward, sliced, true);
  plan->edge.lanes_rows = choose_lanes(plan, shape, EdgeUse::kForward, sliced);
  if (plan->edge.lanes.cpl == 0) plan->edge.lanes = plan->edge.lanes_rows;  // counts that only three channels per lane divide
  plan->edge.lanes_one = choose_lanes(plan, shape, EdgeUse::kOneGradient, sliced);
  plan->edge.lanes_sums = choose_lanes(plan, shape, EdgeUse::kSums, sliced);
  plan->edge.lanes_output = choose_lanes(plan, shape, EdgeUse::kOutputAndWeights, sliced);
  plan->edge.lanes_all = choose_lanes(plan, shape, EdgeUse::kAllGradients, sliced);
  for (const EdgeLanes* lanes : {&plan->edge.lanes, &plan->edge.lanes_rows, &plan->edge.lanes_one, &plan->edge.lanes_sums, &plan->edge.lanes_output, &plan->edge.lanes_all})
    if (lanes->cpl == 0) return;
  plan->edge.shape = shape;
}

int forward(const luna_uvu_plan* plan, const DeviceTables& dt, const luna_graph* graph, const void* x, const void* y,
            const void* w, void* out, bool accumulate, cudaStream_t stream) {
  const EdgeForwardArgs args{x, y, w, out, accumulate};
  const EdgeLanes& lanes = shares_rows(graph->num_nodes, graph->num_edges, dt.sm_count) ? plan->edge.lanes : plan->edge.lanes_rows;
  return with_instance(plan, lanes, [&](auto kernels) { return kernels.forward(plan, dt, graph, lanes, args, stream); });
}

int backward(const luna_uvu_plan* plan, const DeviceTables& dt, const luna_graph* graph, const void* x, const void* y,
             const void* w, const void* g, void* gx, bool acc_x, void* gy, bool acc_y, void* gw, bool acc_w, void* scratch,
             int64_t scratch_bytes, cudaStream_t stream) {
  const EdgeBackwardArgs args{x, y, w, g, gx, gy, gw, acc_x, acc_y, acc_w, scratch, scratch_bytes, nullptr};
  const EdgeLanes& lanes = gy && (gx || gw) ? plan->edge.lanes_all : (gx ? plan->edge.lanes_sums : plan->edge.lanes_one);
  return with_instance(plan, lanes, [&](auto kernels) { return kernels.backward(plan, dt, graph, lanes, args, stream); });
}

int output_and_weights(const luna_uvu_plan* plan, const DeviceTables& dt, const luna_graph* graph, const void* x, const void* y,
                       const void* w, const void* g, void* out, void* gw, cudaStream_t stream) {
  const EdgeBackwardArgs args{x, y, w, g, nullptr, nullptr, gw, false, false, false, nullptr, 0, out};
  const EdgeLanes& lanes = plan->edge.lanes_output;
  return with_instance(plan, lanes, [&](auto kernels) { return kernels.backward(plan, dt, graph, lanes, args, stream); });
}

bool joins_output(const luna_uvu_plan* plan) {
  bool joins = false;
  with_instance(plan, plan->edge.lanes_output, [&](auto kernels) {
    joins = kernels.joins_output();
    return LUNA_OK;
  });
  return joins;
}

int canonical_l2(const luna_uvu_plan* plan) {
  int top = -1;
  for (int mask : kEdgeShapeMasks[plan->edge.shape])
    if ((mask & (mask + 1)) != 0) return -1;
  for (int mask = kEdgeShapeMasks[plan->edge.shape][1]; mask != 0; mask >>= 1) ++top;
  return top;
}

size_t smem_bytes(const luna_uvu_plan* plan, bool backward, int max_smem) {
  size_t bytes = 0;
  for (const EdgeLanes* lanes : {backward ? &plan->edge.lanes_all : &plan->edge.lanes, backward ? &plan->edge.lanes_all : &plan->edge.lanes_rows})
    with_instance(plan, *lanes, [&](auto kernels) {
      bytes = std::max(bytes, kernels.smem_bytes(plan, *lanes, backward, max_smem));
      return LUNA_OK;
    });
  return bytes;
}

}  // namespace edgek
}  // namespace luna
