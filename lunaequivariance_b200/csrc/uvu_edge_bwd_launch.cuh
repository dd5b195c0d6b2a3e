// Launches of the backward kernels of the edge family.
#pragma once

#include "uvu_edge_bwd.cuh"
#include "uvu_pair_bwd.cuh"

namespace luna {
namespace edgek {

// K: the EdgeBwd of the kernel.
template <typename T, typename S, typename K, bool FULL>
EdgeLaunch edge_bwd_launch(const Tuning& tuning, const EdgeLanes& lanes, int ch, int max_smem) {
  const size_t w_row = static_cast<size_t>(S::paths) * ch * sizeof(T);
  const size_t x_row = static_cast<size_t>(S::XD) * ch * sizeof(T), g_row = static_cast<size_t>(S::OD) * ch * sizeof(T);
  EdgeLaunch launch;
  const int max_teams = capped_warps(tuning, K::template warps<FULL>) / lanes.team_warps;
  for (int teams = max_teams; teams >= 1 && launch.warps == 0; --teams)
    for (int option = 0; option < 3; ++option) {  // three or two stages with g in them, or two and g by degree
      const int stages = option == 0 ? 3 : 2, split = option == 2;
      size_t team = split ? stages * w_row + g_row : stages * (w_row + g_row);
      team = (std::max(team, x_row) + 127) / 128 * 128;
      const size_t bytes = teams * (team + (kEdgeMaxStages + kEdgeMaxSlots) * sizeof(uint64_t) + sizeof(unsigned) + sizeof(TeamPart)) +
                           (static_cast<size_t>(teams) * lanes.team_warps * K::warp_elems(lanes.team_warps)) * sizeof(T);
      if (bytes > static_cast<size_t>(max_smem)) continue;
      launch.warps = teams * lanes.team_warps;
      launch.stages = stages;
      launch.split = split;
      launch.bytes = bytes;
      launch.team_elems = static_cast<int>(team / sizeof(T));
      break;
    }
  return launch;
}

template <typename T, int CPL, typename S, bool WX, bool WM, bool WY, bool FULL, bool DST, bool SLICED, bool PAIR, bool ADD = false>
int launch_edge_bwd(const luna_uvu_plan* plan, const DeviceTables& dt, const luna_graph* graph,
                    const EdgeLanes& lanes, const EdgeBackwardArgs& a, cudaStream_t stream) {
  using K = EdgeBwd<T, CPL, S, WX, WM, WY>;
  static_assert(!PAIR || (FULL && !SLICED), "two edges at a time: a half warp's full set of channels");
  void (*kernel)(EdgeBwdParams<T, K::terms>);
  if constexpr (PAIR)
    kernel = pair_bwd_kernel<T, CPL, S, WX, WM, WY, DST, ADD>;
  else
    kernel = edge_bwd_kernel<T, CPL, S, WX, WM, WY, FULL, DST, SLICED, ADD>;
  EdgeBwdParams<T, K::terms> P;
  P.x = static_cast<const T*>(DST ? a.g : a.x);
  P.y = static_cast<const T*>(a.y);
  P.w = static_cast<const T*>(ADD ? a.gw : a.w);
  P.g = static_cast<const T*>(DST ? a.x : a.g);
  P.gx = static_cast<T*>(DST ? a.out : a.gx);
  P.gy = static_cast<T*>(a.gy);
  P.gw = static_cast<T*>(a.gw);
  P.dst = DST ? graph->src : graph->dst;
  P.src_rowptr = DST ? graph->dst_rowptr : graph->src_rowptr;
  P.edge_ids = DST ? nullptr : graph->edge_ids_by_src;
  const EdgeTables& tables = dt.edge[DST ? 1 : 0];
  if constexpr (WY)
    for (int t = 0; t < S::terms; ++t) P.term[t] = static_cast<T>(plan->edge.term_c[DST ? 1 : 0][t]);
  P.prog_c = static_cast<const T*>(tables.prog_c);
  P.prog_j = tables.prog_j;
  for (int c = 0; c < S::coff(-1, -1, -1); ++c) P.coef[c] = static_cast<T>(plan->edge.coef[DST ? 1 : 0][c]);
  P.status = dt.status;
  P.tile_counters = next_tile_counters(plan, dt);
  P.num_rows = !DST && graph->num_src_nodes > 0 ? graph->num_src_nodes : graph->num_nodes;
  P.ch = plan->edge.ch / lanes.slices;
  P.row_ch = plan->edge.ch;
  P.team_warps = lanes.team_warps;
  P.need_w = ADD || WX || a.gx != nullptr || a.gy != nullptr;
  P.acc_x = a.acc_x;
  P.acc_y = a.acc_y;
  P.acc_w = !ADD && a.acc_w;
  P.gy_part = graph->num_edges * S::YD;
  if (SLICED && WY) {
    const int64_t need = lanes.slices * P.gy_part * static_cast<int64_t>(sizeof(T));
    if (a.scratch == nullptr || a.scratch_bytes < need)
      return fail(LUNA_ERR_SCRATCH, "backward needs %lld bytes of scratch for the slices' parts of gy", static_cast<long long>(need));
    if (!aligned_to(a.scratch, 16)) return fail(LUNA_ERR_MISALIGNED, "scratch must be 16-byte aligned");
    P.gy = static_cast<T*>(a.scratch);
    P.acc_y = 0;
  }
  EdgeLaunch launch;
  if constexpr (PAIR)
    launch = pair_bwd_launch<T, S, PairBwd<T, CPL, S, WX, WM, WY>>(plan->tuning, P.ch, dt.max_smem_optin);
  else
    launch = edge_bwd_launch<T, S, K, FULL>(plan->tuning, lanes, P.ch, dt.max_smem_optin);
  if (launch.warps == 0) return fail(LUNA_ERR_UNSUPPORTED, "the rows of an edge do not fit the shared memory of this device");
  P.stages = launch.stages;
  P.team_elems = launch.team_elems;
  P.split = launch.split;
  P.teams = launch.warps / lanes.team_warps;
  const int64_t edges = graph->num_edges;
  P.rows_per_edge = static_cast<float>(static_cast<double>(P.num_rows) / static_cast<double>(std::max<int64_t>(edges, 1)));
  const int ctas = SLICED ? slice_ctas(dt.sm_count, lanes.slices) : dt.sm_count;
  const int64_t tile = edges_per_warp(plan->tuning, 64);
  const int64_t sources = graph->num_src_nodes > 0 ? graph->num_src_nodes : graph->num_nodes;
  EdgeSplit cut = edge_split(P.num_rows, edges, ctas, P.teams, lanes.team_warps, tile, lanes.edges,
                             (DST ? sources : graph->num_nodes) * S::OD * plan->edge.ch * static_cast<int64_t>(sizeof(T)), false);
  P.num_edges = edges;
  P.parts = cut.parts;
  P.every_row = 1;
  P.tile_rows = cut.tile_rows;
  P.tile_edges = tile_edges_for(edges, static_cast<int64_t>(ctas) * P.teams, tile);
  P.num_tiles = ceil_div(std::max<int64_t>(P.num_rows, 1), P.tile_rows);
  // A whole graph of some density, or a shard of one (its own rows plus a halo at most half as large), has hardly any
  // rows without edges, and tiles of a fixed number of rows are even without any search.  A piece of a graph (a
  // destination range against all source rows) has long runs of rows without edges: its tiles are cut by edge count,
  // and the rows that are jumped over are cleared here.
  const bool whole = DST || graph->num_src_nodes <= 0 || graph->num_src_nodes <= graph->num_nodes + graph->num_nodes / 2;
  if (!(whole && (cut.parts || static_cast<double>(edges) >= 8.0 * static_cast<double>(P.num_rows)))) {
    P.every_row = 0;
    if (!cut.parts) {
      P.tile_rows = 0;
      P.num_tiles = ceil_div(std::max<int64_t>(edges, 1), P.tile_edges);
      cut.blocks = std::max<int64_t>(1, std::min<int64_t>(ctas, ceil_div(P.num_tiles, P.teams)));
    }
    if (WX && P.gx && !a.acc_x)
      LUNA_CUDA_CHECK(cudaMemsetAsync(P.gx, 0, static_cast<size_t>(P.num_rows) * S::XD * plan->edge.ch * sizeof(T), stream));
  }
  static KernelSetup setup;
  const int rc = setup.once(reinterpret_cast<const void*>(kernel), dt.max_smem_optin);
  if (rc != LUNA_OK) return rc;
  const dim3 grid(static_cast<unsigned>(cut.blocks), static_cast<unsigned>(lanes.slices));
  // An early start where weights come in and their gradients leave: beyond the size of L2 it costs more than the launch that it hides.
  // Back to back, dL/dw alone, from 16 / 32 / 64 / 128 MB of weights on: FP32 -5 / -3 / -2 / +0.6 %, FP64 -5 / -2 / -1 / +1.3 %; (1, 1, 0),
  // 48 FP64 channels, 0.26 M edges, 200 MB +16 %.  Launches that write no weight gradients are at no size slower on average.
  const int64_t weights = P.num_edges * S::paths * plan->edge.ch * static_cast<int64_t>(sizeof(T));
  if (a.gw == nullptr || weights <= kEarlyWeights)
    launch_early(kernel, grid, launch.warps * 32, launch.bytes, stream, P);
  else
    kernel<<<grid, launch.warps * 32, launch.bytes, stream>>>(P);
  LUNA_LAUNCH_CHECK("backward (edge family)");
  if (SLICED && WY) {
    reduce_gy_partial<T><<<static_cast<unsigned>(ceil_div(P.gy_part, 256)), 256, 0, stream>>>(
        P.gy, static_cast<T*>(a.gy), P.gy_part, lanes.slices, a.acc_y ? 1 : 0);
    LUNA_LAUNCH_CHECK("sum of the slices' parts of gy");
  }
  return LUNA_OK;
}

// Whether output and gw come in one launch: unless the sums cost half the warps that gw alone has (128 channels of a first layer).
// Forward and gw in turn, and together: FP64, (2, 3, 3), 128 channels, 0.4 M edges 3.83 -> 2.75 ms; FP32, the same, 1.05 M edges
// 3.95 -> 3.13; (2, 2, 2), 64 channels, 5.2 M edges 6.72 -> 5.09; (0, 3, 3), 128 channels, 1.05 M edges 1.06 -> 1.20.
template <typename T, int CPL, typename S>
constexpr bool edge_joins_output() {
  using R = Transposed<S>;
  return 2 * EdgeBwd<T, CPL, R, true, true, false>::template warps<true> > EdgeBwd<T, CPL, R, false, true, false>::template warps<true>;
}

// ID: the shape's number, which tells with CPL and PAIR which uses have kernels.
template <typename T, int CPL, int ID, bool FULL, bool SLICED, bool PAIR>
int dispatch_edge_bwd(const luna_uvu_plan* plan, const DeviceTables& dt, const luna_graph* graph,
                      const EdgeLanes& lanes, const EdgeBackwardArgs& a, cudaStream_t stream) {
  using S = ShapeOf<ID>;
  const bool wx = a.gx != nullptr, ww = a.gw != nullptr, wy = a.gy != nullptr;
  auto compiled = [](EdgeUse use) { return SLICED || (PAIR ? edge_paired<T, CPL, ID>(use) : edge_alone<T, CPL, ID>(use)); };
  if constexpr (edge_joins_output<T, CPL, S>() && compiled(EdgeUse::kOutputAndWeights)) {
    if (a.out)
      return launch_edge_bwd<T, CPL, Transposed<S>, true, true, false, FULL, true, SLICED, PAIR>(plan, dt, graph, lanes, a, stream);
  }
  // One gradient per edge and none per row.  FP64, degrees (2, 3, 3), 128 channels, 1.05 M edges: rows by source 5.91 ms
  // (gw) and 6.44 ms (gy), by destination 5.36 and 5.95 ms.
  if constexpr (compiled(EdgeUse::kOneGradient)) {
    if (!a.out && !wx && ww != wy) {
      constexpr bool dst = S::OD >= S::XD;
      using R = std::conditional_t<dst, Transposed<S>, S>;
      if (ww && a.acc_w)
        return launch_edge_bwd<T, CPL, R, false, true, false, FULL, dst, SLICED, PAIR, true>(plan, dt, graph, lanes, a, stream);
      return ww ? launch_edge_bwd<T, CPL, R, false, true, false, FULL, dst, SLICED, PAIR>(plan, dt, graph, lanes, a, stream)
                : launch_edge_bwd<T, CPL, R, false, false, true, FULL, dst, SLICED, PAIR>(plan, dt, graph, lanes, a, stream);
    }
  }
  if constexpr (compiled(EdgeUse::kAllGradients)) {
    if (wy) return launch_edge_bwd<T, CPL, S, true, true, true, FULL, false, SLICED, PAIR>(plan, dt, graph, lanes, a, stream);
  }
  if constexpr (compiled(EdgeUse::kSums)) {
    if (!wy && wx) return launch_edge_bwd<T, CPL, S, true, true, false, FULL, false, SLICED, PAIR>(plan, dt, graph, lanes, a, stream);
  }
  return wx || wy || ww || a.out ? fail(LUNA_ERR_UNSUPPORTED, "no kernel of this layout for these gradients") : LUNA_OK;
}

}  // namespace edgek
}  // namespace luna
