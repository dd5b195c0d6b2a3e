// Launches of the forward kernels of the edge family.
#pragma once

#include "uvu_edge_fwd.cuh"
#include "uvu_pair_fwd.cuh"

namespace luna {
namespace edgek {

template <typename T, int CPL, typename S, bool FULL, bool SLICED, bool PAIR>
int launch_edge_fwd(const luna_uvu_plan* plan, const DeviceTables& dt, const luna_graph* graph,
                    const EdgeLanes& lanes, const EdgeForwardArgs& a, cudaStream_t stream) {
  static_assert(!PAIR || (FULL && !SLICED), "two edges at a time: a half warp's full set of channels");
  void (*kernel)(EdgeFwdParams<T>);
  if constexpr (PAIR)
    kernel = pair_fwd_kernel<T, CPL, S>;
  else
    kernel = edge_fwd_kernel<T, CPL, S, FULL, SLICED>;
  EdgeFwdParams<T> P;
  P.x = static_cast<const T*>(a.x);
  P.y = static_cast<const T*>(a.y);
  P.w = static_cast<const T*>(a.w);
  P.out = static_cast<T*>(a.out);
  P.src = graph->src;
  P.dst_rowptr = graph->dst_rowptr;
  P.prog_c = static_cast<const T*>(dt.edge[0].prog_c);
  P.prog_j = dt.edge[0].prog_j;
  for (int c = 0; c < S::coff(-1, -1, -1); ++c) P.coef[c] = static_cast<T>(plan->edge.coef[0][c]);
  P.status = dt.status;
  P.tile_counters = next_tile_counters(plan, dt);
  P.num_rows = graph->num_nodes;
  P.ch = plan->edge.ch / lanes.slices;
  P.row_ch = plan->edge.ch;
  P.team_warps = lanes.team_warps;
  P.accumulate = a.accumulate ? 1 : 0;
  EdgeLaunch launch = PAIR ? pair_fwd_launch<T, CPL, S>(plan->tuning, P.ch, dt.max_smem_optin)
                           : edge_fwd_launch<T, CPL, S, FULL>(plan->tuning, lanes, P.ch, dt.max_smem_optin);
  if (launch.warps == 0) return fail(LUNA_ERR_UNSUPPORTED, "the rows of an edge do not fit the shared memory of this device");
  P.stages = launch.stages;
  P.ring_elems = launch.team_elems;
  P.teams = launch.warps / lanes.team_warps;
  const int ctas = SLICED ? slice_ctas(dt.sm_count, lanes.slices) : dt.sm_count;
  // Teams that share rows come in twos, fours or eights: of seven or thirteen none could share one.  Whatever the number of rows, so that
  // a piece of such a graph has the same groups.  Ten teams in twos and eight in eights, 24 / 100 / 300 / 440 nodes of 30 edges: FP64
  // (2, 2, 2), 64 channels 16.8 / 20.9 / 22.8 / 26.1 and 7.9 / 9.2 / 22.0 / 23.6 us, (3, 3, 0) 10.2 / 12.6 / 13.9 / 14.7 and 5.8 / 6.6 / 15.0 /
  // 16.3; FP32 (2, 3, 3), fourteen and twelve, 18.4 / 22.8 / 24.8 / 27.8 and 11.2 / 13.3 / 17.2 / 19.8.
  if (shares_rows(graph->num_nodes, graph->num_edges, ctas) && P.teams > 4) {
    P.teams -= P.teams > 8 ? P.teams % 4 : P.teams % 2;
    launch.warps = P.teams * lanes.team_warps;
  }
  const int64_t sources = graph->num_src_nodes > 0 ? graph->num_src_nodes : graph->num_nodes;
  const EdgeSplit split =
      edge_split(graph->num_nodes, graph->num_edges, ctas, P.teams, lanes.team_warps, 64, lanes.edges,
                 sources * plan->X * static_cast<int64_t>(sizeof(T)), true);
  P.group = split.group;
  P.num_edges = graph->num_edges;
  P.rows_per_edge = static_cast<float>(static_cast<double>(P.num_rows) / static_cast<double>(std::max<int64_t>(P.num_edges, 1)));
  P.parts = split.parts;
  P.tile_rows = split.tile_rows;
  P.num_tiles = ceil_div(std::max<int64_t>(graph->num_nodes, 1), split.tile_rows);
  static KernelSetup setup;
  const int rc = setup.once(reinterpret_cast<const void*>(kernel), dt.max_smem_optin);
  if (rc != LUNA_OK) return rc;
  const dim3 grid(static_cast<unsigned>(split.blocks), static_cast<unsigned>(lanes.slices));
  launch_early(kernel, grid, launch.warps * 32, launch.bytes, stream, P);
  LUNA_LAUNCH_CHECK("forward (edge family)");
  return LUNA_OK;
}

}  // namespace edgek
}  // namespace luna
