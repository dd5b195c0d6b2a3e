// The edge kernels of one element type, channels per lane and shape.  The build compiles this file once for each
// combination (LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE), so that they compile in parallel.
#include "uvu_edge_bwd_launch.cuh"
#include "uvu_edge_fwd_launch.cuh"

namespace luna {
namespace edgek {

template <>
int EdgeKernels<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE>::forward(const luna_uvu_plan* plan, const DeviceTables& dt,
                                                                      const luna_graph* graph, const EdgeLanes& lanes, const EdgeForwardArgs& a,
                                                                      cudaStream_t stream) {
  using S = ShapeOf<LUNA_EDGE_SHAPE>;
  if constexpr (edge_sliced(LUNA_EDGE_SHAPE) && LUNA_EDGE_CPL != 3) {
    if (lanes.slices > 1) return launch_edge_fwd<LUNA_EDGE_T, LUNA_EDGE_CPL, S, true, true, false>(plan, dt, graph, lanes, a, stream);
  }
  if constexpr (edge_paired<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE>(EdgeUse::kForward)) {
    if (lanes.edges == 2) return launch_edge_fwd<LUNA_EDGE_T, LUNA_EDGE_CPL, S, true, false, true>(plan, dt, graph, lanes, a, stream);
  }
  if constexpr (edge_alone<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE>(EdgeUse::kForward)) {
    if (plan->edge.ch == 32 * LUNA_EDGE_CPL)
      return launch_edge_fwd<LUNA_EDGE_T, LUNA_EDGE_CPL, S, true, false, false>(plan, dt, graph, lanes, a, stream);
    return launch_edge_fwd<LUNA_EDGE_T, LUNA_EDGE_CPL, S, false, false, false>(plan, dt, graph, lanes, a, stream);
  } else {
    return fail(LUNA_ERR_UNSUPPORTED, "no forward kernel of this layout");
  }
}

template <>
int EdgeKernels<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE>::backward(const luna_uvu_plan* plan, const DeviceTables& dt,
                                                                       const luna_graph* graph, const EdgeLanes& lanes, const EdgeBackwardArgs& a,
                                                                       cudaStream_t stream) {
  if constexpr (edge_sliced(LUNA_EDGE_SHAPE) && LUNA_EDGE_CPL != 3) {
    if (lanes.slices > 1)
      return dispatch_edge_bwd<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE, true, true, false>(plan, dt, graph, lanes, a, stream);
  }
  if (lanes.edges == 2)
    return dispatch_edge_bwd<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE, true, false, true>(plan, dt, graph, lanes, a, stream);
  if (plan->edge.ch == 32 * LUNA_EDGE_CPL)
    return dispatch_edge_bwd<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE, true, false, false>(plan, dt, graph, lanes, a, stream);
  return dispatch_edge_bwd<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE, false, false, false>(plan, dt, graph, lanes, a, stream);
}

template <>
bool EdgeKernels<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE>::joins_output() {
  return edge_joins_output<LUNA_EDGE_T, LUNA_EDGE_CPL, ShapeOf<LUNA_EDGE_SHAPE>>();
}

template <>
size_t EdgeKernels<LUNA_EDGE_T, LUNA_EDGE_CPL, LUNA_EDGE_SHAPE>::smem_bytes(const luna_uvu_plan* plan, const EdgeLanes& lanes,
                                                                            bool backward, int max_smem) {
  using S = ShapeOf<LUNA_EDGE_SHAPE>;
  const int ch = plan->edge.ch / lanes.slices;
  if (lanes.edges == 2)
    return backward ? pair_bwd_launch<LUNA_EDGE_T, S, PairBwd<LUNA_EDGE_T, LUNA_EDGE_CPL, S, true, true, true>>(plan->tuning, ch, max_smem).bytes
                    : pair_fwd_launch<LUNA_EDGE_T, LUNA_EDGE_CPL, S>(plan->tuning, ch, max_smem).bytes;
  if (!backward)
    return ch == 32 * LUNA_EDGE_CPL ? edge_fwd_launch<LUNA_EDGE_T, LUNA_EDGE_CPL, S, true>(plan->tuning, lanes, ch, max_smem).bytes
                                    : edge_fwd_launch<LUNA_EDGE_T, LUNA_EDGE_CPL, S, false>(plan->tuning, lanes, ch, max_smem).bytes;
  using K = EdgeBwd<LUNA_EDGE_T, LUNA_EDGE_CPL, S, true, true, true>;
  return edge_bwd_launch<LUNA_EDGE_T, S, K, true>(plan->tuning, lanes, ch, max_smem).bytes;
}

}  // namespace edgek
}  // namespace luna
