// Forward kernel for narrow blocks: a warp walks two edges at a time, one on each half of its lanes.
//
// With 16, 32 or 48 channels the arithmetic of an edge is a few dozen instructions per warp, and what an edge costs beside
// it - waits, copies, addresses, the coupling matrices - is several times that.  Here a lane owns CPL channels of
// half a warp, 16 * CPL channels in all, and both halves run the same instructions on an edge each.  One edge per warp and
// two, degrees (2, 2, 2), 0.2 M edges, forward / all gradients: FP32, 32 channels 0.116 / 0.259 -> 0.105 / 0.216 ms, 16
// channels 0.118 / 0.278 -> 0.089 / 0.177; FP64, 16 channels 0.148 / 0.460 -> 0.105 / 0.248; (0, 1, 1), 16 channels, 0.8 M
// edges 0.190 / 0.424 -> 0.133 / 0.223.  What bounds it is still issue: the weights alone take 0.045 ms at 32 channels.
//
// The edges of a tile are taken in pairs from its first one, whatever the rows.  Where a row ends between the two edges of
// a pair, the second half leaves its sum of that row in memory, begins the next row with that pair, and the first half adds
// what it has when it is done.  Either way the sum of a row that lies in one tile is that of its first, third, ... edges plus that
// of the others, wherever the tile begins.  Where the call adds to its output, a row that ends inside a pair is (what is there +
// the second half's) + the first half's, any other what is there + both; a row cut by equal parts is paired anew in each part.
#pragma once

#include "uvu_edge_fwd.cuh"

namespace luna {
namespace edgek {

// Elements of a stage that one half's rows take: with spread packets an odd multiple of 16, so that the halves' lanes read
// different banks.
template <typename PK>
__host__ __device__ constexpr int pair_half(int elems) {
  return PK::spread && elems % 32 == 0 ? elems + 16 : elems;
}
template <typename T, int CPL, typename S>
struct PairFwd {
  static constexpr int words = sizeof(T) / 4;
  static constexpr int max_warps = warps_for((S::OD + S::XD) * CPL * words + 4 * S::m_rounds * words + S::m_rounds + 1 + 44);
};

// 16 * CPL channels.
template <typename T, int CPL, typename S>
__global__ void __launch_bounds__(PairFwd<T, CPL, S>::max_warps * 32, 1)
    pair_fwd_kernel(const __grid_constant__ EdgeFwdParams<T> P) {
  using PK = PkT<T, CPL, UsePairs<T, CPL>::value>;
  using V = typename PK::V;
  constexpr int NP = PK::NP;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  let_next_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4, place = lane & 15;
  constexpr int ch = 16 * CPL, lanes = 16, W = S::paths * ch, X = S::XD * ch, O = S::OD * ch, half_elems = pair_half<PK>(W + X), stage_elems = 2 * half_elems;
  const int stages = P.stages, own = lane_first<PK>(place);

  T* const ring = reinterpret_cast<T*>(smem_raw) + static_cast<size_t>(warp) * P.ring_elems;
  T* const mbuf = reinterpret_cast<T*>(smem_raw) + static_cast<size_t>(P.teams) * P.ring_elems +
                  static_cast<size_t>(warp * 2 + half) * (2 * S::m_elems);  // two per half
  uint64_t* const bars = reinterpret_cast<uint64_t*>(reinterpret_cast<T*>(smem_raw) +
                                                     static_cast<size_t>(P.teams) * (P.ring_elems + 4 * S::m_elems)) +
                         warp * kEdgeMaxStages;
  TeamPart* const kept = reinterpret_cast<TeamPart*>(bars + (P.teams - warp) * kEdgeMaxStages);
  if (lane == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&bars[s], 2);  // both halves' copies
    fence_barrier_init();
  }
  HalfMatrixProgram<T, S> program;
  program.load(P.prog_c, P.prog_j, place);
  __syncthreads();
  wait_for_previous();

  const bool issuing = place == 0;  // a half's copies are its first lane's
  const uint32_t w_bytes = static_cast<uint32_t>(W * sizeof(T)), x_bytes = static_cast<uint32_t>(X * sizeof(T));
  auto issue = [&](int e, int s_node, bool real, int s) {  // by the issuing lane of either half, of its edge
    T* to = ring + static_cast<size_t>(s) * stage_elems + half * half_elems;
    mbar_arrive_expect_tx(&bars[s], real ? w_bytes + x_bytes : 0u);
    if (!real) return;
    bulk_copy_g2s_hint(to, P.w + static_cast<int64_t>(e) * W, w_bytes, &bars[s], l2_policy_evict_first());
    bulk_copy_g2s(to + W, P.x + static_cast<int64_t>(s_node) * X, x_bytes, &bars[s]);
  };

  V acc[S::OD * NP];
#pragma unroll
  for (int a = 0; a < S::OD * NP; ++a) acc[a] = zero_packet<V>();
  int s = 0;
  uint32_t parity = 0;
  bool alive = true;
  int buf = 0;
  const bool grouped = P.group > 1, parts = P.parts != 0;
  int open_row = -1;  // whose sum goes to shared memory, to be added to what the next team has of it
  const int in_group = warp % P.group, group_id = warp / P.group, groups = P.teams / P.group;
  const unsigned total = gridDim.x * static_cast<unsigned>(grouped ? groups : P.teams);
  unsigned unit = grouped ? blockIdx.x + gridDim.x * group_id : blockIdx.x * P.teams + warp;
  const unsigned units = parts ? total : static_cast<unsigned>(grouped ? P.num_rows : P.num_tiles);

  // acc of one half to row n, added to what is there if `add`, and zero again
  auto store = [&](int n, int by, bool add) {
    if (half == by) {
      const bool rest = grouped || n == open_row;
      T* to = rest ? ring : P.out + static_cast<int64_t>(n) * O;
      static_for<0, 4>([&](auto l3c) {
        constexpr int l3 = decltype(l3c)::value, d3 = 2 * l3 + 1;
        if constexpr (S::has(S::MO, l3))
          lane_store_block<PK, T, d3>(to + ch * S::ooff(l3) + own * d3, lanes, &acc[S::ooff(l3) * NP], !rest && add);
      });
#pragma unroll
      for (int a = 0; a < S::OD * NP; ++a) acc[a] = zero_packet<V>();
    }
  };
  const bool accumulate = P.accumulate != 0;
  // both halves' sums to the first one
  auto gather = [&] {
#pragma unroll
    for (int a = 0; a < S::OD * NP; ++a) {
      const V other = shfl_xor_packet(acc[a], 16);
      acc[a] = half == 0 ? vadd(acc[a], other) : zero_packet<V>();
    }
  };

#pragma unroll 1
  while (unit < units) {
    unsigned unit_after = unit + total;
    int n = static_cast<int>(unit), n_hi = n + 1, e, e_end;
    if (parts) {
      const TeamPart part = team_part(P.dst_rowptr, P.num_rows, P.num_edges, P.rows_per_edge, warp, P.teams, lane);
      n = part.n;
      n_hi = part.n_hi;
      e = part.pos;
      e_end = part.end;
      open_row = part.open_row();
      if (lane == 0) kept[warp] = part;  // for the end of the launch
    } else if (!grouped) {
      unit_after = static_cast<unsigned>(take_tile(P.tile_counters, total, lane));
      const int64_t first = unit * P.tile_rows, end = first + P.tile_rows;
      n = static_cast<int>(first);
      n_hi = static_cast<int>(end < P.num_rows ? end : P.num_rows);
    }
    if (!parts) {
      e = P.dst_rowptr[n];
      e_end = P.dst_rowptr[n_hi];
    }
    if (grouped) {
      const int first = e;
      const int64_t count = e_end - e;
      e = first + static_cast<int>(count * in_group / P.group);
      e_end = first + static_cast<int>(count * (in_group + 1) / P.group);
    }
    int mine = e + half;  // this half's edge
    if (issuing) {
      for (int d = 0, stage = s; d < stages; ++d) {
        const int ahead = mine + 2 * d;
        if (e + 2 * d < e_end) issue(ahead, ahead < e_end ? P.src[ahead] : 0, ahead < e_end, stage);
        if (++stage == stages) stage = 0;
      }
    }
    int src_ahead = issuing && mine + 2 * stages < e_end ? P.src[mine + 2 * stages] : 0;
    T y_next = place < S::YD && mine < e_end ? P.y[static_cast<int64_t>(mine) * S::YD + place] : T(0);
    program.run(y_next, mbuf + buf * S::m_elems, place);
    y_next = place < S::YD && mine + 2 < e_end ? P.y[static_cast<int64_t>(mine + 2) * S::YD + place] : T(0);
    __syncwarp();
    int row_end = first_row_end(P.dst_rowptr, n, n_hi, e_end);
#pragma unroll 1
    for (; e < e_end; e += 2, mine += 2) {
#pragma unroll 1
      while (e >= row_end) {  // rows that ended before this pair
        gather();
        store(n, 0, accumulate);
        row_end = min(P.dst_rowptr[++n + 1], e_end);
      }
      const bool straddle = e + 1 >= row_end && e + 1 < e_end;  // the second edge is of a later row
      if (straddle) store(n, 1, accumulate);
      if (!edge_wait(&bars[s], parity, alive)) {
        if (lane == 0) atomicExch(P.status, 1);
        alive = false;
      }
      const T* ws = ring + static_cast<size_t>(s) * stage_elems + half * half_elems + own;
      const T* xs = ws - own + W;
      program.run(y_next, mbuf + (buf ^ 1) * S::m_elems, place);  // of the next pair; of no use after the last one
      if (place < S::YD && mine + 4 < e_end) y_next = P.y[static_cast<int64_t>(mine + 4) * S::YD + place];
      const T* m_now = mbuf + buf * S::m_elems;
      if (mine < e_end) forward_edge<T, PK, S>(ws, xs, ch, own, lanes, m_now, P.coef, acc);
      buf ^= 1;
      fence_async_shared();  // what was read of this stage, before it is refilled
      __syncwarp();          // every lane is done with it and with the matrices
      if (issuing && e + 2 * stages < e_end) {
        issue(mine + 2 * stages, src_ahead, mine + 2 * stages < e_end, s);
        if (mine + 2 * stages + 2 < e_end) src_ahead = P.src[mine + 2 * stages + 2];
      }
      if (++s == stages) {
        s = 0;
        parity ^= 1u;
      }
      if (straddle) {  // the first half ended row n; the rows up to the second half's have no edges
        bool add = true;
#pragma unroll 1
        do {
          store(n, 0, add);
          add = accumulate;
          row_end = min(P.dst_rowptr[++n + 1], e_end);
        } while (e + 1 >= row_end);
      }
    }
    gather();
#pragma unroll 1
    for (; n < n_hi; ++n) store(n, 0, accumulate);
    if (grouped) {  // the parts of the row, in order
      const int threads = P.group * 32;
      const T* parts = reinterpret_cast<const T*>(smem_raw) + static_cast<size_t>(group_id * P.group) * P.ring_elems;
      named_barrier(1 + group_id, threads);
      T* to = P.out + static_cast<int64_t>(unit) * O;
      for (int a = static_cast<int>(threadIdx.x) - group_id * threads; a < O; a += threads) {
        T sum = parts[a];
        for (int g = 1; g < P.group; ++g) sum += parts[static_cast<size_t>(g) * P.ring_elems + a];
        to[a] = P.accumulate ? to[a] + sum : sum;
      }
      fence_async_shared();  // threads have written and read the ring; its next users are bulk copies
      named_barrier(1 + group_id, threads);
    }
    unit = unit_after;
  }
  if (parts) {
    merge_parts(kept, P.teams, P.dst_rowptr, reinterpret_cast<const T*>(smem_raw), P.ring_elems, O,
                [&](int row, int a) { return P.out + static_cast<int64_t>(row) * O + a; });
  } else if (!grouped) {
    leave_tiles(P.tile_counters, total, lane);
  }
  if (!alive)  // let copies that are still in flight land before the CTA's shared memory is released
    for (int d = 0; d < stages; ++d) edge_wait(&bars[d], d < s ? parity : parity ^ 1u, false);
}

template <typename T, int CPL, typename S>
EdgeLaunch pair_fwd_launch(const Tuning& tuning, int ch, int max_smem) {
  const size_t stage = 2 * static_cast<size_t>(pair_half<PkT<T, CPL, UsePairs<T, CPL>::value>>((S::paths + S::XD) * ch)) * sizeof(T), row = static_cast<size_t>(S::OD) * ch * sizeof(T);
  EdgeLaunch launch;
  const int max_warps = capped_warps(tuning, PairFwd<T, CPL, S>::max_warps);
  for (int warps = max_warps; warps >= 1 && launch.warps == 0; --warps)
    for (int stages = warps * 2 > max_warps ? 3 : kEdgeMaxStages; stages >= 2; --stages) {
      const size_t ring = (std::max(stages * stage, row) + 127) / 128 * 128;
      const size_t bytes = warps * (ring + 4 * S::m_elems * sizeof(T) + kEdgeMaxStages * sizeof(uint64_t) + sizeof(TeamPart));
      if (bytes > static_cast<size_t>(max_smem)) continue;
      launch.warps = warps;
      launch.stages = stages;
      launch.bytes = bytes;
      launch.team_elems = static_cast<int>(ring / sizeof(T));
      break;
    }
  return launch;
}

}  // namespace edgek
}  // namespace luna
