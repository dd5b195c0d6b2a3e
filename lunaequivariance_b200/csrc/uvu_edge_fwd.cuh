// Forward kernel of the edge family:  out[t] = sum_{e: dst e = t} sum_p w_p * (M^p(y_e)^T x[src e]).
//
// Per edge the warp turns the edge attributes into the coupling matrices M^p[i][k] = sum_j C^p_ijk y_j (the entries the
// coupling tensors leave zero for every y are skipped, at compile time), a lane multiplies them into its channels:
// out_k += sum_i M[i][k] * (x_i * w).  FP32 with more than one channel per lane runs on packed two-wide FMAs (three: a pair and a scalar).
// The matrices of the next edge are made while the current edge is computed: its attributes sit one per lane and reach
// the lane that needs them by shuffles, so nothing waits for shared memory in between.
#pragma once

#include "uvu_edge.cuh"

namespace luna {
namespace edgek {

template <typename T>
struct EdgeFwdParams {
  const T *x, *y, *w;
  T* out;
  const int *src, *dst_rowptr;
  const T* prog_c;               // [2][m_total] coefficients of the two attributes an entry depends on
  const unsigned short* prog_j;  // [m_total] the two attributes, 8 bits each
  T coef[kEdgeMaxCoefs];         // of the paths with a degree of zero
  int* status;
  unsigned* tile_counters;
  int64_t num_rows, num_edges, tile_rows, num_tiles;
  float rows_per_edge;
  int ch;          // channels per block, or of a slice of it
  int row_ch;      // channels per block
  int team_warps;  // warps per team
  int teams;       // per CTA
  int group;       // teams that share a row, or 1
  int parts;       // equal parts of the edges
  int stages;
  int ring_elems;  // per team
  int accumulate;
};

template <typename T, int CPL, typename S>
struct EdgeFwd {
  static constexpr int words = sizeof(T) / 4;
  static constexpr int m_elems = S::m_elems;
  static constexpr int registers = (S::OD + S::XD) * CPL * words + S::m_rounds * 2 * words + (S::m_rounds + 1) / 2 + 44;
  // FULL, in FP64 with few matrices: the estimate is a little high.  (2, 2, 2), 64 channels, 0.26 M edges 5 % faster with sixteen warps
  // than with twelve, but 48 channels on 24 lanes 233 -> 256 us, 96 in two warps, 24 nodes, 16.0 -> 18.6.
  template <bool FULL>
  static constexpr int warps = warps_for(registers, FULL && sizeof(T) == 8 && S::m_total <= 64 ? 5 : 0);
  static constexpr size_t team_bytes = 2 * static_cast<size_t>(m_elems) * sizeof(T);
};

// out_k += sum_i M[i][k] * (x_i * w) for one path, over the entries of M that the pattern has.  xl / al: a lane's packets of
// x and of the sums, of degrees l1 and l3; wq: its first weight; buffer: the edge's matrices.
template <typename T, typename PK, typename S, int l1, int l2, int l3, typename V>
__device__ __forceinline__ void forward_path(const T* wq, int lanes, const T* buffer, const V* xl, V* al) {
  constexpr int NP = PK::NP;
  using PT = CgPattern<l1, l2, l3>;
  const T* matrix = buffer + S::moff(l1, l2, l3);
  V w2[NP], xw[NP];
  T m[4];
  lane_load<PK, T>(wq, lanes, w2);
  static_for<0, PT::n>([&](auto tc) {
    constexpr int t = decltype(tc)::value;
    if constexpr (edge_new_entry<PT>(t)) {
      constexpr int i = PT::t[t].i, k = PT::t[t].k, entry = edge_entry<PT>(t);
      if constexpr (entry % 4 == 0) edge_load_four<T>(matrix + entry, m);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        if constexpr (edge_new_row<PT>(t)) xw[p] = vmul(xl[i * NP + p], w2[p]);
        al[k * NP + p] = vfma(bcast_packet(m[entry % 4], V{}), xw[p], al[k * NP + p]);
      }
    }
  });
}
// The paths with a degree of zero, c their coefficient: out_k += (c y w) x_k, (c w x) y_k or (c w) sum_i y_i x_i.
template <typename T, typename PK, typename S, int l1, int l2, int l3, typename V>
__device__ __forceinline__ void forward_diagonal(const T* wq, int lanes, const T* buffer, T c, const V* xl, V* al) {
  constexpr int NP = PK::NP;
  T y[8];
  edge_attributes<S, l2>(buffer, y);
  V w2[NP];
  lane_load<PK, T>(wq, lanes, w2);
  const V scale = bcast_packet(l2 == 0 ? c * y[0] : c, V{});
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    V cw = vmul(scale, w2[p]);
    if constexpr (l2 == 0) {
#pragma unroll
      for (int k = 0; k < 2 * l3 + 1; ++k) al[k * NP + p] = vfma(cw, xl[k * NP + p], al[k * NP + p]);
    } else if constexpr (l1 == 0) {
      cw = vmul(cw, xl[p]);
#pragma unroll
      for (int k = 0; k < 2 * l3 + 1; ++k) al[k * NP + p] = vfma(bcast_packet(y[k], V{}), cw, al[k * NP + p]);
    } else {
      V sum = vmul(bcast_packet(y[0], V{}), xl[p]);
#pragma unroll
      for (int i = 1; i < 2 * l1 + 1; ++i) sum = vfma(bcast_packet(y[i], V{}), xl[i * NP + p], sum);
      al[p] = vfma(cw, sum, al[p]);
    }
  }
}
// All paths of an edge, for a lane's channels.  ws: its first weight; xs: the edge's row of x.
template <typename T, typename PK, typename S, typename V>
__device__ __forceinline__ void forward_edge(const T* ws, const T* xs, int ch, int own, int lanes, const T* buffer,
                                             const T* coef, V* acc) {
  constexpr int NP = PK::NP;
  static_for<0, 4>([&](auto l1c) {
    constexpr int l1 = decltype(l1c)::value;
    if constexpr (S::has(S::MX, l1)) {
      constexpr int d1 = 2 * l1 + 1;
      V xl[d1 * NP];
      lane_load_block<PK, T, d1>(xs + ch * S::xoff(l1) + own * d1, lanes, xl);
      static_for<0, 4>([&](auto l3c) {
        constexpr int l3 = decltype(l3c)::value;
        static_for<0, 4>([&](auto l2c) {
          constexpr int l2 = decltype(l2c)::value;
          if constexpr (S::ok(l1, l2, l3)) {
            const T* wq = ws + S::rank(l1, l2, l3) * ch;
            V* al = &acc[S::ooff(l3) * NP];
            if constexpr (S::diagonal(l1, l2, l3))
              forward_diagonal<T, PK, S, l1, l2, l3>(wq, lanes, buffer, coef[S::coff(l1, l2, l3)], xl, al);
            else
              forward_path<T, PK, S, l1, l2, l3>(wq, lanes, buffer, xl, al);
          }
        });
      });
    }
  });
}

// The end of a launch in equal parts.  Not inlined, and with nothing of the kernel's own handed over: else the compiler schedules the
// loop over the edges differently.  Forward, inlined and like this: (1, 1, 1), 64 channels, 4.3 M edges 864 -> 796 us; FP64 (2, 3, 3),
// 64 channels, 0.66 M edges 1,285 -> 1,180.
template <typename T, int CPL, typename S, bool FULL, bool SLICED>
static __device__ __noinline__ void merge_forward(const EdgeFwdParams<T>& P) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* const rings = reinterpret_cast<T*>(smem_raw);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(rings + static_cast<size_t>(P.teams) * P.ring_elems +
                                                     static_cast<size_t>(P.teams) * (2 * EdgeFwd<T, CPL, S>::m_elems));
  unsigned* const tickets = reinterpret_cast<unsigned*>(bars + P.teams * kEdgeMaxStages);
  const int ch = FULL ? 32 * CPL : P.ch, row_ch = SLICED ? P.row_ch : ch, first_ch = SLICED ? static_cast<int>(blockIdx.y) * ch : 0;
  merge_parts(reinterpret_cast<TeamPart*>(tickets + P.teams), P.teams, P.dst_rowptr, rings, P.ring_elems, S::OD * ch, [&](int row, int a) {
    return P.out + static_cast<int64_t>(row) * (S::OD * row_ch) + (SLICED ? slice_element<S>(S::MO, a, ch, row_ch, first_ch) : a);
  });
}

// FULL: one warp per edge and 32 * CPL channels, known to the compiler.  SLICED: these are a slice of wider blocks.
template <typename T, int CPL, typename S, bool FULL, bool SLICED>
__global__ void __launch_bounds__(EdgeFwd<T, CPL, S>::template warps<FULL> * 32, 1)
    edge_fwd_kernel(const __grid_constant__ EdgeFwdParams<T> P) {
  using K = EdgeFwd<T, CPL, S>;
  using PK = EdgePacket<T, CPL, edge_spread(S::XD, S::paths)>;
  using V = typename PK::V;
  constexpr int NP = PK::NP;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  let_next_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team_warps = FULL ? 1 : P.team_warps;
  const int team = FULL ? warp : warp / team_warps, member = warp - team * team_warps;
  const int ch = FULL ? 32 * CPL : P.ch, stages = P.stages;
  const int W = S::paths * ch, X = S::XD * ch, O = S::OD * ch;
  const int stage_elems = W + X;
  static_assert(FULL || !SLICED, "a slice is one warp's full set of channels");
  const int row_ch = SLICED ? P.row_ch : ch, first_ch = SLICED ? static_cast<int>(blockIdx.y) * ch : 0;
  const int w_row = S::paths * row_ch, x_row = S::XD * row_ch, o_row = S::OD * row_ch;  // in memory
  unsigned* const counters = P.tile_counters + (SLICED ? 2 * blockIdx.y : 0);

  T* ring = reinterpret_cast<T*>(smem_raw) + static_cast<size_t>(team) * P.ring_elems;
  T* mbuf = reinterpret_cast<T*>(smem_raw) + static_cast<size_t>(P.teams) * P.ring_elems +
            static_cast<size_t>(team) * (2 * K::m_elems);
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<T*>(smem_raw) +
                                               static_cast<size_t>(P.teams) * P.ring_elems +
                                               static_cast<size_t>(P.teams) * (2 * K::m_elems)) +
                   team * kEdgeMaxStages;
  unsigned* tickets = reinterpret_cast<unsigned*>(bars + (P.teams - team) * kEdgeMaxStages);
  TeamPart* const kept = reinterpret_cast<TeamPart*>(tickets + P.teams);
  if (member == 0 && lane == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&bars[s], 1);
    fence_barrier_init();
  }

  MatrixProgram<T, S> program;
  program.load(P.prog_c, P.prog_j, lane, member, team_warps);
  __syncthreads();
  wait_for_previous();

  const int cpw = ch / team_warps;  // channels of this warp
  const int lanes = FULL ? 32 : cpw / CPL;
  const int own = FULL ? lane_first<PK>(lane) : member * cpw + lane_first<PK>(min(lane, lanes - 1));  // first channel of this lane
  const bool active = FULL || lane < lanes;
  const bool leader = member == 0 && lane == 0;
  const bool issuing = SLICED || leader;  // the pieces of a slice are copied by all lanes
  const uint32_t w_bytes = static_cast<uint32_t>(W * sizeof(T)), x_bytes = static_cast<uint32_t>(X * sizeof(T));
  auto issue = [&](int edge, int s_node, int s) {  // by the issuing lanes
    const int64_t e = edge;
    T* to = ring + static_cast<size_t>(s) * stage_elems;
    if constexpr (SLICED) {
      if (lane == 0) mbar_arrive_expect_tx(&bars[s], w_bytes + x_bytes);
      __syncwarp();
      for (int p = lane; p < S::paths; p += 32)
        bulk_copy_g2s_hint(to + p * ch, P.w + e * w_row + p * row_ch + first_ch, static_cast<uint32_t>(ch * sizeof(T)), &bars[s],
                           l2_policy_evict_first());
      static_for<0, 4>([&](auto lc) {
        constexpr int l = decltype(lc)::value, d = 2 * l + 1;
        if constexpr (S::has(S::MX, l)) {
          if (lane == l)
            bulk_copy_g2s(to + W + ch * S::xoff(l), P.x + static_cast<int64_t>(s_node) * x_row + row_ch * S::xoff(l) + first_ch * d,
                          static_cast<uint32_t>(ch * d * sizeof(T)), &bars[s]);
        }
      });
    } else {
      mbar_arrive_expect_tx(&bars[s], w_bytes + x_bytes);
      bulk_copy_g2s_hint(to, P.w + e * W, w_bytes, &bars[s], l2_policy_evict_first());
      bulk_copy_g2s(to + W, P.x + static_cast<int64_t>(s_node) * X, x_bytes, &bars[s]);
    }
  };

  V acc[S::OD * NP];
  int s = 0;            // stage of the next edge; the ring keeps turning from one row to the next
  uint32_t parity = 0;  // phase of that stage's barrier
  bool alive = true;
  int buf = 0;          // matrix buffer of the current edge

  const bool grouped = P.group > 1, parts = P.parts != 0;
  int open_row = -1;  // whose sum goes to shared memory, to be added to what the next team has of it
  const int in_group = team % P.group, group_id = team / P.group, groups = P.teams / P.group;
  // edges and rows fit 31 bits, and every register counts
  const unsigned total = gridDim.x * static_cast<unsigned>(grouped ? groups : P.teams);
  // a group takes every total-th row; a team's first tile is its own number, and further ones come from a counter, one
  // ahead of need, so that a team that started late or met long rows simply takes fewer
  unsigned unit = grouped ? blockIdx.x + gridDim.x * group_id : blockIdx.x * P.teams + team;
  const unsigned units = parts ? total : static_cast<unsigned>(grouped ? P.num_rows : P.num_tiles);
#pragma unroll 1
  while (unit < units) {
    unsigned unit_after = unit + total;
    int n = static_cast<int>(unit), n_hi = n + 1, e, e_end;
    if (parts) {
      const TeamPart part = team_part(P.dst_rowptr, P.num_rows, P.num_edges, P.rows_per_edge, team, P.teams, lane);
      n = part.n;
      n_hi = part.n_hi;
      e = part.pos;
      e_end = part.end;
      open_row = part.open_row();
      if (leader) kept[team] = part;  // for the end of the launch
    } else if (!grouped) {
      if (team_warps == 1) {
        unit_after = static_cast<unsigned>(take_tile(counters, total, lane));
      } else {
        if (leader) tickets[team] = atomicAdd(&counters[0], 1u);
        team_sync(team_warps, team);
        unit_after = total + tickets[team];
        team_sync(team_warps, team);
      }
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
    // all stages are empty here: fill them in ring order from the current one
    if (issuing) {
      for (int d = 0, stage = s; d < stages; ++d) {
        if (e + d < e_end) issue(e + d, P.src[e + d], stage);
        if (++stage == stages) stage = 0;
      }
    }
    // source node of the edge that is issued in the next iteration, attributes of the next edge
    int src_ahead = issuing && e + stages < e_end ? P.src[e + stages] : 0;
    T y_next = lane < S::YD && e < e_end ? P.y[static_cast<int64_t>(e) * S::YD + lane] : T(0);
    program.run(y_next, mbuf + buf * K::m_elems, lane, member, team_warps);
    if (lane < S::YD && e + 1 < e_end) y_next = P.y[static_cast<int64_t>(e + 1) * S::YD + lane];
    team_sync(team_warps, team);
#pragma unroll 1
    for (; n < n_hi; ++n) {
      const int row_end = min(P.dst_rowptr[n + 1], e_end);
#pragma unroll
      for (int a = 0; a < S::OD * NP; ++a) acc[a] = zero_packet<V>();
#pragma unroll 1
      for (; e < row_end; ++e) {
        if (!edge_wait(&bars[s], parity, alive)) {
          if (lane == 0) atomicExch(P.status, 1);
          alive = false;
        }
        const T* ws = ring + static_cast<size_t>(s) * stage_elems + own;
        const T* xs = ring + static_cast<size_t>(s) * stage_elems + W;
        program.run(y_next, mbuf + (buf ^ 1) * K::m_elems, lane, member, team_warps);  // of the next edge; of no use after the last one
        if (lane < S::YD && e + 2 < e_end) y_next = P.y[static_cast<int64_t>(e + 2) * S::YD + lane];
        const T* m_now = mbuf + buf * K::m_elems;
        forward_edge<T, PK, S>(ws, xs, ch, own, lanes, m_now, P.coef, acc);
        buf ^= 1;
        fence_async_shared();         // what was read of this stage, before it is refilled
        team_sync(team_warps, team);  // every lane is done with it and with the matrices
        if (issuing && e + stages < e_end) {
          issue(e + stages, src_ahead, s);
          if (e + stages + 1 < e_end) src_ahead = P.src[e + stages + 1];
        }
        if (++s == stages) {
          s = 0;
          parity ^= 1u;
        }
      }
      if (active) {
        const bool rest = grouped || n == open_row;
        T* to = rest ? ring : P.out + static_cast<int64_t>(n) * o_row;
        const int block = rest ? ch : row_ch, at = rest ? own : first_ch + own;
        static_for<0, 4>([&](auto l3c) {
          constexpr int l3 = decltype(l3c)::value, d3 = 2 * l3 + 1;
          if constexpr (S::has(S::MO, l3))
            lane_store_block<PK, T, d3>(to + block * S::ooff(l3) + at * d3, lanes, &acc[S::ooff(l3) * NP],
                                        !rest && P.accumulate);
        });
      }
    }
    if (grouped) {  // the parts of the row, in order
      const int barrier = 1 + (team_warps > 1 ? P.teams : 0) + group_id;
      const int threads = P.group * team_warps * 32;
      const T* parts = reinterpret_cast<const T*>(smem_raw) + static_cast<size_t>(group_id * P.group) * P.ring_elems;
      named_barrier(barrier, threads);
      T* to = P.out + static_cast<int64_t>(unit) * o_row;
      for (int a = static_cast<int>(threadIdx.x) - group_id * threads; a < O; a += threads) {
        T sum = parts[a];
        for (int g = 1; g < P.group; ++g) sum += parts[static_cast<size_t>(g) * P.ring_elems + a];
        T* put = to + (SLICED ? slice_element<S>(S::MO, a, ch, row_ch, first_ch) : a);
        *put = P.accumulate ? *put + sum : sum;
      }
      fence_async_shared();  // threads have written and read the ring; its next users are bulk copies
      named_barrier(barrier, threads);
    }
    unit = unit_after;
  }
  if (parts) {
    merge_forward<T, CPL, S, FULL, SLICED>(P);
  } else if (!grouped && member == 0) {
    leave_tiles(counters, total, lane);
  }
  if (!alive)  // let copies that are still in flight land before the CTA's shared memory is released
    for (int d = 0; d < stages; ++d) edge_wait(&bars[d], d < s ? parity : parity ^ 1u, false);
}

// As many teams as fit the shared memory with three stages each (two, if they are then more).
template <typename T, int CPL, typename S, bool FULL>
EdgeLaunch edge_fwd_launch(const Tuning& tuning, const EdgeLanes& lanes, int ch, int max_smem) {
  using K = EdgeFwd<T, CPL, S>;
  const size_t stage = static_cast<size_t>(S::paths + S::XD) * ch * sizeof(T);
  const size_t row = static_cast<size_t>(S::OD) * ch * sizeof(T);
  EdgeLaunch launch;
  const int max_teams = capped_warps(tuning, K::template warps<FULL>) / lanes.team_warps;
  for (int teams = max_teams; teams >= 1 && launch.warps == 0; --teams) {
    // With more than twenty teams of three channels per lane and the long gathered rows of (1, 1, 0) the plain loads of attributes and
    // indices wait behind the bulk copies: 96 channels, 0.26 M edges, 16 / 20 / 22 / 24 teams 59 / 55 / 94 / 121 us.  (0, 1, 1), half as many bytes
    // in flight, 59 / 53 / 53 / 50.
    if (CPL == 3 && teams > 16 && 3 * max_teams * stage > 150 * 1024) continue;
    for (int stages = teams * 2 > max_teams ? 3 : kEdgeMaxStages; stages >= 2; --stages) {
      const size_t ring = (std::max(stages * stage, row) + 127) / 128 * 128;
      const size_t bytes = teams * (ring + K::team_bytes + kEdgeMaxStages * sizeof(uint64_t) + sizeof(unsigned) + sizeof(TeamPart));
      if (bytes > static_cast<size_t>(max_smem)) continue;
      launch.warps = teams * lanes.team_warps;
      launch.stages = stages;
      launch.bytes = bytes;
      launch.team_elems = static_cast<int>(ring / sizeof(T));
      break;
    }
  }
  return launch;
}

}  // namespace edgek
}  // namespace luna
