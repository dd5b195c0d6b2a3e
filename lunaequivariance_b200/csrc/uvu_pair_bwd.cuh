// Backward kernel for narrow blocks: a warp walks two edges at a time, one on each half of its lanes (uvu_pair_fwd.cuh says
// why, and how pairs meet the ends of rows).  The arithmetic of an edge, the staging and the order of events are those of
// uvu_edge_bwd.cuh; a lane keeps the row of its own half's edge in registers.
#pragma once

#include "uvu_edge_bwd.cuh"
#include "uvu_pair_fwd.cuh"

namespace luna {
namespace edgek {

template <typename T, int CPL, typename S, bool WX, bool WM, bool WY>
struct PairBwd {
  using Edge = EdgeBwd<T, CPL, S, WX, WM, WY>;
  using Packet = PkT<T, CPL, UsePairs<T, CPL>::value>;
  static constexpr int m_elems = WM ? S::m_elems : 0;  // of each half
  static constexpr int red_rows = Edge::red_rows, red_pass = Edge::red_pass, red_row = Edge::red_row;
  static constexpr int warp_elems = 2 * m_elems + (WY ? red_pass * red_row : 0);
  static constexpr int program_regs = WM ? 4 * S::m_rounds * Edge::words + S::m_rounds + 1 : 0;
  static constexpr int registers = Edge::state + program_regs + 44;
  static constexpr int max_warps = warps_for(registers);
};

// 16 * CPL channels.  DST: rows by destination (S, x and g exchanged).  ADD: gw alone, added to; w names gw.
template <typename T, int CPL, typename S, bool WX, bool WM, bool WY, bool DST, bool ADD>
__global__ void __launch_bounds__(PairBwd<T, CPL, S, WX, WM, WY>::max_warps * 32, 1)
    pair_bwd_kernel(const __grid_constant__ EdgeBwdParams<T, EdgeBwd<T, CPL, S, WX, WM, WY>::terms> P) {
  using K = PairBwd<T, CPL, S, WX, WM, WY>;
  using PK = PkT<T, CPL, UsePairs<T, CPL>::value>;
  using V = typename PK::V;
  constexpr int NP = PK::NP;
  static_assert(!ADD || (WM && !WX && !WY), "the weights' place in a stage must be free");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  let_next_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4, place = lane & 15;
  constexpr int ch = 16 * CPL, lanes = 16, W = S::paths * ch, X = S::XD * ch, O = S::OD * ch, half_elems = pair_half<PK>(W + O), stage_elems = 2 * half_elems;
  const int stages = P.stages, own = lane_first<PK>(place);

  T* const base = reinterpret_cast<T*>(smem_raw);
  T* const ring = base + static_cast<size_t>(warp) * P.team_elems;
  T* const warp_mem = base + static_cast<size_t>(P.teams) * P.team_elems + static_cast<size_t>(warp) * K::warp_elems;
  T* const mbuf = warp_mem + half * K::m_elems;
  T* const red = warp_mem + 2 * K::m_elems;
  uint64_t* const full =
      reinterpret_cast<uint64_t*>(base + static_cast<size_t>(P.teams) * (P.team_elems + K::warp_elems)) + warp * kEdgeMaxStages;
  TeamPart* const kept = reinterpret_cast<TeamPart*>(full + (P.teams - warp) * kEdgeMaxStages);

  if (lane == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&full[s], 2);  // both halves' copies
    fence_barrier_init();
  }
  HalfMatrixProgram<T, S> program;
  if constexpr (WM) program.load(P.prog_c, P.prog_j, place);
  __syncthreads();
  wait_for_previous();

  const bool issuing = place == 0;  // a half's copies are its first lane's
  const bool want_x = WX && P.gx != nullptr, storing = WM && P.gw != nullptr;
  const uint32_t w_bytes = P.need_w ? static_cast<uint32_t>(W * sizeof(T)) : 0u, g_bytes = static_cast<uint32_t>(O * sizeof(T));

  auto load_stage = [&](int e, int d, int st) {  // by the issuing lane of either half, of its edge; e < 0: none
    T* to = ring + static_cast<size_t>(st) * stage_elems + half * half_elems;
    mbar_arrive_expect_tx(&full[st], e >= 0 ? w_bytes + g_bytes : 0u);
    if (e < 0) return;
    if (w_bytes) bulk_copy_g2s_hint(to, P.w + static_cast<int64_t>(e) * W, w_bytes, &full[st], l2_policy_evict_first());
    bulk_copy_g2s(to + W, P.g + static_cast<int64_t>(d) * O, g_bytes, &full[st]);
  };

  V xr[S::XD * NP], gxr[WX ? S::XD * NP : 1], gy2[WY ? S::YD : 1];
  if constexpr (WX) {
#pragma unroll
    for (int a = 0; a < S::XD * NP; ++a) gxr[a] = zero_packet<V>();
  }
  int st = 0;
  uint32_t parity = 0;
  bool alive = true;

  auto unit_body = [&](auto l3c, T* wrow) {
    constexpr int l3 = decltype(l3c)::value, d3 = 2 * l3 + 1;
    V g2[d3 * NP];
    lane_load_block<PK, T, d3>(wrow + W + ch * S::ooff(l3) + own * d3, lanes, g2);
    static_for<0, 4>([&](auto l1c) {
      constexpr int l1 = decltype(l1c)::value;
      static_for<0, 4>([&](auto l2c) {
        constexpr int l2 = decltype(l2c)::value;
        if constexpr (S::ok(l1, l2, l3))
          backward_path<T, PK, S, l1, l2, l3, WX, WM, WY, ADD, V>(wrow + S::rank(l1, l2, l3) * ch + own, lanes, storing, xr, gxr,
                                                                gy2, g2, mbuf, P.term, P.coef);
      });
    });
  };
  const bool parts = P.parts != 0, every_row = P.every_row != 0;
  int open_row = -1;  // whose sum goes to shared memory, to be added to what the next team has of it
  const bool acc_x = P.acc_x != 0;
  // gxr of one half to row n, added to what is there if `add`, and zero again
  auto store = [&](int n, int by, bool add) {
    if constexpr (WX) {
      if (half == by) {
        if (want_x) {
          const bool rest = n == open_row;
          T* to = rest ? ring : P.gx + static_cast<int64_t>(n) * X;
          static_for<0, 4>([&](auto l1c) {
            constexpr int l1 = decltype(l1c)::value, d = 2 * l1 + 1;
            if constexpr (S::has(S::MX, l1))
              lane_store_block<PK, T, d>(to + ch * S::xoff(l1) + own * d, lanes, &gxr[S::xoff(l1) * NP], !rest && add);
          });
        }
#pragma unroll
        for (int a = 0; a < S::XD * NP; ++a) gxr[a] = zero_packet<V>();
      }
    }
  };
  auto gather = [&] {  // both halves' sums to the first one
    if constexpr (WX) {
#pragma unroll
      for (int a = 0; a < S::XD * NP; ++a) {
        const V other = shfl_xor_packet(gxr[a], 16);
        gxr[a] = half == 0 ? vadd(gxr[a], other) : zero_packet<V>();
      }
    }
  };

  const unsigned total = gridDim.x * static_cast<unsigned>(P.teams);
  unsigned unit = blockIdx.x * P.teams + warp;
  const unsigned units = parts ? total : static_cast<unsigned>(P.num_tiles);
  int seen_row = 0, seen_pos = 0;  // a row boundary this warp has seen, and where its edges begin
#pragma unroll 1
  while (unit < units) {
    unsigned unit_after = unit + total;
    int n, n_hi, pos, p_end;
    if (parts) {
      const TeamPart part = team_part(P.src_rowptr, P.num_rows, P.num_edges, P.rows_per_edge, warp, P.teams, lane);
      n = part.n;
      n_hi = part.n_hi;
      pos = part.pos;
      p_end = part.end;
      open_row = part.open_row();
      if (lane == 0) kept[warp] = part;  // for the end of the launch
    } else {
      unit_after = static_cast<unsigned>(take_tile(P.tile_counters, total, lane));
      if (P.tile_rows > 0) {
        const int64_t first = unit * P.tile_rows, end = first + P.tile_rows;
        n = static_cast<int>(first);
        n_hi = static_cast<int>(end < P.num_rows ? end : P.num_rows);
      } else {
        const int64_t guess =
            seen_row + static_cast<int64_t>(static_cast<float>(unit * P.tile_edges - seen_pos) * P.rows_per_edge);
        n = unit == 0 ? 0
                      : static_cast<int>(warp_lower_bound_guess(P.src_rowptr, P.num_rows, unit * P.tile_edges, guess, lane));
        n_hi = static_cast<int>(unit + 1 == units ? P.num_rows
                                                  : warp_lower_bound_near(P.src_rowptr, P.num_rows, (unit + int64_t(1)) * P.tile_edges,
                                                                          n, lane));
      }
    }
    unit = unit_after;
    if (n >= n_hi) continue;  // a row with more edges than a tile spans several tile numbers
    if (!parts) {
      pos = P.src_rowptr[n];
      p_end = P.src_rowptr[n_hi];
      seen_row = n_hi;
      seen_pos = p_end;
    }
    // of this half: ids of the edges of the current and the next four pairs (-1: none), destinations of the first four
    auto id_at = [&](int p) { return p < p_end ? (DST ? p : P.edge_ids[p]) : -1; };
    auto dst_of = [&](int e) { return e >= 0 ? P.dst[e] : 0; };
    int e0 = id_at(pos + half), e1 = id_at(pos + half + 2), e2 = id_at(pos + half + 4), e3 = id_at(pos + half + 6),
        e4 = id_at(pos + half + 8);
    int d0 = dst_of(e0), d1 = dst_of(e1), d2 = dst_of(e2), d3n = dst_of(e3);
    if (issuing) {
      for (int k = 0, stage = st; k < stages; ++k) {
        if (pos + 2 * k < p_end) load_stage(k == 0 ? e0 : (k == 1 ? e1 : e2), k == 0 ? d0 : (k == 1 ? d1 : d2), stage);
        if (++stage == stages) stage = 0;
      }
    }
    T y_next = T(0);
    if constexpr (WM) {
      if (place < S::YD && e0 >= 0) y_next = P.y[static_cast<int64_t>(e0) * S::YD + place];
      program.run(y_next, mbuf, place);
      if (place < S::YD && e1 >= 0) y_next = P.y[static_cast<int64_t>(e1) * S::YD + place];
    }
    __syncwarp();
    int refill_stage = -1;  // a stage whose rows are on their way back, to be refilled with the pair `stages` after it
    int pe = min(P.src_rowptr[n + 1], p_end), have = -1;  // the row whose x this half holds
    // the row after n that holds position `to`, or the next one if rows without edges are written too
    auto next_row = [&](int to) {
      ++n;
      if (!every_row && P.src_rowptr[n + 1] <= to)
        n = static_cast<int>(warp_lower_bound(P.src_rowptr, P.num_rows, to + int64_t(1), lane)) - 1;
      pe = min(P.src_rowptr[n + 1], p_end);
    };
    if (!every_row && pos >= pe && pos < p_end) {  // the tile's first rows have no edges
      --n;
      next_row(pos);
    }
#pragma unroll 1
    for (; pos < p_end; pos += 2) {
#pragma unroll 1
      while (pos >= pe) {  // rows that ended before this pair
        gather();
        store(n, 0, acc_x);
        next_row(pos);
      }
      const bool straddle = pos + 1 >= pe && pos + 1 < p_end;  // the second edge is of a later row
      int mine = n;
      if (straddle) {
        store(n, 1, acc_x);
        const int first_row = n;
#pragma unroll 1
        do {
          next_row(pos + 1);
        } while (pos + 1 >= pe);
        mine = half == 0 ? first_row : n;
        if (WX && every_row && half == 0 && want_x && !P.acc_x) {  // rows without edges in between
#pragma unroll 1
          for (int row = first_row + 1; row < n; ++row)
            for (int a = place; a < X; a += 16) P.gx[static_cast<int64_t>(row) * X + a] = T(0);
        }
      }
      if (mine != have) {
        have = mine;
        static_for<0, 4>([&](auto l1c) {
          constexpr int l1 = decltype(l1c)::value;
          if constexpr (S::has(S::MX, l1)) {
            constexpr int d = 2 * l1 + 1;
            lane_load_block<PK, T, d>(P.x + static_cast<int64_t>(mine) * X + ch * S::xoff(l1) + own * d, lanes, &xr[S::xoff(l1) * NP]);
          }
        });
      }
      if constexpr (WY) {
#pragma unroll
        for (int j = 0; j < S::YD; ++j) gy2[j] = zero_packet<V>();
      }
      if (!edge_wait(&full[st], parity, alive)) {
        if (lane == 0) atomicExch(P.status, 3);
        alive = false;
      }
      T* const wrow = ring + static_cast<size_t>(st) * stage_elems + half * half_elems;
      const bool valid = e0 >= 0;
      static_for<0, 4>([&](auto l3c) {
        constexpr int l3 = decltype(l3c)::value;
        if constexpr (S::has(S::MO, l3)) {
          if (valid) unit_body(l3c, wrow);
          if constexpr (S::ooff(l3) == 0) {  // after the first degree: the rows sent back have left their stage by now
            if (refill_stage >= 0 && issuing) {
              bulk_wait_group_read_all();
              if (pos + 2 * (stages - 1) < p_end) load_stage(stages == 2 ? e1 : e2, stages == 2 ? d1 : d2, refill_stage);
            }
            refill_stage = -1;
          }
        }
      });
      fence_async_shared();  // gradient writes, before the bulk store reads the stage, and reads, before it is refilled
      __syncwarp();          // every lane is done with the stage and the matrices
      if (issuing) {
        if (storing) {
          if (valid) {
            T* row = P.gw + static_cast<int64_t>(e0) * W;
            if (P.acc_w)
              bulk_reduce_add_s2g(row, wrow, static_cast<uint32_t>(W * sizeof(T)));
            else
              bulk_copy_s2g_hint(row, wrow, static_cast<uint32_t>(W * sizeof(T)), l2_policy_evict_first());
            bulk_commit_group();
          }
        } else if (pos + 2 * stages < p_end) {
          load_stage(stages == 2 ? e2 : e3, stages == 2 ? d2 : d3n, st);
        }
      }
      if (storing) refill_stage = st;
      if constexpr (WM) {
        program.run(y_next, mbuf, place);
        if (place < S::YD && e2 >= 0) y_next = P.y[static_cast<int64_t>(e2) * S::YD + place];
      }
      if constexpr (WY) {
        // the lanes' partial gy rows through the reduction tile: entries 2r and 2r + 1 in tile row r; two lanes of each half
        // sum a row's 16, eight each
        constexpr int passes = (K::red_rows + K::red_pass - 1) / K::red_pass;
        static_for<0, passes>([&](auto qc) {
          constexpr int first = decltype(qc)::value * K::red_pass;
          constexpr int rows = K::red_rows - first < K::red_pass ? K::red_rows - first : K::red_pass;
          static_for<0, rows>([&](auto rc) {
            constexpr int j = 2 * (first + decltype(rc)::value);
            Vec<T, 2> pr;
            pr.a[0] = hsum(gy2[j]);
            if constexpr (j + 1 < S::YD) {
              pr.a[1] = hsum(gy2[j + 1]);
            } else {
              pr.a[1] = T(0);
            }
            *reinterpret_cast<Vec<T, 2>*>(red + decltype(rc)::value * K::red_row + lane * 2) = pr;
          });
          __syncwarp();
          constexpr int per = 16 / static_cast<int>(sizeof(T));
          const int r = min(lane & 7, rows - 1);
          const T* seg = red + r * K::red_row + (lane >> 3) * 16;
          T s0 = T(0), s1 = T(0);
#pragma unroll
          for (int v = 0; v < 16 / per; ++v) {
            const Vec<T, per> q = reinterpret_cast<const Vec<T, per>*>(seg)[v];
#pragma unroll
            for (int c = 0; c < per; c += 2) {
              s0 += q.a[c];
              s1 += q.a[c + 1];
            }
          }
          s0 += __shfl_xor_sync(0xffffffffu, s0, 8);
          s1 += __shfl_xor_sync(0xffffffffu, s1, 8);
          if (place < rows && valid) {
            const int j = 2 * (first + place);
            T* to = P.gy + static_cast<int64_t>(e0) * S::YD + j;
            to[0] = P.acc_y ? to[0] + s0 : s0;
            if (j + 1 < S::YD) to[1] = P.acc_y ? to[1] + s1 : s1;
          }
          __syncwarp();
        });
      } else {
        __syncwarp();
      }
      if (straddle) store(mine, 0, true);  // the first half's row ended; the second half began row n
      e0 = e1;
      e1 = e2;
      e2 = e3;
      e3 = e4;
      d0 = d1;
      d1 = d2;
      d2 = d3n;
      d3n = dst_of(e3);
      e4 = id_at(pos + half + 10);
      if (++st == stages) {
        st = 0;
        parity ^= 1u;
      }
    }
    if constexpr (WX) {
      if (open_row >= 0) {  // the last row's sum goes to shared memory: bulk stores must have read the ring
        if (issuing) bulk_wait_group_read_all();
        __syncwarp();
      }
      gather();
      if (every_row) {
#pragma unroll 1
        for (; n < n_hi; ++n) store(n, 0, acc_x);
      } else if (p_end > P.src_rowptr[n]) {
        store(n, 0, acc_x);
      }
    }
    if (WM && issuing) bulk_wait_group_read_all();  // the next rows' copies reuse the stages
  }
  if (!parts) {
    leave_tiles(P.tile_counters, total, lane);
  } else if constexpr (WX) {
    if (want_x)
      merge_parts(kept, P.teams, P.src_rowptr, base, P.team_elems, X,
                  [&](int row, int a) { return P.gx + static_cast<int64_t>(row) * X + a; });
  }
  if (WM && issuing) bulk_wait_group_read_all();
  if (!alive)  // let copies that are still in flight land before the CTA's shared memory is released
    for (int d = 0; d < stages; ++d) edge_wait(&full[d], d < st ? parity : parity ^ 1u, false);
}

// K: the PairBwd of the kernel.
template <typename T, typename S, typename K>
EdgeLaunch pair_bwd_launch(const Tuning& tuning, int ch, int max_smem) {
  const size_t stage = 2 * static_cast<size_t>(pair_half<typename K::Packet>((S::paths + S::OD) * ch)) * sizeof(T), row = static_cast<size_t>(S::XD) * ch * sizeof(T);
  EdgeLaunch launch;
  for (int warps = capped_warps(tuning, K::max_warps); warps >= 1 && launch.warps == 0; --warps)
    for (int stages = 3; stages >= 2; --stages) {
      const size_t ring = (std::max(stages * stage, row) + 127) / 128 * 128;
      const size_t bytes = warps * (ring + K::warp_elems * sizeof(T) + kEdgeMaxStages * sizeof(uint64_t) + sizeof(TeamPart));
      if (bytes > static_cast<size_t>(max_smem)) continue;
      launch.warps = warps;
      launch.stages = stages;
      launch.bytes = bytes;
      launch.team_elems = static_cast<int>(ring / sizeof(T));
      break;
    }
  return launch;
}

// Whether the kernels of 16 * CPL channels walk two edges at a time, with CPL channels on each lane of a half warp: what is
// compiled and what is chosen.  One to three channels per lane, if the rows of two pairs leave room for eight warps.  With fewer it
// loses: FP64, 32 channels, degrees (2, 3, 3), six warps, all gradients of 0.4 M edges 1.30 -> 1.75 ms.  Four FP32 channels for shapes
// whose paths all have a degree of zero and whose degrees end at 2.  The others have more arithmetic in an edge than beside it, or
// too many registers: (2, 2, 2), 64 channels, all gradients of 0.24 M edges 0.345 -> 0.391 ms with two at a time; (0, 3, 3), forward of
// 0.8 M edges 0.249 -> 0.475.  Of these the forward at degree 2 only: one edge and two, forward / all gradients / dL/dy / dL/dw, 0.8 M
// edges: (1, 1, 1) 165 / 555 / 322 / 416 -> 174 / 380 / 194 / 260 us; (1, 1, 0) 143 / 476 / 330 / 250 -> 156 / 310 / 188 / 231; (0, 2, 2),
// 1.05 M edges, 282 / 710 / 422 / 518 -> 215 / 478 / 250 / 332; (2, 2, 0) 233 / 545 / 370 / 424 -> 176 / 439 / 215 / 268.
// Three channels per lane with six or seven warps: for one gradient alone, whose state is small.  48 channels, one edge and two,
// dL/dy / dL/dw: (2, 3, 3), 0.4 M edges 505 / 519 -> 432 / 476 us; FP64 (0, 3, 3), 0.4 M edges, 336 / 287 -> 248 / 214; but forward
// and all gradients of (3, 3, 3), 0.2 M edges, 289 / 756 -> 333 / 1,245, and FP64 (3, 3, 0), all, 661 -> 772.
// Two channels per lane with eight warps, where one edge with one channel per lane has sixteen, or where the state is far above the
// registers' share: shapes with coupling matrices, several gradients.  32 channels, two edges and one: FP32 (3, 3, 3), 0.4 M
// edges, all gradients 1,123 -> 897 us, dL/dx with dL/dw 709 -> 602, output with dL/dw 700 -> 563; (2, 3, 3), all, 678 -> 595; FP64
// (2, 2, 2), 0.4 M edges, 517 -> 488 and 504 -> 432, but all, eight warps and twelve, 617 -> 682.
template <typename T, typename S, bool WY>
constexpr bool pair_crowded() {
  using Two = PairBwd<T, 2, S, true, true, WY>;
  return Two::max_warps == 8 && (EdgeBwd<T, 1, S, true, true, WY>::template warps<true> >= 16 || Two::registers > 190);
}
template <typename T, int CPL, int ID>
constexpr bool edge_paired(EdgeUse use) {
  using S = ShapeOf<ID>;
  if (CPL == 2 && S::m_total > 0) {
    if (use == EdgeUse::kAllGradients && pair_crowded<T, S, true>()) return false;
    if (use == EdgeUse::kSums && pair_crowded<T, S, false>()) return false;
    if (use == EdgeUse::kOutputAndWeights && pair_crowded<T, Transposed<S>, false>()) return false;
  }
  constexpr int top = top_degree(S::MX | S::MO), row = S::paths + (S::XD > S::OD ? S::XD : S::OD);
  constexpr int bytes = 4 * row * 16 * CPL * static_cast<int>(sizeof(T));
  const bool four = CPL == 4 && sizeof(T) == 4 && S::m_total == 0 && (top == 2 || (top == 1 && use != EdgeUse::kForward));
  return (CPL <= 3 || four) && bytes <= (CPL == 3 && use == EdgeUse::kOneGradient ? 31 : 24) * 1024;
}

// The estimate of what a lane of the kernel needs.
template <typename T, int CPL, typename S>
constexpr int registers_of(EdgeUse use) {
  using R = Transposed<S>;
  using One = std::conditional_t<S::OD >= S::XD, R, S>;
  switch (use) {
    case EdgeUse::kForward: return EdgeFwd<T, CPL, S>::registers;
    case EdgeUse::kSums: return EdgeBwd<T, CPL, S, true, true, false>::registers;
    case EdgeUse::kOutputAndWeights: return EdgeBwd<T, CPL, R, true, true, false>::registers;
    case EdgeUse::kAllGradients: return EdgeBwd<T, CPL, S, true, true, true>::registers;
    default: return std::max(EdgeBwd<T, CPL, One, false, false, true>::registers, EdgeBwd<T, CPL, One, false, true, false>::registers);
  }
}
// Whether the kernels of one edge at a time are compiled for teams (for slices: edge_sliced).  Three channels per lane are not where the
// state is far above the registers: FP64 (3, 3, 3) but for one gradient alone, and (2, 3, 3) for output with dL/dw.
template <typename T, int CPL, int ID>
constexpr bool edge_alone(EdgeUse use) {
  return CPL != 3 || registers_of<T, CPL, ShapeOf<ID>>(use) <= (use == EdgeUse::kForward ? 255 : 280);
}

}  // namespace edgek
}  // namespace luna
