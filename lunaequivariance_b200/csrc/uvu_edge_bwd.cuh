// Backward kernel of the edge family: gx, gy and gw of one pass over the edges, grouped by source row.
//
// With the pattern of every coupling tensor compiled in, a path is a straight line over its terms t = (i, j, k):
//     s_i   = sum_k M_ik g_k                 M_ik = sum_j c_ijk y_j is made by the warp, one edge ahead
//     gx_i += w_p s_i,   gw_p = sum_i x_i s_i
//     P_ik  = sum over the lane's channels of (x_i w_p) g_k,    gy_j += c_t P_ik
// so gx stays in registers for the whole row, gy is contracted inside each lane and only its few values cross lanes,
// and the weight gradients overwrite the weights in shared memory and leave as one row with one bulk store (or one bulk
// add, when a call accumulates).
//
// Staging.  A stage holds an edge's weight row and, where two such stages per team fit, its g[dst] row.  Where they do
// not, g goes through two slots, one for the highest output degree and one for the others, each refilled for the next
// edge as soon as its degrees are done (one slot per degree: 2 % slower, for the two more waits and copies per edge).
// Weights are not read at all by calls that want gw alone: gw does not depend on them.
//
// Rows by destination.  A call that wants gw alone, or gy alone, needs no sums over rows, and the form is symmetric in x
// and g: with the roles of (x, source) and (g, destination) exchanged the rows are destinations, whose edges lie one after
// the other in memory, g stays in registers for the row and x is gathered.  Taken where a row of x is no longer than a row
// of g, which is then the smaller gather (layers that widen their degrees, first layers most of all).
//
// Output and gw in one pass.  With the roles exchanged a row's sum is the output, so the kernel of gx and gw, by destination,
// makes the output and gw together: the second order of force training wants both for the same operands, and they share the
// weights' and the features' way from memory and the products of the coupling matrices with x.
//
// gw alone, added to what is there: the rows that are added to arrive in the stages in the weights' place, and the sums
// begin with them.
//
// The coefficients of the coupling terms are kernel parameters: an operand of the FMA that uses them, instead of a load from a
// table in shared memory, whose pipe is the busiest one at (2, 2, 2) with 64 channels (61 % of its wavefronts).  All gradients,
// table and parameters: (2, 2, 2), 64 channels, 5.2 M edges 6.95 -> 6.43 ms; (3, 3, 3), 64 channels, 0.8 M edges 3.27 -> 3.01;
// (2, 3, 3), 128 channels, FP64, 0.4 M edges 5.33 -> 4.36, dL/dy alone in FP32, 1.05 M edges 2.34 -> 2.13.
//
// Every wait is bounded; a wait that runs out sets the plan's status word.
#pragma once

#include "uvu_edge.cuh"

namespace luna {
namespace edgek {

constexpr int kEdgeMaxSlots = 2;

// N: coupling terms that the kernel reads.
template <typename T, int N>
struct EdgeBwdParams {
  const T *x, *y, *w, *g;
  T *gx, *gy, *gw;
  const int *dst, *src_rowptr, *edge_ids;
  const T* prog_c;               // [2][m_total] coefficients of the two attributes a matrix entry depends on
  const unsigned short* prog_j;  // [m_total] the two attributes, 8 bits each
  T term[N];                     // coefficients of the coupling terms
  T coef[kEdgeMaxCoefs];         // of the paths with a degree of zero
  int* status;
  unsigned* tile_counters;
  int64_t num_rows, num_edges, tile_rows, tile_edges, num_tiles;  // tile_rows 0: tiles are stretches of tile_edges edges
  float rows_per_edge;
  int ch, row_ch;  // channels per block, or of a slice of it; channels per block
  int64_t gy_part;  // elements between the slices' parts of gy
  int team_warps, teams;
  int parts;      // equal parts of the edges instead of tiles
  int every_row;  // rows without edges are written too, and not cleared beforehand
  int stages, split;
  int team_elems;  // shared memory per team
  int need_w;
  int acc_x, acc_y, acc_w;
};

// What is computed: WX gx, WM the rows s_i that gx and gw are made of, WY gy.
template <typename T, int CPL, typename S, bool WX, bool WM, bool WY>
struct EdgeBwd {
  static constexpr int words = sizeof(T) / 4;
  static constexpr int pair = PkT<T, CPL, UsePairs<T, CPL>::value>::W;
  // registers for the state a lane keeps, and for its part of the matrix program
  static constexpr int state =
      (S::XD * CPL * (WX ? 2 : 1) + (WY ? S::YD * pair : 0) + (2 * S::LO + 1) * CPL) * words;
  static constexpr int program_regs = WM ? S::m_rounds * 2 * words + (S::m_rounds + 1) / 2 : 0;
  static constexpr int registers = state + program_regs + 48;  // an estimate; beyond 255 it spills hundreds of bytes
  template <bool FULL>
  static constexpr int warps = warps_for(registers, slack_for<T, S>(WM, FULL));
  // slots of g: the highest degree has one, the others share one
  static constexpr int slot_of(int l3) { return l3 == S::LO && S::ooff(S::LO) > 0 ? 1 : 0; }
  static constexpr int slots = slot_of(S::LO) + 1;
  static constexpr int slot_begin(int h) {  // first component
    for (int l = 0; l <= S::LO; ++l)
      if (S::has(S::MO, l) && slot_of(l) == h) return S::ooff(l);
    return S::OD;
  }
  static constexpr int red_rows = WY ? (S::YD + 1) / 2 : 0;
  static constexpr int red_pass = red_rows > 4 && sizeof(T) == 8 ? 4 : red_rows;  // rows of the tile at a time
  static constexpr int red_row = 64 + 16 / static_cast<int>(sizeof(T));
  static constexpr int m_elems = WM ? S::m_elems : 0;
  // per warp: coupling matrices, reduction tile and, in teams of several warps, two reduced gy rows
  static constexpr int warp_elems(int team_warps) {
    return m_elems + (WY ? red_pass * red_row + (team_warps > 1 ? 64 : 0) : 0);
  }
  static constexpr int terms = WY && S::terms > 0 ? S::terms : 1;
};

// One path for a lane's packets.  xl / gxl: the lane's x and gx packets of degree l1; g2: its g packets of degree l3;
// w2: its weights; dot receives (ADD: is added) sum_i x_i s_i; gyl: the accumulators of degree l2.  The arithmetic of a row i is issued
// in batches of independent instructions, so that the latency of one is covered by the others with few warps resident.
template <typename T, typename PK, typename S, int l1, int l2, int l3, bool WX, bool WM, bool WY, bool ADD, typename V>
__device__ __forceinline__ void edge_path(const V* xl, V* gxl, V* gyl, const V* g2, const V* w2, V* dot, const T* mbuf,
                                          const T* term) {
  constexpr int NP = PK::NP;
  using PT = CgPattern<l1, l2, l3>;
  constexpr int n = PT::n;
  constexpr int toff = S::toff(l1, l2, l3), moff = S::moff(l1, l2, l3);
  static_for<0, n>([&](auto tc) {
    constexpr int t0 = decltype(tc)::value;
    if constexpr (edge_new_row<PT>(t0)) {
      constexpr int i = PT::t[t0].i;
      constexpr int t1 = edge_row_end<PT>(t0);
      // groups of four table entries that cover the row
      constexpr int e0 = edge_entry<PT>(t0), e1 = edge_entry<PT>(t1 - 1);
      constexpr int m_lo = e0 / 4, m_hi = e1 / 4;
      T mm[WM ? 4 * (m_hi - m_lo + 1) : 1];
      if constexpr (WM)
        static_for<m_lo, m_hi + 1>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          edge_load_four<T>(mbuf + moff + 4 * q, mm + 4 * (q - m_lo));
        });
      if constexpr (WY) {
        V xw[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) xw[p] = vmul(xl[i * NP + p], w2[p]);
        V pik[e1 - e0 + 1];
        static_for<t0, t1>([&](auto uc) {
          constexpr int t = decltype(uc)::value;
          if constexpr (edge_new_entry<PT>(t)) {
            constexpr int k = PT::t[t].k, slot = edge_entry<PT>(t) - e0;
            pik[slot] = vmul(xw[0], g2[k * NP]);
#pragma unroll
            for (int p = 1; p < NP; ++p) pik[slot] = vfma(xw[p], g2[k * NP + p], pik[slot]);
          }
        });
        static_for<t0, t1>([&](auto uc) {
          constexpr int t = decltype(uc)::value;
          constexpr int j = PT::t[t].j, slot = edge_entry<PT>(t) - e0;
          gyl[j] = vfma(bcast_packet(term[toff + t], V{}), pik[slot], gyl[j]);
        });
      }
      if constexpr (WM) {
        V sa[NP];
        static_for<t0, t1>([&](auto uc) {
          constexpr int t = decltype(uc)::value;
          if constexpr (edge_new_entry<PT>(t)) {
            constexpr int k = PT::t[t].k, e = edge_entry<PT>(t), r = e - e0;
            const V c = bcast_packet(mm[e - 4 * m_lo], V{});
#pragma unroll
            for (int p = 0; p < NP; ++p) {
              if constexpr (r == 0) {
                sa[p] = vmul(c, g2[k * NP + p]);
              } else {
                sa[p] = vfma(c, g2[k * NP + p], sa[p]);
              }
            }
          }
        });
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          if constexpr (WX) gxl[i * NP + p] = vfma(w2[p], sa[p], gxl[i * NP + p]);
          dot[p] = t0 == 0 && !ADD ? vmul(xl[i * NP + p], sa[p]) : vfma(xl[i * NP + p], sa[p], dot[p]);
        }
      }
    }
  });
}

// The same for a path with a degree of zero, whose coupling tensor is c times the identity of the other two degrees:
//     l2 = 0:  d = x . g       gx += (c y w) g      gy += c (w . d)      gw = (c y) d
//     l1 = 0:  s = c (y . g)   gx += w s            gy += (c x w) g      gw = x s
//     l3 = 0:  s = y . x       gx += (c g w) y      gy += (c g w) x      gw = (c g) s
// two to three operations per component instead of the five and a half of edge_path, and nothing of a table.  Seven of the
// eleven paths of degrees (2, 2, 2) are like that, eight of the seventeen of (2, 3, 3).  Forward and backward with all paths in
// edge_path, and like this: (2, 3, 3), 128 channels, 2.6 M edges 15.88 -> 15.33 ms; (3, 3, 3), 64 channels, 1.6 M edges 8.99
// -> 8.54; (2, 2, 2), 64 channels, 5.2 M edges 10.23 -> 9.98; FP64 force step, 1.05 M edges 34.8 -> 33.9.
template <typename T, typename PK, typename S, int l1, int l2, int l3, bool WX, bool WM, bool WY, bool ADD, typename V>
__device__ __forceinline__ void edge_diagonal(const V* xl, V* gxl, V* gyl, const V* g2, const V* w2, V* dot, const T* mbuf, T c) {
  constexpr int NP = PK::NP, d = 2 * (l1 > l3 ? l1 : l3) + 1;
  T y[8];
  if constexpr (WM) edge_attributes<S, l2>(mbuf, y);
  const V cc = bcast_packet(c, V{});
  if constexpr (l2 == 0) {
    V sum[NP];
#pragma unroll
    for (int i = 0; i < d; ++i)
#pragma unroll
      for (int p = 0; p < NP; ++p)
        sum[p] = i == 0 ? vmul(xl[p], g2[p]) : vfma(xl[i * NP + p], g2[i * NP + p], sum[p]);
    if constexpr (WY) {
      V all = vmul(w2[0], sum[0]);
#pragma unroll
      for (int p = 1; p < NP; ++p) all = vfma(w2[p], sum[p], all);
      gyl[0] = vfma(cc, all, gyl[0]);
    }
    if constexpr (WM) {
      const V cy = bcast_packet(c * y[0], V{});
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        dot[p] = ADD ? vfma(cy, sum[p], dot[p]) : vmul(cy, sum[p]);
        if constexpr (WX) {
          const V wy = vmul(cy, w2[p]);
#pragma unroll
          for (int i = 0; i < d; ++i) gxl[i * NP + p] = vfma(wy, g2[i * NP + p], gxl[i * NP + p]);
        }
      }
    }
  } else if constexpr (l1 == 0) {
    if constexpr (WY) {
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const V xw = vmul(vmul(cc, xl[p]), w2[p]);
#pragma unroll
        for (int k = 0; k < d; ++k) gyl[k] = vfma(xw, g2[k * NP + p], gyl[k]);
      }
    }
    if constexpr (WM) {
      V sum[NP];
#pragma unroll
      for (int k = 0; k < d; ++k)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const V yk = bcast_packet(y[k], V{});
          sum[p] = k == 0 ? vmul(yk, g2[p]) : vfma(yk, g2[k * NP + p], sum[p]);
        }
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const V s = vmul(cc, sum[p]);
        dot[p] = ADD ? vfma(xl[p], s, dot[p]) : vmul(xl[p], s);
        if constexpr (WX) gxl[p] = vfma(w2[p], s, gxl[p]);
      }
    }
  } else {
    V cg[NP], cgw[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      cg[p] = vmul(cc, g2[p]);
      cgw[p] = vmul(cg[p], w2[p]);
    }
    if constexpr (WY) {
#pragma unroll
      for (int i = 0; i < d; ++i)
#pragma unroll
        for (int p = 0; p < NP; ++p) gyl[i] = vfma(cgw[p], xl[i * NP + p], gyl[i]);
    }
    if constexpr (WM) {
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        V sum = vmul(bcast_packet(y[0], V{}), xl[p]);
#pragma unroll
        for (int i = 1; i < d; ++i) sum = vfma(bcast_packet(y[i], V{}), xl[i * NP + p], sum);
        dot[p] = ADD ? vfma(cg[p], sum, dot[p]) : vmul(cg[p], sum);
        if constexpr (WX) {
#pragma unroll
          for (int i = 0; i < d; ++i) gxl[i * NP + p] = vfma(bcast_packet(y[i], V{}), cgw[p], gxl[i * NP + p]);
        }
      }
    }
  }
}

// A path of an edge, for a lane's channels: wq its weights in the stage, which the gradients replace if `keep`.
template <typename T, typename PK, typename S, int l1, int l2, int l3, bool WX, bool WM, bool WY, bool ADD, typename V>
__device__ __forceinline__ void backward_path(T* wq, int lanes, bool keep, const V* xr, V* gxr, V* gy2, const V* g2,
                                              const T* mbuf, const T* term, const T* coef) {
  constexpr int NP = PK::NP;
  V w2[NP], dot[NP];
  lane_load<PK, T>(wq, lanes, w2);
  if constexpr (ADD) {
#pragma unroll
    for (int p = 0; p < NP; ++p) dot[p] = w2[p];
  }
  const V* xl = &xr[S::xoff(l1) * NP];
  V *gxl = &gxr[WX ? S::xoff(l1) * NP : 0], *gyl = &gy2[WY ? S::yoff(l2) : 0];
  if constexpr (S::diagonal(l1, l2, l3))
    edge_diagonal<T, PK, S, l1, l2, l3, WX, WM, WY, ADD, V>(xl, gxl, gyl, g2, w2, dot, mbuf, coef[S::coff(l1, l2, l3)]);
  else
    edge_path<T, PK, S, l1, l2, l3, WX, WM, WY, ADD, V>(xl, gxl, gyl, g2, w2, dot, mbuf, term);
  if (WM && keep) lane_store<PK, T>(wq, lanes, dot);  // the gradients leave with the row
}

// FULL: one warp per edge and 32 * CPL channels, known to the compiler.  SLICED: these are a slice of wider blocks.  DST: rows
// by destination (S, x and g exchanged).  ADD: gw alone, added to; w names gw.
template <typename T, int CPL, typename S, bool WX, bool WM, bool WY, bool FULL, bool DST, bool SLICED, bool ADD>
__global__ void __launch_bounds__(EdgeBwd<T, CPL, S, WX, WM, WY>::template warps<FULL> * 32, 1)
    edge_bwd_kernel(const __grid_constant__ EdgeBwdParams<T, EdgeBwd<T, CPL, S, WX, WM, WY>::terms> P) {
  using K = EdgeBwd<T, CPL, S, WX, WM, WY>;
  using PK = EdgePacket<T, CPL, edge_spread(S::OD, S::paths)>;
  using V = typename PK::V;
  constexpr int NP = PK::NP;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  let_next_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team_warps = FULL ? 1 : P.team_warps;
  const int team = FULL ? warp : warp / team_warps, member = warp - team * team_warps;
  const int ch = FULL ? 32 * CPL : P.ch, stages = P.stages;
  const int W = S::paths * ch, X = S::XD * ch, O = S::OD * ch;
  const bool split = P.split != 0;
  const int stage_elems = W + (split ? 0 : O);
  static_assert(FULL || !SLICED, "a slice is one warp's full set of channels");
  static_assert(!ADD || (WM && !WX && !WY), "the weights' place in a stage must be free");
  const int row_ch = SLICED ? P.row_ch : ch, first_ch = SLICED ? static_cast<int>(blockIdx.y) * ch : 0;
  const int w_row = S::paths * row_ch, x_row = S::XD * row_ch, o_row = S::OD * row_ch;  // in memory
  unsigned* const counters = P.tile_counters + (SLICED ? 2 * blockIdx.y : 0);
  T* const gy_out = SLICED ? P.gy + blockIdx.y * P.gy_part : P.gy;

  T* const base = reinterpret_cast<T*>(smem_raw);
  T* const ring = base + static_cast<size_t>(team) * P.team_elems;
  T* const gslots = ring + static_cast<size_t>(stages) * stage_elems;  // split: the row of g, in slots
  T* const warp_mem = base + static_cast<size_t>(P.teams) * P.team_elems;
  const int warp_elems = K::warp_elems(team_warps);
  T* const mbuf = warp_mem + static_cast<size_t>(warp) * warp_elems;
  T* const red = mbuf + K::m_elems;
  T* const gbuf = red + K::red_pass * K::red_row;
  uint64_t* const all_bars = reinterpret_cast<uint64_t*>(warp_mem + static_cast<size_t>(blockDim.x >> 5) * warp_elems);
  uint64_t* const full = all_bars + team * (kEdgeMaxStages + kEdgeMaxSlots);
  uint64_t* const gfull = full + kEdgeMaxStages;
  unsigned* const tickets = reinterpret_cast<unsigned*>(all_bars + P.teams * (kEdgeMaxStages + kEdgeMaxSlots));
  TeamPart* const kept = reinterpret_cast<TeamPart*>(tickets + P.teams);

  if (member == 0 && lane == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&full[s], 1);
    for (int s = 0; s < K::slots; ++s) mbar_init(&gfull[s], 1);
    fence_barrier_init();
  }
  MatrixProgram<T, S> program;
  if constexpr (WM) program.load(P.prog_c, P.prog_j, lane, 0, 1);
  __syncthreads();
  wait_for_previous();

  const int cpw = ch / team_warps;  // channels of this warp
  const int lanes = FULL ? 32 : cpw / CPL;
  const int own = FULL ? lane_first<PK>(lane) : member * cpw + lane_first<PK>(min(lane, lanes - 1));  // first channel of this lane
  const bool active = FULL || lane < lanes;
  const bool leader = member == 0 && lane == 0;
  const bool issuing = SLICED || leader;  // the pieces of a slice are copied by all lanes
  const bool want_x = WX && P.gx != nullptr, storing = WM && P.gw != nullptr;
  const uint32_t w_bytes = P.need_w ? static_cast<uint32_t>(W * sizeof(T)) : 0u;
  const uint32_t g_bytes = split ? 0u : static_cast<uint32_t>(O * sizeof(T));
  const bool staged = w_bytes + g_bytes != 0u;

  // copies the degrees [from, to) of a slice of row d of g, one degree to a lane
  auto load_pieces = [&](auto from, auto until, T* to, int d, uint64_t* bar) {
    static_for<decltype(from)::value, decltype(until)::value>([&](auto lc) {
      constexpr int l = decltype(lc)::value, d3 = 2 * l + 1;
      if constexpr (S::has(S::MO, l)) {
        if (lane == l)
          bulk_copy_g2s(to + ch * S::ooff(l), P.g + static_cast<int64_t>(d) * o_row + row_ch * S::ooff(l) + first_ch * d3,
                        static_cast<uint32_t>(ch * d3 * sizeof(T)), bar);
      }
    });
  };
  auto load_stage = [&](int e, int d, int st) {  // by the issuing lanes
    if (!staged) return;
    T* to = ring + static_cast<size_t>(st) * stage_elems;
    if constexpr (SLICED) {
      if (lane == 0) mbar_arrive_expect_tx(&full[st], w_bytes + g_bytes);
      __syncwarp();  // also: every lane's stores have read the stage
      if (w_bytes)
        for (int p = lane; p < S::paths; p += 32)
          bulk_copy_g2s_hint(to + p * ch, P.w + static_cast<int64_t>(e) * w_row + p * row_ch + first_ch,
                             static_cast<uint32_t>(ch * sizeof(T)), &full[st], l2_policy_evict_first());
      if (g_bytes) load_pieces(std::integral_constant<int, 0>{}, std::integral_constant<int, 4>{}, to + W, d, &full[st]);
      return;
    }
    mbar_arrive_expect_tx(&full[st], w_bytes + g_bytes);
    if (w_bytes)
      bulk_copy_g2s_hint(to, P.w + static_cast<int64_t>(e) * W, w_bytes, &full[st], l2_policy_evict_first());
    if (g_bytes) bulk_copy_g2s(to + W, P.g + static_cast<int64_t>(d) * O, g_bytes, &full[st]);
  };
  auto load_slot = [&](auto slot, int d) {  // by the issuing lanes
    constexpr int h = decltype(slot)::value, first = K::slot_begin(h), count = K::slot_begin(h + 1) - first;
    const uint32_t bytes = static_cast<uint32_t>(count * ch * sizeof(T));
    if constexpr (SLICED) {
      if (lane == 0) mbar_arrive_expect_tx(&gfull[h], bytes);
      __syncwarp();
      load_pieces(std::integral_constant<int, h == 0 ? 0 : S::LO>{}, std::integral_constant<int, h + 1 == K::slots ? 4 : S::LO>{},
                  gslots, d, &gfull[h]);
      return;
    }
    mbar_arrive_expect_tx(&gfull[h], bytes);
    bulk_copy_g2s(gslots + first * ch, P.g + static_cast<int64_t>(d) * O + first * ch, bytes, &gfull[h]);
  };

  V xr[S::XD * NP], gxr[WX ? S::XD * NP : 1], gy2[WY ? S::YD : 1];
  int st = 0;                       // stage of the current edge; the ring keeps turning from one row to the next
  uint32_t parity = 0, gparity = 0;  // phases of that stage's barrier and of the slots' barriers
  bool alive = true;
  int flip = 0;                     // which of the two reduced gy rows the current edge uses
  auto wait = [&](uint64_t* bar, uint32_t phase, int code) {
    if (!edge_wait(bar, phase, alive)) {
      if (lane == 0) atomicExch(P.status, code);
      alive = false;
    }
  };

  auto unit_body = [&](auto l3c, const T* gblock, T* wrow) {
    constexpr int l3 = decltype(l3c)::value;
    constexpr int d3 = 2 * l3 + 1;
    V g2[d3 * NP];
    lane_load_block<PK, T, d3>(gblock + own * d3, lanes, g2);
    static_for<0, 4>([&](auto l1c) {
      constexpr int l1 = decltype(l1c)::value;
      static_for<0, 4>([&](auto l2c) {
        constexpr int l2 = decltype(l2c)::value;
        if constexpr (S::ok(l1, l2, l3)) {
          backward_path<T, PK, S, l1, l2, l3, WX, WM, WY, ADD, V>(wrow + S::rank(l1, l2, l3) * ch + own, lanes, storing && active,
                                                                xr, gxr, gy2, g2, mbuf, P.term, P.coef);
        }
      });
    });
  };

  const bool parts = P.parts != 0, every_row = P.every_row != 0;
  int open_row = -1;  // whose sum goes to shared memory, to be added to what the next team has of it
  // edges and rows fit 31 bits, and every register counts
  const unsigned total = gridDim.x * static_cast<unsigned>(P.teams);
  unsigned unit = blockIdx.x * P.teams + team;
  const unsigned units = parts ? total : static_cast<unsigned>(P.num_tiles);
  int seen_row = 0, seen_pos = 0;  // a row boundary this warp has seen, and where its edges begin
#pragma unroll 1
  while (unit < units) {
    unsigned unit_after = unit + total;
    int n, n_hi, pos, p_end;
    if (parts) {
      const TeamPart part = team_part(P.src_rowptr, P.num_rows, P.num_edges, P.rows_per_edge, team, P.teams, lane);
      n = part.n;
      n_hi = part.n_hi;
      pos = part.pos;
      p_end = part.end;
      open_row = part.open_row();
      if (leader) kept[team] = part;  // for the end of the launch
    } else {
      if (team_warps == 1) {
        unit_after = static_cast<unsigned>(take_tile(counters, total, lane));
      } else {
        if (leader) tickets[team] = atomicAdd(&counters[0], 1u);
        team_sync(team_warps, team);
        unit_after = total + tickets[team];
        team_sync(team_warps, team);
      }
      if (P.tile_rows > 0) {
        const int64_t first = unit * P.tile_rows, end = first + P.tile_rows;
        n = static_cast<int>(first);
        n_hi = static_cast<int>(end < P.num_rows ? end : P.num_rows);
      } else {
        // tile t: the rows whose edges begin in [t, t + 1) * tile_edges of the source-sorted edge order (guessed from
        // where the warp's previous tile ended, assuming rows of average length in between)
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
    // ids of the current and the next four edges, destinations of the first four of them
    auto edge_at = [&](int p) { return DST ? p : P.edge_ids[p]; };
    auto id_at = [&](int p) { return p < p_end ? edge_at(p) : -1; };
    auto dst_of = [&](int e) { return e >= 0 ? P.dst[e] : 0; };
    int e0 = id_at(pos), e1 = id_at(pos + 1), e2 = id_at(pos + 2), e3 = id_at(pos + 3), e4 = id_at(pos + 4);
    int d0 = dst_of(e0), d1 = dst_of(e1), d2 = dst_of(e2), d3n = dst_of(e3);
    auto id_ahead = [&](int k) { return k == 1 ? e1 : (k == 2 ? e2 : e3); };
    auto dst_ahead = [&](int k) { return k == 1 ? d1 : (k == 2 ? d2 : d3n); };
    if (issuing && e0 >= 0) {
      load_stage(e0, d0, st);
      for (int k = 1, stage = st; k < stages; ++k) {
        if (++stage == stages) stage = 0;
        if (id_ahead(k) >= 0) load_stage(id_ahead(k), dst_ahead(k), stage);
      }
      if (split) static_for<0, K::slots>([&](auto h) { load_slot(h, d0); });
    }
    T y_next = lane < S::YD && e0 >= 0 ? P.y[static_cast<int64_t>(e0) * S::YD + lane] : T(0);
    if constexpr (WM) program.run(y_next, mbuf, lane, 0, 1);
    if (WM && e1 >= 0 && lane < S::YD) y_next = P.y[static_cast<int64_t>(e1) * S::YD + lane];
    __syncwarp();
    int refill_stage = -1;  // a stage whose row is on its way back, to be refilled with the edge `stages` after it
#pragma unroll 1
    for (; n < n_hi; ++n) {
      const int pe = min(P.src_rowptr[n + 1], p_end);
      if (!every_row && pos >= pe) {
        // A row without edges in a piece of a graph, which has long runs of them (their gx is cleared beforehand): jump
        // to the row that holds the next edge instead of walking the run one dependent load at a time.
        if (pos >= p_end) break;
        n = static_cast<int>(warp_lower_bound(P.src_rowptr, P.num_rows, pos + 1, lane)) - 2;
        continue;
      }
      if (pos < pe) {
        static_for<0, 4>([&](auto l1c) {
          constexpr int l1 = decltype(l1c)::value;
          if constexpr (S::has(S::MX, l1)) {
            constexpr int d = 2 * l1 + 1;
            lane_load_block<PK, T, d>(P.x + static_cast<int64_t>(n) * x_row + row_ch * S::xoff(l1) + (first_ch + own) * d, lanes, &xr[S::xoff(l1) * NP]);
          }
        });
        if (!active) {
#pragma unroll
          for (int a = 0; a < S::XD * NP; ++a) xr[a] = zero_packet<V>();
        }
      }
      if constexpr (WX) {
#pragma unroll
        for (int a = 0; a < S::XD * NP; ++a) gxr[a] = zero_packet<V>();
      }
#pragma unroll 1
      for (; pos < pe; ++pos) {
        if constexpr (WY) {
#pragma unroll
          for (int j = 0; j < S::YD; ++j) gy2[j] = zero_packet<V>();
        }
        if (staged) wait(&full[st], parity, 3);
        T* wrow = ring + static_cast<size_t>(st) * stage_elems;
        const bool more = pos + 1 < p_end;
        static_for<0, 4>([&](auto l3c) {
          constexpr int l3 = decltype(l3c)::value;
          if constexpr (S::has(S::MO, l3)) {
            constexpr int slot = K::slot_of(l3);
            if constexpr (S::ooff(l3) == K::slot_begin(slot)) {
              if (split) wait(&gfull[slot], gparity, 2);
            }
            unit_body(l3c, (split ? gslots : wrow + W) + ch * S::ooff(l3), wrow);
            if constexpr (l3 != S::LO && S::ooff(l3) + 2 * l3 + 1 == K::slot_begin(slot + 1)) {
              if (split) {  // the slot is done with; the last one is refilled at the end of the edge
                fence_async_shared();
                team_sync(team_warps, team);
                if (issuing && more) load_slot(std::integral_constant<int, slot>{}, d1);
              }
            }
            if constexpr (S::ooff(l3) == 0) {  // after the first degree: the row sent back has left its stage by now
              if (refill_stage >= 0 && issuing) {
                bulk_wait_group_read_all();
                if (id_ahead(stages - 1) >= 0) load_stage(id_ahead(stages - 1), dst_ahead(stages - 1), refill_stage);
              }
              refill_stage = -1;
            }
          }
        });
        fence_async_shared();         // gradient writes, before the bulk store reads the stage, and reads, before it is refilled
        team_sync(team_warps, team);  // every lane is done with the stage, the last slot and the scalars
        if (issuing) {
          if (split && more) load_slot(std::integral_constant<int, K::slots - 1>{}, d1);
          if (storing) {
            T* row = P.gw + static_cast<int64_t>(e0) * w_row + first_ch;
            auto send = [&](int at, int from, uint32_t bytes) {
              if (P.acc_w)
                bulk_reduce_add_s2g(row + at, wrow + from, bytes);
              else
                bulk_copy_s2g_hint(row + at, wrow + from, bytes, l2_policy_evict_first());
            };
            if constexpr (SLICED) {
              for (int p = lane; p < S::paths; p += 32) send(p * row_ch, p * ch, static_cast<uint32_t>(ch * sizeof(T)));
            } else {
              send(0, 0, static_cast<uint32_t>(W * sizeof(T)));
            }
            bulk_commit_group();
          } else if (pos + stages < p_end) {
            const int k = stages;
            load_stage(k == 2 ? e2 : (k == 3 ? e3 : e4), k == 2 ? d2 : d3n, st);
          }
        }
        if (storing) refill_stage = st;
        if constexpr (WM) program.run(y_next, mbuf, lane, 0, 1);
        if (WM && pos + 2 < p_end && lane < S::YD) y_next = P.y[static_cast<int64_t>(e2) * S::YD + lane];
        if constexpr (WY) {
          // the lanes' partial gy rows through the reduction tile: entries 2r and 2r + 1 in tile row r; four lanes sum
          // a row, a quarter each.  Idle lanes bring in zeros: what they computed is 0 times the last lane's w and g.
          constexpr int passes = (K::red_rows + K::red_pass - 1) / K::red_pass;
          static_for<0, passes>([&](auto qc) {
            constexpr int first = decltype(qc)::value * K::red_pass;
            constexpr int rows = K::red_rows - first < K::red_pass ? K::red_rows - first : K::red_pass;
            static_for<0, rows>([&](auto rc) {
              constexpr int j = 2 * (first + decltype(rc)::value);
              Vec<T, 2> pr;
              pr.a[0] = active ? hsum(gy2[j]) : T(0);
              if constexpr (j + 1 < S::YD) {
                pr.a[1] = active ? hsum(gy2[j + 1]) : T(0);
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
            s0 += __shfl_xor_sync(0xffffffffu, s0, 16);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 16);
            if (lane < rows) {
              const int j = 2 * (first + lane);
              if (team_warps > 1) {
                *reinterpret_cast<Vec<T, 2>*>(gbuf + flip * 32 + j) = Vec<T, 2>{{s0, s1}};
              } else {
                T* to = gy_out + static_cast<int64_t>(e0) * S::YD + j;
                to[0] = P.acc_y ? to[0] + s0 : s0;
                if (j + 1 < S::YD) to[1] = P.acc_y ? to[1] + s1 : s1;
              }
            }
            __syncwarp();
          });
          if (team_warps > 1) {
            team_sync(team_warps, team);
            if (member == 0 && lane < S::YD) {
              T sum = gbuf[flip * 32 + lane];
              for (int m = 1; m < team_warps; ++m) sum += gbuf[m * warp_elems + flip * 32 + lane];
              T* to = gy_out + static_cast<int64_t>(e0) * S::YD + lane;
              *to = P.acc_y ? *to + sum : sum;
            }
            flip ^= 1;
          }
        } else {
          __syncwarp();
        }
        e0 = e1;
        e1 = e2;
        e2 = e3;
        e3 = e4;
        d0 = d1;
        d1 = d2;
        d2 = d3n;
        if (pos + 4 < p_end) d3n = P.dst[e3];
        e4 = pos + 5 < p_end ? edge_at(pos + 5) : -1;
        gparity ^= 1u;
        if (++st == stages) {
          st = 0;
          parity ^= 1u;
        }
      }
      if constexpr (WX) {
        const bool rest = n == open_row;
        if (rest) {  // goes to shared memory: bulk stores must have read the ring
          if (issuing) bulk_wait_group_read_all();
          team_sync(team_warps, team);
        }
        if (want_x && active) {
          T* to = rest ? ring : P.gx + static_cast<int64_t>(n) * x_row;
          const int block = rest ? ch : row_ch, at = rest ? own : first_ch + own;
          static_for<0, 4>([&](auto l1c) {
            constexpr int l1 = decltype(l1c)::value, d = 2 * l1 + 1;
            if constexpr (S::has(S::MX, l1))
              lane_store_block<PK, T, d>(to + block * S::xoff(l1) + at * d, lanes, &gxr[S::xoff(l1) * NP],
                                         !rest && P.acc_x);
          });
        }
      }
    }
    if (WM && issuing) bulk_wait_group_read_all();  // the next rows' copies reuse the stages
  }
  if (!parts) {
    if (member == 0) leave_tiles(counters, total, lane);
  } else if constexpr (WX) {
    if (want_x)
      merge_parts(kept, P.teams, P.src_rowptr, base, P.team_elems, X, [&](int row, int a) {
        return P.gx + static_cast<int64_t>(row) * x_row + (SLICED ? slice_element<S>(S::MX, a, ch, row_ch, first_ch) : a);
      });
  }
  if (WM && issuing) bulk_wait_group_read_all();
  if (!alive) {  // let copies that are still in flight land before the CTA's shared memory is released
    for (int d = 0; d < stages; ++d) edge_wait(&full[d], d < st ? parity : parity ^ 1u, false);
    for (int d = 0; d < K::slots; ++d) edge_wait(&gfull[d], gparity ^ 1u, false);
  }
}

}  // namespace edgek
}  // namespace luna
