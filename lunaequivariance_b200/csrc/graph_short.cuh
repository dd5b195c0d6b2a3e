// Graph tables of graphs whose rows are short, at most kShortRow edges on either side: the same tables as the general kernels
// of graph.cu, by counting instead of sorting.
//
// What bounds the tables is the number of dependent launches, not bytes.  The general way is two radix sorts of many launches
// each.  Here it is five launches and one memset:
//   short_edges    copies and checks the edges; counts the edges of every source, a count's old value being the edge's place
//                  in its row, in no particular order; notes where the edges of a destination begin and end
//   short_counts   histograms, by blocks of nodes, of the three orders' keys, which are below 256 where rows are short, and
//                  sums of degrees and pieces; the last block to finish turns them into where each block begins
//   short_nodes    row pointers, orders and tiers: a node's place is its block's, plus its rank among the block's nodes of the
//                  same key, which a match within the warp and a scan over the warps give
//   short_scatter  edge ids to their sources' rows
//   short_rows     a warp sorts a row's edge ids in registers (ascending, so the order in which they came does not matter) and
//                  writes the row's pieces
// A longer row sets a flag, at which the launches that follow do nothing, and the caller goes on with the sorts from the edges that
// short_edges has copied and checked.
//
// 1.05 M edges, 20,000 nodes, the five launches: 10, 10, 6, 9 and 9 us; the whole call, with the allocations before it and the
// synchronisation at its end, 201 -> 105 us, 93 with launches that overlap (launch_early), and 88 since the last block of
// short_counts sums two columns to a thread and scans two orders at a time (14 us before).  short_edges is not bound by its atomics
// (a copy of the same bytes takes 4.5 us); short_counts is a chain of dependent steps, of which one block does the last.  Blocks of
// 1,024 nodes halve that block's sums but make short_nodes slower (6 -> 8 us).
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.h"

namespace luna {
namespace {

constexpr int kShortRow = 255;
constexpr int kShortKeys = 256;
constexpr int kShortSets = 3;  // orders: destinations, sources, source rows by their last piece
constexpr int kShortBlock = 512;
constexpr int kShortWarps = kShortBlock / 32;
// ShortTables::head.  The flags are words of their own because one launch may set both.
constexpr int kHeadUnfit = 0, kHeadPieces = 1, kHeadFinished = 2, kHeadLongRow = 3, kHeadWords = 4;

struct ShortTables {
  int64_t nodes, src_nodes, edges, blocks;
  int* head;  // an index unfit, number of pieces, blocks that have finished, a long row; zero, like the next three, at the start
  int32_t *first, *last;  // [nodes] edges of a destination
  int32_t* count;         // [src_nodes] edges of a source
  uint16_t* place;        // [edges] within the source's row
  int32_t* histogram;     // [blocks][kShortSets * kShortKeys], then of the blocks before
  int32_t* sums;          // [blocks][3] edges by destination, edges by source, pieces; then of the blocks before
  int32_t* key_begin;     // [kShortSets * kShortKeys] nodes of the set with a smaller key
  int32_t* full_begin;    // [kShortKeys] full pieces of sources with a smaller key, and behind them the number of all
  int32_t *full_at, *part_at;  // [src_nodes] places of a row's pieces in the order of pieces
  int32_t *src, *dst, *iota, *dst_rowptr, *src_rowptr, *edge_ids, *node_order, *source_node_order, *tiers;
  int32_t *segment_nodes, *segment_begin, *segment_end, *segment_rowptr, *segment_order;
};

// Whether the edges are for others: unfit, or for the general kernels.
__device__ __forceinline__ bool short_given_up(const ShortTables& t) { return (t.head[kHeadUnfit] | t.head[kHeadLongRow]) != 0; }

struct ShortNode {
  int in, out, pieces;
  int key[kShortSets];  // kShortKeys: the node is not in the set
};
__device__ __forceinline__ ShortNode short_node(const ShortTables& t, int64_t n) {
  ShortNode node{0, 0, 0, {kShortKeys, kShortKeys, kShortKeys}};
  if (n < t.nodes) {
    node.in = t.last[n] - t.first[n];
    node.key[0] = kShortRow - min(node.in, kShortRow);
  }
  if (n < t.src_nodes) {
    node.out = t.count[n];
    node.pieces = max(1, (node.out + 31) >> 5);
    const int out = min(node.out, kShortRow);
    node.key[1] = kShortRow - out;
    node.key[2] = (31 - (out & 31)) * 8 + 7 - (out >> 5);
  }
  return node;
}

constexpr int kShortEdges = 4;  // per thread
template <typename Index>
__global__ void __launch_bounds__(256) short_edges(const Index* __restrict__ src, const Index* __restrict__ dst, ShortTables t) {
  let_next_start();
  wait_for_previous();
  const int64_t begin = static_cast<int64_t>(blockIdx.x) * (256 * kShortEdges) + threadIdx.x;
  Index s[kShortEdges], d[kShortEdges], before[kShortEdges], after[kShortEdges];
#pragma unroll
  for (int k = 0; k < kShortEdges; ++k) {
    const int64_t e = begin + 256 * k;
    s[k] = e < t.edges ? src[e] : 0;
    d[k] = e < t.edges ? dst[e] : 0;
    before[k] = e > 0 && e < t.edges ? dst[e - 1] : -1;
    after[k] = e + 1 < t.edges ? dst[e + 1] : -1;
  }
  bool fit[kShortEdges];
#pragma unroll
  for (int k = 0; k < kShortEdges; ++k) {
    const int64_t e = begin + 256 * k;
    const bool bad = s[k] < 0 || s[k] >= t.src_nodes || d[k] < 0 || d[k] >= t.nodes || (e > 0 && before[k] > d[k]);
    if (e < t.edges && bad) t.head[kHeadUnfit] = 1;
    fit[k] = e < t.edges && !bad;
  }
  // In a large graph a thread's first edge is counted, the copies are made meanwhile, and the others are counted if no row has turned
  // out to be long: the atomics of a row with a good part of all edges wait for one another, 1.4 ns each.  1.05 M edges, 87,000 of them
  // in one row, the whole call with the sorts that follow 354 -> 247 us; 64,000 edges are too few to be worth the second trip.
  const bool wary = gridDim.x > 64;
  int place[kShortEdges];
#pragma unroll
  for (int k = 0; k < kShortEdges; ++k) place[k] = fit[k] && (k == 0 || !wary) ? atomicAdd(t.count + s[k], 1) : -1;
#pragma unroll
  for (int k = 0; k < kShortEdges; ++k) {
    const int64_t e = begin + 256 * k;
    if (!fit[k]) continue;
    t.src[e] = static_cast<int32_t>(s[k]);
    t.dst[e] = static_cast<int32_t>(d[k]);
    t.iota[e] = static_cast<int32_t>(e);
    if (before[k] != d[k]) t.first[d[k]] = static_cast<int32_t>(e);
    if (after[k] != d[k]) t.last[d[k]] = static_cast<int32_t>(e + 1);
  }
  if (wary) {
    if (place[0] == kShortRow) t.head[kHeadLongRow] = 1;
    if (__syncthreads_or(place[0] >= kShortRow || (threadIdx.x == 0 && __ldcg(t.head + kHeadLongRow) != 0))) return;
#pragma unroll
    for (int k = 1; k < kShortEdges; ++k)
      if (fit[k]) place[k] = atomicAdd(t.count + s[k], 1);
  }
#pragma unroll
  for (int k = 0; k < kShortEdges; ++k) {
    if (place[k] >= 0) t.place[begin + 256 * k] = static_cast<uint16_t>(place[k]);
    if (place[k] == kShortRow) t.head[kHeadLongRow] = 1;  // short_counts would find it too, later
  }
}

// Sums over the block's threads before this one, of three numbers; all: over all threads.
struct ShortSum {
  int v[3];
};
__device__ __forceinline__ ShortSum short_scan(ShortSum mine, ShortSum* all, int (*shared)[3]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ShortSum sum = mine;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int step = 1; step < 32; step *= 2) {
      const int other = __shfl_up_sync(0xffffffffu, sum.v[c], step);
      if (lane >= step) sum.v[c] += other;
    }
  if (lane == 31)
    for (int c = 0; c < 3; ++c) shared[warp][c] = sum.v[c];
  __syncthreads();
  ShortSum before{{0, 0, 0}};
  *all = before;
#pragma unroll
  for (int w = 0; w < kShortWarps; ++w)
    for (int c = 0; c < 3; ++c) {
      const int part = shared[w][c];
      if (w < warp) before.v[c] += part;
      all->v[c] += part;
    }
#pragma unroll
  for (int c = 0; c < 3; ++c) before.v[c] += sum.v[c] - mine.v[c];
  __syncthreads();
  return before;
}

__global__ void __launch_bounds__(kShortBlock) short_counts(ShortTables t) {
  let_next_start();
  wait_for_previous();
  __shared__ int histogram[kShortSets * kShortKeys];
  __shared__ int scan[kShortWarps][3];
  __shared__ int finished;
  if (__syncthreads_or(short_given_up(t))) return;
  for (int i = threadIdx.x; i < kShortSets * kShortKeys; i += kShortBlock) histogram[i] = 0;
  __syncthreads();
  const ShortNode node = short_node(t, static_cast<int64_t>(blockIdx.x) * kShortBlock + threadIdx.x);
  const bool lost = __syncthreads_or(node.in > kShortRow || node.out > kShortRow) != 0;
  if (lost) {
    if (threadIdx.x == 0) t.head[kHeadLongRow] = 1;
    return;  // the other blocks' last one never comes
  }
#pragma unroll
  for (int s = 0; s < kShortSets; ++s)
    if (node.key[s] < kShortKeys) atomicAdd(&histogram[s * kShortKeys + node.key[s]], 1);
  ShortSum all;
  short_scan(ShortSum{{node.in, node.out, node.pieces}}, &all, scan);  // and a barrier
  int32_t* const mine = t.histogram + static_cast<int64_t>(blockIdx.x) * (kShortSets * kShortKeys);
  for (int i = threadIdx.x; i < kShortSets * kShortKeys; i += kShortBlock) mine[i] = histogram[i];
  if (threadIdx.x < 3) t.sums[blockIdx.x * 3 + threadIdx.x] = all.v[threadIdx.x];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) finished = atomicAdd(&t.head[kHeadFinished], 1);
  __syncthreads();
  if (finished != static_cast<int>(t.blocks) - 1) return;
  __threadfence();

  // the last block: what the blocks before each block have, two columns to a thread and 24 blocks of both at a time
  constexpr int kColumns = kShortSets * kShortKeys + 3, kAtOnce = 24;
  static_assert(kColumns <= 2 * kShortBlock, "a thread has two columns");
  int32_t* column[2];
  int stride[2], total[2] = {0, 0};
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int i = static_cast<int>(threadIdx.x) + c * kShortBlock;
    const bool keys = i < kShortSets * kShortKeys;
    column[c] = i >= kColumns ? nullptr : (keys ? t.histogram + i : t.sums + (i - kShortSets * kShortKeys));
    stride[c] = keys ? kShortSets * kShortKeys : 3;
  }
  for (int64_t b = 0; b < t.blocks; b += kAtOnce) {
    int part[2][kAtOnce];
#pragma unroll
    for (int k = 0; k < kAtOnce; ++k)
#pragma unroll
      for (int c = 0; c < 2; ++c) part[c][k] = column[c] && b + k < t.blocks ? __ldcg(column[c] + (b + k) * stride[c]) : 0;
#pragma unroll
    for (int k = 0; k < kAtOnce; ++k)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (column[c] && b + k < t.blocks) column[c][(b + k) * stride[c]] = total[c];
        total[c] += part[c][k];
      }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int i = static_cast<int>(threadIdx.x) + c * kShortBlock;
    if (i < kShortSets * kShortKeys) histogram[i] = total[c];
    if (i == kColumns - 1) t.head[kHeadPieces] = total[c];
  }
  __syncthreads();
  // keys: nodes before, and for the orders by degree the edges and the full pieces before.  The first half of the threads has the
  // first set, with the third set's nodes, and the second half the second set, from which the first one's totals are taken off.
  static_assert(kShortBlock == 2 * kShortKeys, "a half of the threads has a key each");
  const int set = static_cast<int>(threadIdx.x) / kShortKeys, key = static_cast<int>(threadIdx.x) % kShortKeys;
  const int nodes = histogram[set * kShortKeys + key], degree = kShortRow - key;
  const int weight = nodes * (set == 0 ? degree : degree >> 5);
  ShortSum before = short_scan(ShortSum{{nodes, weight, set == 0 ? histogram[2 * kShortKeys + key] : 0}}, &all, scan);
  if (set == 0) {
    t.key_begin[key] = before.v[0];
    t.key_begin[2 * kShortKeys + key] = before.v[2];
    for (int k = 1; k < 4; ++k) {  // tier k ends with the row that brings the edges to k quarters
      const int quarter = static_cast<int>(static_cast<int64_t>(k) * t.edges / 4);
      if (quarter > before.v[1] && quarter <= before.v[1] + weight)
        t.tiers[k - 1] = before.v[0] + (quarter - before.v[1] + degree - 1) / degree;
      if (quarter == 0 && key == 0) t.tiers[k - 1] = 1;
    }
  } else {
    before.v[0] -= static_cast<int>(t.nodes);
    before.v[1] -= static_cast<int>(t.edges);  // of at most a hundred million (short_rows_likely)
    t.key_begin[kShortKeys + key] = before.v[0];
    t.full_begin[key] = before.v[1];
    if (key == kShortKeys - 1) t.full_begin[kShortKeys] = before.v[1] + weight;
  }
}

__global__ void __launch_bounds__(kShortBlock) short_nodes(ShortTables t) {
  let_next_start();
  wait_for_previous();
  __shared__ uint16_t before[kShortWarps][kShortKeys];  // nodes of a key in a warp, then in the warps before
  __shared__ int scan[kShortWarps][3];
  if (short_given_up(t)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n = static_cast<int64_t>(blockIdx.x) * kShortBlock + threadIdx.x;
  const ShortNode node = short_node(t, n);
  ShortSum all;
  ShortSum begin = short_scan(ShortSum{{node.in, node.out, node.pieces}}, &all, scan);
#pragma unroll
  for (int c = 0; c < 3; ++c) begin.v[c] += t.sums[blockIdx.x * 3 + c];
  if (n < t.nodes) t.dst_rowptr[n] = begin.v[0];
  if (n == t.nodes - 1) t.dst_rowptr[n + 1] = begin.v[0] + node.in;
  if (n < t.src_nodes) {
    t.src_rowptr[n] = begin.v[1];
    t.segment_rowptr[n] = begin.v[2];
  }
  if (n == t.src_nodes - 1) {
    t.src_rowptr[n + 1] = begin.v[1] + node.out;
    t.segment_rowptr[n + 1] = begin.v[2] + node.pieces;
  }
  for (int s = 0; s < kShortSets; ++s) {
    for (int i = threadIdx.x; i < kShortWarps * kShortKeys; i += kShortBlock) (&before[0][0])[i] = 0;
    __syncthreads();
    const int key = node.key[s];
    const unsigned same = __match_any_sync(0xffffffffu, key);
    const int in_warp = __popc(same & ((1u << lane) - 1u));
    if (key < kShortKeys && in_warp == 0) before[warp][key] = static_cast<uint16_t>(__popc(same));
    __syncthreads();
    if (threadIdx.x < kShortKeys) {
      int sum = 0;
#pragma unroll
      for (int w = 0; w < kShortWarps; ++w) {
        const int part = before[w][threadIdx.x];
        before[w][threadIdx.x] = static_cast<uint16_t>(sum);
        sum += part;
      }
    }
    __syncthreads();
    if (key < kShortKeys) {
      const int column = s * kShortKeys + key;
      const int in_key = t.histogram[static_cast<int64_t>(blockIdx.x) * (kShortSets * kShortKeys) + column] + before[warp][key] + in_warp;
      const int at = t.key_begin[column] + in_key;
      if (s == 0) t.node_order[at] = static_cast<int32_t>(n);
      if (s == 1) {
        t.source_node_order[at] = static_cast<int32_t>(n);
        t.full_at[n] = t.full_begin[key] + in_key * (node.out >> 5);
      }
      // the pieces that are shorter than 32 edges follow the full ones, those of rows without edges end the list
      if (s == 2) t.part_at[n] = node.out == 0 ? t.head[kHeadPieces] - static_cast<int>(t.src_nodes - at) : t.full_begin[kShortKeys] + at;
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) short_scatter(ShortTables t) {
  let_next_start();
  wait_for_previous();
  if (short_given_up(t)) return;
  const int64_t begin = static_cast<int64_t>(blockIdx.x) * (256 * kShortEdges) + threadIdx.x;
  int at[kShortEdges];
#pragma unroll
  for (int k = 0; k < kShortEdges; ++k) {
    const int64_t e = begin + 256 * k;
    at[k] = e < t.edges ? t.src_rowptr[t.src[e]] + t.place[e] : -1;
  }
#pragma unroll
  for (int k = 0; k < kShortEdges; ++k)
    if (at[k] >= 0) t.edge_ids[at[k]] = static_cast<int32_t>(begin + 256 * k);
}

// Sorts a row of up to 32 * N ids, element a * 32 + lane in v[a] (bitonic).
template <int N>
__device__ __forceinline__ void short_sort(int32_t* row, int edges, int lane) {
  int v[N];
#pragma unroll
  for (int a = 0; a < N; ++a) v[a] = a * 32 + lane < edges ? row[a * 32 + lane] : 0x7fffffff;
#pragma unroll
  for (int size = 2; size <= 32 * N; size *= 2) {
#pragma unroll
    for (int step = size / 2; step > 0; step /= 2) {
      if (step >= 32) {
#pragma unroll
        for (int a = 0; a < N; ++a) {
          const int b = a ^ (step / 32);
          if (b <= a) continue;
          const bool up = ((a * 32) & size) == 0;
          const int lo = min(v[a], v[b]), hi = max(v[a], v[b]);
          v[a] = up ? lo : hi;
          v[b] = up ? hi : lo;
        }
      } else {
#pragma unroll
        for (int a = 0; a < N; ++a) {
          const int other = __shfl_xor_sync(0xffffffffu, v[a], step);
          const bool up = ((a * 32 + lane) & size) == 0, lower = (lane & step) == 0;
          v[a] = up == lower ? min(v[a], other) : max(v[a], other);
        }
      }
    }
  }
#pragma unroll
  for (int a = 0; a < N; ++a)
    if (a * 32 + lane < edges) row[a * 32 + lane] = v[a];
}

__global__ void __launch_bounds__(256) short_rows(ShortTables t) {
  let_next_start();
  wait_for_previous();
  if (short_given_up(t)) return;
  const int lane = threadIdx.x & 31;
  const int64_t n = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) >> 5;
  if (n >= t.src_nodes) return;
  const int row = t.src_rowptr[n], row_end = t.src_rowptr[n + 1], edges = row_end - row;
  const int piece = t.segment_rowptr[n] + lane, from = row + 32 * lane;
  if (lane < max(1, (edges + 31) >> 5)) {
    t.segment_nodes[piece] = static_cast<int32_t>(n);
    t.segment_begin[piece] = from;
    t.segment_end[piece] = min(from + 32, row_end);
    t.segment_order[lane < edges >> 5 ? t.full_at[n] + lane : t.part_at[n]] = piece;
  }
  if (edges <= 1) return;
  if (edges <= 32)
    short_sort<1>(t.edge_ids + row, edges, lane);
  else if (edges <= 64)
    short_sort<2>(t.edge_ids + row, edges, lane);
  else if (edges <= 128)
    short_sort<4>(t.edge_ids + row, edges, lane);
  else
    short_sort<8>(t.edge_ids + row, edges, lane);
}

// A row of more than 255 edges costs the launches above, of which all but the first do nothing, and a synchronisation before the sorts
// begin: one row of 300 edges, 20,000 nodes of 52 on average 199 -> 222 us, 200,000 of 8 258 -> 305; without that row 103 and 179.
// Such rows are rare where the average is a third of that, so up to there it is tried.  The limit of the nodes is that of the one
// block that sums all blocks' histograms: 2,048 of them take it some 0.2 ms, as much as the general way has launches for.
constexpr int64_t kShortMostBlocks = 2048;
inline bool short_rows_likely(int64_t nodes, int64_t src_nodes, int64_t edges) {
  return edges <= 96 * std::min(nodes, src_nodes) && std::max(nodes, src_nodes) <= kShortMostBlocks * kShortBlock;
}

// Tables in the scratch; returns the bytes.  Zero at the start: from `head` to `zeroed`.
inline size_t short_layout(ShortTables* t, unsigned char* scratch, size_t* zeroed) {
  size_t cursor = 0;
  auto take = [&](auto** table, int64_t entries) {
    using Entry = std::remove_reference_t<decltype(**table)>;
    *table = reinterpret_cast<Entry*>(scratch + cursor);
    cursor += (static_cast<size_t>(entries) * sizeof(Entry) + 15) / 16 * 16;
  };
  t->blocks = ceil_div(std::max(t->nodes, t->src_nodes), kShortBlock);
  take(&t->head, kHeadWords);
  take(&t->first, t->nodes);
  take(&t->last, t->nodes);
  take(&t->count, t->src_nodes);
  *zeroed = cursor;
  take(&t->place, t->edges);
  take(&t->histogram, t->blocks * kShortSets * kShortKeys);
  take(&t->sums, t->blocks * 3);
  take(&t->key_begin, kShortSets * kShortKeys);
  take(&t->full_begin, kShortKeys + 1);
  take(&t->full_at, t->src_nodes);
  take(&t->part_at, t->src_nodes);
  return cursor;
}

// Everything but the synchronisation; t.head tells how it went.
template <typename Index>
int short_tables(const void* src, const void* dst, const ShortTables& t, size_t zeroed, cudaStream_t stream) {
  const unsigned edge_blocks = static_cast<unsigned>(ceil_div(t.edges, 256 * kShortEdges)), node_blocks = static_cast<unsigned>(t.blocks);
  LUNA_CUDA_CHECK(cudaMemsetAsync(t.head, 0, zeroed, stream));
  launch_early(short_edges<Index>, edge_blocks, 256, 0, stream, static_cast<const Index*>(src), static_cast<const Index*>(dst), t);
  LUNA_LAUNCH_CHECK("graph edge copies");
  launch_early(short_counts, node_blocks, kShortBlock, 0, stream, t);
  LUNA_LAUNCH_CHECK("graph node counts");
  launch_early(short_nodes, node_blocks, kShortBlock, 0, stream, t);
  LUNA_LAUNCH_CHECK("graph node tables");
  launch_early(short_scatter, edge_blocks, 256, 0, stream, t);
  LUNA_LAUNCH_CHECK("graph edge ids");
  launch_early(short_rows, static_cast<unsigned>(ceil_div(t.src_nodes, 8)), 256, 0, stream, t);
  LUNA_LAUNCH_CHECK("graph rows");
  return LUNA_OK;
}

}  // namespace
}  // namespace luna
