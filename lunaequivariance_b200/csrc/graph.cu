// Graph tables on the device: index bounds / sortedness scan, CSR row pointers by destination and by source, the
// stable permutation of edge ids grouped by source, degree-descending node orders, edge quarters and the source rows'
// pieces of 32 edges.  Everything runs on the caller's stream with caller-provided scratch; no atomics on the tables,
// which are the same whatever the launch.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include "graph_short.cuh"

namespace luna {
namespace {

constexpr int kThreads = 256;

struct Bounds {
  long long min_index;
  long long max_src;
  long long max_dst;
  int unsorted;
  int pad;
};

template <typename Index>
__global__ void bounds_kernel(const Index* __restrict__ src, const Index* __restrict__ dst, int64_t edges,
                              Bounds* __restrict__ result) {
  long long lo = INT64_MAX, hi_s = INT64_MIN, hi_d = INT64_MIN;
  int unsorted = 0;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < edges;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const long long s = src[e], d = dst[e];
    lo = min(lo, min(s, d));
    hi_s = max(hi_s, s);
    hi_d = max(hi_d, d);
    if (e > 0 && dst[e - 1] > d) unsorted = 1;
  }
  for (int offset = 16; offset > 0; offset >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, offset));
    hi_s = max(hi_s, __shfl_xor_sync(0xffffffffu, hi_s, offset));
    hi_d = max(hi_d, __shfl_xor_sync(0xffffffffu, hi_d, offset));
    unsorted |= __shfl_xor_sync(0xffffffffu, unsorted, offset);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&result->min_index, lo);
    atomicMax(&result->max_src, hi_s);
    atomicMax(&result->max_dst, hi_d);
    if (unsorted) atomicOr(&result->unsorted, 1);
  }
}

__global__ void init_bounds(Bounds* result) {
  result->min_index = INT64_MAX;
  result->max_src = INT64_MIN;
  result->max_dst = INT64_MIN;
  result->unsorted = 0;
}

// ---- the tables -------------------------------------------------------------------------------------------------------
// Everything about nodes comes from one radix sort and one scan.  With E edges and `span` = E + 32, the sort keys are
//   destination rows   E - degree                                         -> node_order
//   source rows        span + E - degree                                  -> source_node_order
//   source rows again  2 span + (31 - r) (E / 32 + 1) + E / 32 - degree / 32,  r = degree % 32
// The third set ranks the pieces of source rows that are shorter than 32 edges: by length, then by degree, then by
// node.  The scan runs over the degrees in node_order (for the tiers), the numbers of full pieces in source_node_order
// (where a row's full pieces stand in the order of pieces) and the numbers of pieces by node (the pieces' row
// pointers).  Sums are taken modulo 2^32: only differences within a set, which are smaller, are used.
// What bounds it is the number of dependent launches, 3 to 17 us each: 16 of them, 135 us on the device for 1.05 M edges
// and 20,000 nodes, 201 us for the whole call.  Graphs whose rows all have at most 255 edges are built by counting
// (graph_short.cuh) in 88; this is the way for longer rows, for luna_graph_build, and for graphs of over a million nodes.
struct TableSizes {
  int64_t nodes, src_nodes, edges;
  bool segments;
  __host__ __device__ int64_t span() const { return edges + 32; }
  __host__ __device__ int64_t items() const { return nodes + src_nodes * (segments ? 2 : 1); }
};

// Narrow copies of the edge list and the identity permutation.  An index out of its range, or an unsorted destination,
// sets `bad`, and the kernels that follow then do nothing.
template <typename Index>
__global__ void copy_edges(const Index* __restrict__ src, const Index* __restrict__ dst, TableSizes z,
                           int32_t* __restrict__ src_out, int32_t* __restrict__ dst_out, int32_t* __restrict__ iota,
                           int* __restrict__ bad) {
  const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= z.edges) return;
  const int64_t s = src[e], d = dst[e];
  src_out[e] = static_cast<int32_t>(s);
  dst_out[e] = static_cast<int32_t>(d);
  iota[e] = static_cast<int32_t>(e);
  if (s < 0 || s >= z.src_nodes || d < 0 || d >= z.nodes || (e > 0 && dst[e - 1] > dst[e])) *bad = 1;
}

__device__ __forceinline__ int64_t first_not_below(const int32_t* __restrict__ sorted, int64_t count, int64_t value) {
  int64_t lo = 0, hi = count;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (sorted[mid] < value)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Row pointers by binary search in the two sorted edge lists, and the sort keys.  A warp makes 31 rows; its last lane only
// finds where the next begins.  For 1.05 M edges and 20,000 nodes: 12 us, after 7 us of copy_edges; copies with a count of
// the rows by atomics took 27 us, behind 69 us of a bounds scan whose every warp went to the same three words.
template <typename Key>
__global__ void row_pointers(const int32_t* __restrict__ dst, const int32_t* __restrict__ sorted_src, TableSizes z,
                             int32_t* __restrict__ dst_rowptr, int32_t* __restrict__ src_rowptr, Key* __restrict__ keys,
                             int32_t* __restrict__ values, const int* __restrict__ bad) {
  if (*bad) return;
  const int lane = threadIdx.x & 31;
  int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t dst_warps = (z.nodes + 31) / 31;  // nodes + 1 pointers, 31 to a warp
  const bool by_src = warp >= dst_warps;
  if (by_src) warp -= dst_warps;
  const int64_t rows = by_src ? z.src_nodes : z.nodes, n = warp * 31 + lane;
  const int64_t begin = n >= rows ? z.edges : first_not_below(by_src ? sorted_src : dst, z.edges, n);
  const int64_t end = __shfl_down_sync(0xffffffffu, begin, 1);
  if (lane == 31 || n > rows) return;
  (by_src ? src_rowptr : dst_rowptr)[n] = static_cast<int32_t>(begin);
  if (n == rows) return;
  const int64_t degree = end - begin, item = by_src ? z.nodes + n : n;
  keys[item] = static_cast<Key>((by_src ? z.span() : 0) + z.edges - degree);
  values[item] = static_cast<int32_t>(n);
  if (by_src && z.segments) {
    const int64_t full = degree >> 5, rest = degree & 31;
    keys[z.nodes + z.src_nodes + n] =
        static_cast<Key>(2 * z.span() + (31 - rest) * (z.edges / 32 + 1) + z.edges / 32 - full);
    values[z.nodes + z.src_nodes + n] = static_cast<int32_t>(n);
  }
}

template <typename Key>
struct ScanInput {
  const Key* keys;  // sorted
  const int32_t* src_rowptr;
  TableSizes z;
  __host__ __device__ uint32_t operator()(int64_t i) const {
    if (i < z.nodes) return static_cast<uint32_t>(z.edges - static_cast<int64_t>(keys[i]));
    if (i < z.nodes + z.src_nodes)
      return static_cast<uint32_t>((z.edges + z.span() - static_cast<int64_t>(keys[i])) >> 5);
    const int64_t n = i - z.nodes - z.src_nodes;
    if (n >= z.src_nodes) return 0u;
    const uint32_t pieces = (static_cast<uint32_t>(src_rowptr[n + 1] - src_rowptr[n]) + 31u) >> 5;
    return pieces > 0u ? pieces : 1u;
  }
};

// Per sorted item: the orders, the tiers, and where the pieces of a source row stand in the order of pieces.  With F full
// pieces among S: the full ones come first, then those of 31, 30, ... edges, and the rows without edges end the list.
__global__ void node_tables(const int32_t* __restrict__ sorted, const uint32_t* __restrict__ scan, TableSizes z,
                            int32_t* __restrict__ node_order, int32_t* __restrict__ source_node_order,
                            int32_t* __restrict__ tiers, const int32_t* __restrict__ src_rowptr,
                            int32_t* __restrict__ full_at, int32_t* __restrict__ part_at,
                            int32_t* __restrict__ segment_rowptr, const int* __restrict__ bad) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= z.items() || *bad) return;
  const int32_t n = sorted[i];
  const int64_t second = z.nodes, third = z.nodes + z.src_nodes;
  if (i < second) {
    node_order[i] = n;
    if (!z.segments) return;
    for (int k = 1; k < 4; ++k) {  // tier k ends with the row that brings the edges to k quarters
      const uint32_t quarter = static_cast<uint32_t>(static_cast<int64_t>(k) * z.edges / 4);
      if ((i == 0 || scan[i] < quarter) && scan[i + 1] >= quarter) tiers[k - 1] = static_cast<int32_t>(i + 1);
    }
  } else if (i < third) {
    source_node_order[i - second] = n;
    if (z.segments) full_at[n] = static_cast<int32_t>(scan[i] - scan[second]);
  } else {
    const int64_t rank = i - third;
    const int64_t full = static_cast<uint32_t>(scan[third] - scan[second]);
    const int64_t all = static_cast<uint32_t>(scan[third + z.src_nodes] - scan[third]);
    part_at[n] = static_cast<int32_t>(src_rowptr[n + 1] == src_rowptr[n] ? all - (z.src_nodes - rank) : full + rank);
    segment_rowptr[rank] = static_cast<int32_t>(scan[i] - scan[third]);
    if (rank + 1 == z.src_nodes) segment_rowptr[z.src_nodes] = static_cast<int32_t>(all);
  }
}

__global__ void segment_tables(const int32_t* __restrict__ segment_rowptr, const int32_t* __restrict__ src_rowptr,
                               const int32_t* __restrict__ full_at, const int32_t* __restrict__ part_at, TableSizes z,
                               int32_t* __restrict__ nodes, int32_t* __restrict__ begin, int32_t* __restrict__ end,
                               int32_t* __restrict__ order, const int* __restrict__ bad) {
  const int64_t piece = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (*bad || piece >= segment_rowptr[z.src_nodes]) return;
  const int64_t n = first_not_below(segment_rowptr, z.src_nodes + 1, piece + 1) - 1;
  const int32_t local = static_cast<int32_t>(piece) - segment_rowptr[n];
  const int32_t row = src_rowptr[n], row_end = src_rowptr[n + 1], from = row + 32 * local;
  nodes[piece] = static_cast<int32_t>(n);
  begin[piece] = from;
  end[piece] = min(from + 32, row_end);
  order[local < (row_end - row) >> 5 ? full_at[n] + local : part_at[n]] = static_cast<int32_t>(piece);
}

size_t align_up(size_t v) { return (v + 255) / 256 * 256; }

int bits_for(uint64_t max_value) {
  int bits = 1;
  while (bits < 64 && (max_value >> bits) != 0) ++bits;
  return bits;
}

struct ScratchLayout {
  size_t bad, src_sorted, iota, keys, keys_sorted, values, values_sorted, scan, full_at, part_at, cub_temp, cub_bytes, total;
};

// Keys of 32 bits reach 1.4 billion edges.
bool wide_keys(const TableSizes& z) { return 3 * static_cast<uint64_t>(z.span()) > 0xffffffffull; }

template <typename Key>
size_t cub_need(const TableSizes& z) {
  size_t edge_sort = 0, node_sort = 0, scan = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, edge_sort, static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr),
                                  static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr), z.edges);
  cub::DeviceRadixSort::SortPairs(nullptr, node_sort, static_cast<const Key*>(nullptr), static_cast<Key*>(nullptr),
                                  static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr), z.items());
  cub::DeviceScan::ExclusiveSum(nullptr, scan,
                                thrust::make_transform_iterator(thrust::counting_iterator<int64_t>(0), ScanInput<Key>{}),
                                static_cast<uint32_t*>(nullptr), z.items() + 1);
  return std::max(edge_sort, std::max(node_sort, scan)) + 256;
}

ScratchLayout layout(TableSizes z) {
  z.segments = true;
  ScratchLayout l{};
  const size_t edges = static_cast<size_t>(std::max<int64_t>(z.edges, 1)), items = static_cast<size_t>(z.items()) + 1;
  const size_t key = wide_keys(z) ? 8 : 4;
  l.cub_bytes = wide_keys(z) ? cub_need<uint64_t>(z) : cub_need<uint32_t>(z);
  size_t cursor = 0;
  auto take = [&](size_t bytes) {
    const size_t at = cursor;
    cursor += align_up(bytes);
    return at;
  };
  l.bad = take(sizeof(Bounds));
  l.src_sorted = take(edges * 4);
  l.iota = take(edges * 4);
  l.keys = take(items * key);
  l.keys_sorted = take(items * key);
  l.values = take(items * 4);
  l.values_sorted = take(items * 4);
  l.scan = take(items * 4);
  l.full_at = take(static_cast<size_t>(z.src_nodes) * 4 + 4);
  l.part_at = take(static_cast<size_t>(z.src_nodes) * 4 + 4);
  l.cub_temp = take(l.cub_bytes);
  ShortTables t{};
  t.nodes = z.nodes;
  t.src_nodes = z.src_nodes;
  t.edges = z.edges;
  size_t zeroed = 0;
  l.total = short_rows_likely(z.nodes, z.src_nodes, z.edges) ? std::max(cursor, short_layout(&t, nullptr, &zeroed)) : cursor;
  return l;
}

unsigned grid(int64_t threads) { return static_cast<unsigned>(std::max<int64_t>(1, ceil_div(threads, kThreads))); }

// Launches everything; *bad (in the scratch) tells whether the edge list was fit for it.  `copied`: the narrow copies and the
// identity are there already, and checked, and *bad is zero.
template <typename Key>
int build_tables(const void* src, const void* dst, int index_bits, const TableSizes& z, const luna_graph_out& out,
                 const luna_graph_pieces* pieces, unsigned char* scratch, const ScratchLayout& l, bool copied, cudaStream_t stream) {
  auto at = [&](size_t offset) { return reinterpret_cast<int32_t*>(scratch + offset); };
  int* bad = at(l.bad);
  Key *keys = reinterpret_cast<Key*>(scratch + l.keys), *keys_sorted = reinterpret_cast<Key*>(scratch + l.keys_sorted);
  uint32_t* scan = reinterpret_cast<uint32_t*>(scratch + l.scan);
  void* temp = scratch + l.cub_temp;
  size_t temp_bytes = l.cub_bytes;
  if (!copied) LUNA_CUDA_CHECK(cudaMemsetAsync(bad, 0, sizeof(int), stream));
  if (z.edges > 0) {
    int32_t* iota = pieces ? pieces->edge_ids_by_dst : at(l.iota);
    if (!copied) {
      if (index_bits == 64)
        copy_edges<int64_t><<<grid(z.edges), kThreads, 0, stream>>>(static_cast<const int64_t*>(src),
                                                                    static_cast<const int64_t*>(dst), z, out.src, out.dst, iota, bad);
      else
        copy_edges<int32_t><<<grid(z.edges), kThreads, 0, stream>>>(static_cast<const int32_t*>(src),
                                                                    static_cast<const int32_t*>(dst), z, out.src, out.dst, iota, bad);
      LUNA_LAUNCH_CHECK("graph edge copies");
    }
    // stable grouping of edge ids by source
    LUNA_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(temp, temp_bytes, static_cast<const int32_t*>(out.src), at(l.src_sorted),
                                                    static_cast<const int32_t*>(iota), out.edge_ids_by_src, z.edges, 0,
                                                    bits_for(static_cast<uint64_t>(std::max<int64_t>(z.src_nodes - 1, 1))), stream));
  }
  row_pointers<Key><<<grid(((z.nodes + 31) / 31 + (z.src_nodes + 31) / 31) * 32), kThreads, 0, stream>>>(
      out.dst, at(l.src_sorted), z, out.dst_rowptr, out.src_rowptr, keys, at(l.values), bad);
  LUNA_LAUNCH_CHECK("graph row pointers");
  if (z.items() == 0) return LUNA_OK;
  temp_bytes = l.cub_bytes;
  LUNA_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(temp, temp_bytes, static_cast<const Key*>(keys), keys_sorted,
                                                  static_cast<const int32_t*>(at(l.values)), at(l.values_sorted), z.items(), 0,
                                                  bits_for(3 * static_cast<uint64_t>(z.span())), stream));
  if (z.segments) {
    temp_bytes = l.cub_bytes;
    LUNA_CUDA_CHECK(cub::DeviceScan::ExclusiveSum(
        temp, temp_bytes,
        thrust::make_transform_iterator(thrust::counting_iterator<int64_t>(0), ScanInput<Key>{keys_sorted, out.src_rowptr, z}),
        scan, z.items() + 1, stream));
  }
  node_tables<<<grid(z.items()), kThreads, 0, stream>>>(at(l.values_sorted), scan, z, out.node_order, out.source_node_order,
                                                       pieces ? pieces->node_tiers : nullptr, out.src_rowptr, at(l.full_at),
                                                       at(l.part_at), pieces ? pieces->segment_rowptr : nullptr, bad);
  LUNA_LAUNCH_CHECK("graph node tables");
  if (z.segments) {
    segment_tables<<<grid(z.src_nodes + z.edges / 32), kThreads, 0, stream>>>(
        pieces->segment_rowptr, out.src_rowptr, at(l.full_at), at(l.part_at), z, pieces->segment_nodes,
        pieces->segment_begin, pieces->segment_end, pieces->segment_order, bad);
    LUNA_LAUNCH_CHECK("graph segment tables");
  }
  return LUNA_OK;
}

int check_tables(const void* src, const void* dst, int index_bits, const TableSizes& z, const luna_graph_out* out,
                 const void* scratch, int64_t scratch_bytes, ScratchLayout* l) {
  if (!out) return fail(LUNA_ERR_INVALID_ARGUMENT, "null output table set");
  if (z.nodes < 0 || z.edges < 0) return fail(LUNA_ERR_INVALID_ARGUMENT, "negative graph size");
  if (std::max(z.nodes, z.src_nodes) >= (1LL << 31) - 1024 || z.edges >= (1LL << 31) - 1024)
    return fail(LUNA_ERR_OVERFLOW, "graph exceeds the 32-bit index range of this build");
  if (index_bits != 32 && index_bits != 64) return fail(LUNA_ERR_INVALID_ARGUMENT, "index_bits must be 32 or 64");
  if (!out->dst_rowptr || !out->src_rowptr) return fail(LUNA_ERR_INVALID_ARGUMENT, "row pointer outputs missing");
  if (z.edges > 0 && (!src || !dst || !out->src || !out->dst || !out->edge_ids_by_src))
    return fail(LUNA_ERR_INVALID_ARGUMENT, "edge tables missing");
  if ((z.nodes > 0 && !out->node_order) || (z.src_nodes > 0 && !out->source_node_order))
    return fail(LUNA_ERR_INVALID_ARGUMENT, "node order outputs missing");
  *l = layout(z);
  if (!scratch || scratch_bytes < static_cast<int64_t>(l->total))
    return fail(LUNA_ERR_SCRATCH, "scratch too small: need %zu bytes", l->total);
  return LUNA_OK;
}

}  // namespace
}  // namespace luna

using namespace luna;

extern "C" int64_t luna_graph_scratch_bytes(int64_t num_nodes, int64_t num_edges) {
  if (num_nodes < 0 || num_edges < 0) return -1;
  return static_cast<int64_t>(layout(TableSizes{num_nodes, num_nodes, num_edges, true}).total);
}

extern "C" int luna_graph_bounds(const void* src, const void* dst, int index_bits, int64_t num_edges,
                                 int64_t* min_index, int64_t* max_src, int64_t* max_dst, int* unsorted,
                                 void* scratch, int64_t scratch_bytes, void* stream_) {
  clear_error();
  if (!min_index || !max_src || !max_dst || !unsorted) return fail(LUNA_ERR_INVALID_ARGUMENT, "null result pointer");
  *min_index = 0;
  *max_src = *max_dst = -1;
  *unsorted = 0;
  if (num_edges == 0) return LUNA_OK;
  if (!src || !dst) return fail(LUNA_ERR_INVALID_ARGUMENT, "null edge list");
  if (index_bits != 32 && index_bits != 64) return fail(LUNA_ERR_INVALID_ARGUMENT, "index_bits must be 32 or 64");
  if (!scratch || scratch_bytes < static_cast<int64_t>(sizeof(Bounds)))
    return fail(LUNA_ERR_SCRATCH, "scratch too small for the bounds scan");
  auto stream = static_cast<cudaStream_t>(stream_);
  auto* result = static_cast<Bounds*>(scratch);
  init_bounds<<<1, 1, 0, stream>>>(result);
  const int blocks = static_cast<int>(std::min<int64_t>(ceil_div(num_edges, kThreads), 592));
  if (index_bits == 64)
    bounds_kernel<int64_t><<<blocks, kThreads, 0, stream>>>(static_cast<const int64_t*>(src),
                                                            static_cast<const int64_t*>(dst), num_edges, result);
  else
    bounds_kernel<int32_t><<<blocks, kThreads, 0, stream>>>(static_cast<const int32_t*>(src),
                                                            static_cast<const int32_t*>(dst), num_edges, result);
  LUNA_LAUNCH_CHECK("graph bounds scan");
  Bounds host{};
  LUNA_CUDA_CHECK(cudaMemcpyAsync(&host, result, sizeof(Bounds), cudaMemcpyDeviceToHost, stream));
  LUNA_CUDA_CHECK(cudaStreamSynchronize(stream));
  *min_index = host.min_index;
  *max_src = host.max_src;
  *max_dst = host.max_dst;
  *unsorted = host.unsorted;
  return LUNA_OK;
}

extern "C" int luna_graph_build(const void* src, const void* dst, int index_bits, int64_t num_nodes,
                                int64_t num_src_nodes, int64_t num_edges, const luna_graph_out* out, void* scratch,
                                int64_t scratch_bytes, void* stream_) {
  clear_error();
  if (num_src_nodes <= 0) num_src_nodes = num_nodes;
  const TableSizes z{num_nodes, num_src_nodes, num_edges, false};
  ScratchLayout l{};
  const int rc = check_tables(src, dst, index_bits, z, out, scratch, scratch_bytes, &l);
  if (rc != LUNA_OK) return rc;
  auto stream = static_cast<cudaStream_t>(stream_);
  auto* base = static_cast<unsigned char*>(scratch);
  return wide_keys(z) ? build_tables<uint64_t>(src, dst, index_bits, z, *out, nullptr, base, l, false, stream)
                      : build_tables<uint32_t>(src, dst, index_bits, z, *out, nullptr, base, l, false, stream);
}

extern "C" int luna_graph_build_all(const void* src, const void* dst, int index_bits, int64_t num_nodes,
                                    int64_t num_src_nodes, int64_t num_edges, const luna_graph_out* out,
                                    const luna_graph_pieces* pieces, int* bad, int64_t* num_segments, void* scratch,
                                    int64_t scratch_bytes, void* stream_) {
  clear_error();
  if (num_src_nodes <= 0) num_src_nodes = num_nodes;
  const TableSizes z{num_nodes, num_src_nodes, num_edges, true};
  ScratchLayout l{};
  const int rc = check_tables(src, dst, index_bits, z, out, scratch, scratch_bytes, &l);
  if (rc != LUNA_OK) return rc;
  if (num_nodes == 0 || num_edges == 0) return fail(LUNA_ERR_INVALID_ARGUMENT, "a graph with nodes and edges is required");
  if (num_src_nodes + num_edges / 32 >= (1LL << 31) - 1024)
    return fail(LUNA_ERR_OVERFLOW, "graph exceeds the 32-bit index range of this build");
  if (!pieces || !bad || !num_segments) return fail(LUNA_ERR_INVALID_ARGUMENT, "null result pointer");
  if (!pieces->edge_ids_by_dst || !pieces->node_tiers || !pieces->segment_nodes || !pieces->segment_begin ||
      !pieces->segment_end || !pieces->segment_rowptr || !pieces->segment_order)
    return fail(LUNA_ERR_INVALID_ARGUMENT, "segment tables missing");
  auto stream = static_cast<cudaStream_t>(stream_);
  auto* base = static_cast<unsigned char*>(scratch);
  const bool copied = short_rows_likely(num_nodes, num_src_nodes, num_edges);
  if (copied) {
    ShortTables t{};
    t.nodes = num_nodes;
    t.src_nodes = num_src_nodes;
    t.edges = num_edges;
    t.src = out->src;
    t.dst = out->dst;
    t.iota = pieces->edge_ids_by_dst;
    t.dst_rowptr = out->dst_rowptr;
    t.src_rowptr = out->src_rowptr;
    t.edge_ids = out->edge_ids_by_src;
    t.node_order = out->node_order;
    t.source_node_order = out->source_node_order;
    t.tiers = pieces->node_tiers;
    t.segment_nodes = pieces->segment_nodes;
    t.segment_begin = pieces->segment_begin;
    t.segment_end = pieces->segment_end;
    t.segment_rowptr = pieces->segment_rowptr;
    t.segment_order = pieces->segment_order;
    size_t zeroed = 0;
    short_layout(&t, base, &zeroed);
    const int launched = index_bits == 64 ? short_tables<int64_t>(src, dst, t, zeroed, stream)
                                          : short_tables<int32_t>(src, dst, t, zeroed, stream);
    if (launched != LUNA_OK) return launched;
    int head[kHeadWords] = {};
    LUNA_CUDA_CHECK(cudaMemcpyAsync(head, t.head, sizeof(head), cudaMemcpyDeviceToHost, stream));
    LUNA_CUDA_CHECK(cudaStreamSynchronize(stream));
    *bad = head[kHeadUnfit];
    *num_segments = *bad ? 0 : head[kHeadPieces];
    if (*bad || !head[kHeadLongRow]) return LUNA_OK;
    // the flag of unfit edges, which is zero, lies where that of the general kernels does, and the rest of the scratch is theirs
    static_assert(kHeadUnfit == 0, "the general kernels' flag is the scratch's first word");
  }
  const int built = wide_keys(z) ? build_tables<uint64_t>(src, dst, index_bits, z, *out, pieces, base, l, copied, stream)
                                 : build_tables<uint32_t>(src, dst, index_bits, z, *out, pieces, base, l, copied, stream);
  if (built != LUNA_OK) return built;
  int flag = 0;
  int32_t count = 0;
  if (!copied) LUNA_CUDA_CHECK(cudaMemcpyAsync(&flag, base + l.bad, sizeof(int), cudaMemcpyDeviceToHost, stream));
  LUNA_CUDA_CHECK(cudaMemcpyAsync(&count, pieces->segment_rowptr + num_src_nodes, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
  LUNA_CUDA_CHECK(cudaStreamSynchronize(stream));
  *bad = flag;
  *num_segments = flag ? 0 : count;
  return LUNA_OK;
}
