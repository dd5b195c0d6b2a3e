"""Every table of a graph built on the GPU against the same tables from torch ops on the CPU: exactly."""

from __future__ import annotations

import pytest
import torch

import lunaequivariance_b200 as luna

pytestmark = pytest.mark.gpu

NAMES = ("src", "dst", "dst_rowptr", "src_rowptr", "edge_ids_by_src", "edge_ids_by_dst", "node_order", "source_node_order",
         "node_tiers")
SEGMENTS = ("nodes", "begin", "end", "rowptr", "order")


def _edges(nodes, source_rows, edges, hub, seed):
    generator = torch.Generator().manual_seed(seed)
    src = torch.randint(source_rows, (edges,), generator=generator)
    if hub:  # most edges leave one node, in a number that is a multiple of a segment's length
        src[: edges // 2 // 32 * 32] = source_rows // 2
        src = src[torch.randperm(edges, generator=generator)]
    return src, torch.sort(torch.randint(nodes, (edges,), generator=generator)).values


# one edge; fewer edges than quarters; rows of exactly 31, 32, 33 rows per warp; rows without edges; more source rows than
# destinations and fewer
@pytest.mark.parametrize("nodes,source_rows,edges,hub", [
    (1, 1, 1, False), (3, 3, 2, False), (30, 30, 3, False), (31, 31, 992, False), (32, 32, 1024, True),
    (62, 62, 4_000, True), (500, 500, 300, False), (64, 900, 5_001, False), (900, 7, 5_001, True), (20_011, 20_011, 200_003, True),
])
@pytest.mark.parametrize("index_dtype", [torch.int32, torch.int64])
def test_tables(nodes, source_rows, edges, hub, index_dtype):
    src, dst = (t.to(index_dtype) for t in _edges(nodes, source_rows, edges, hub, nodes + edges))
    other = None if source_rows == nodes else source_rows
    want = luna.make_graph(src, dst, nodes, num_src_nodes=other)
    got = luna.make_graph(src.cuda(), dst.cuda(), nodes, num_src_nodes=other)
    for name in NAMES:
        torch.testing.assert_close(getattr(got, name).cpu(), getattr(want, name), rtol=0, atol=0, msg=name)
    for name in SEGMENTS:
        torch.testing.assert_close(getattr(got.source_segments, name).cpu(), getattr(want.source_segments, name), rtol=0,
                                   atol=0, msg=f"segment {name}")
    assert got.num_src_nodes == want.num_src_nodes and got.can_split == want.can_split


def _compare(src, dst, nodes, source_rows):
    other = None if source_rows == nodes else source_rows
    want = luna.make_graph(src, dst, nodes, num_src_nodes=other)
    got = luna.make_graph(src.cuda(), dst.cuda(), nodes, num_src_nodes=other)
    for name in NAMES:
        torch.testing.assert_close(getattr(got, name).cpu(), getattr(want, name), rtol=0, atol=0, msg=name)
    for name in SEGMENTS:
        torch.testing.assert_close(getattr(got.source_segments, name).cpu(), getattr(want.source_segments, name), rtol=0,
                                   atol=0, msg=f"segment {name}")
    assert got.num_src_nodes == want.num_src_nodes and got.can_split == want.can_split


# Rows of up to 255 edges are counted into place, a longer one anywhere sends the graph to the general sorts: both sides of the
# line, whole blocks of 512 nodes and one more, every length of a row that is sorted in another number of registers, and rows
# without edges.
@pytest.mark.parametrize("longest", [32, 33, 64, 65, 128, 129, 254, 255, 256])
@pytest.mark.parametrize("nodes,source_rows", [(512, 512), (1_025, 1_025), (513, 700), (1_024, 511)])
def test_longest_row(longest, nodes, source_rows):
    generator = torch.Generator().manual_seed(longest + nodes)
    edges = 12 * nodes
    for hub_side in (0, 1):
        rows = (source_rows, nodes)
        ends = [torch.randint(n - 1, (edges,), generator=generator) for n in rows]  # the last row is the long one
        ends[hub_side][torch.randperm(edges, generator=generator)[:longest]] = rows[hub_side] - 1
        order = torch.argsort(ends[1], stable=True)
        _compare(ends[0][order], ends[1][order], nodes, source_rows)


# More blocks of 512 nodes than the last one to count sums at a time: 24 blocks, one node more, and several turns.
@pytest.mark.parametrize("nodes,source_rows,edges", [(12_288, 12_288, 90_001), (12_289, 12_289, 90_001), (20_011, 20_011, 200_003),
                                                     (1_500, 30_011, 100_000), (100_003, 100_003, 300_001)])
def test_many_blocks_of_nodes(nodes, source_rows, edges):
    src, dst = _edges(nodes, source_rows, edges, False, nodes + edges)
    assert max(src.bincount().max(), dst.bincount().max()) < 256
    _compare(src, dst, nodes, source_rows)


# A row that is too long for counting: the sorts begin with the edges that are copied and checked already.
@pytest.mark.parametrize("by_source", [False, True])
def test_long_row_is_copied_once(by_source):
    src, dst = _edges(600, 600, 9_000, False, 3)
    (src if by_source else dst)[:256] = 0
    order = torch.argsort(dst, stable=True)
    src, dst = src[order].cuda(), dst[order].cuda()
    luna.make_graph(src, dst, 600)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as profile:
        luna.make_graph(src, dst, 600)
        torch.cuda.synchronize()
    kernels = [event.name for event in profile.events() if event.device_type == torch.autograd.DeviceType.CUDA]
    assert any("short_edges" in name for name in kernels) and any("segment_tables" in name for name in kernels), kernels
    assert not any("copy_edges" in name for name in kernels), kernels


@pytest.mark.parametrize("src,dst,match", [
    ([0, 4], [0, 1], "at least 5"), ([0, 1], [0, 4], "at least 5"), ([0, -1], [0, 1], "nonnegative"),
    ([0, 1], [1, 0], "sorted"), ([0, 1 << 32], [0, 1], "at least 4294967297"),
])
def test_unfit_edge_lists_are_refused(src, dst, match):
    with pytest.raises(ValueError, match=match):
        luna.make_graph(torch.tensor(src, device="cuda"), torch.tensor(dst, device="cuda"), 4)
