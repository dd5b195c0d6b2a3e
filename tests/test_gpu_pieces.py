"""A graph's work done in pieces: destination ranges, the host-streaming executor and the overlapped shard step.

All three rest on the same two facts, checked here against one call on the whole graph: the edges of a destination
range are a contiguous slice of the edge list whose per-edge tensors are row ranges of the whole graph's, and the
source-row gradients of the pieces add up (``luna_uvu_conv_bwd_add_gx``).
"""

import pytest
import torch

import bench_workloads as workloads
import lunaequivariance_b200 as luna
from lunaequivariance_b200 import conv as conv_mod
from lunaequivariance_b200 import sharded
from lunaequivariance_b200.streaming import HostStreamedConv
from tests.helpers import all_paths, assert_close, config, random_graph

pytestmark = pytest.mark.gpu
DEVICE = "cuda"


def problem(name, dtype, atoms=240, seed=5):
    in1, in2, out, instructions, _ = config(name)
    module = luna.TensorProductConv(in1, in2, out, instructions, internal_weights=False, shared_weights=False,
                                    dtype=dtype)
    pos, box, cells = workloads.periodic_positions(atoms, workloads.DENSITY, 0, DEVICE, workloads.CUTOFF)
    src, dst, _ = workloads.radius_graph_periodic(pos, box, workloads.CUTOFF, cells)
    graph = luna.make_graph(src, dst, atoms)
    op = module.op
    generator = torch.Generator(device=DEVICE).manual_seed(seed)
    rand = lambda *shape: torch.randn(*shape, generator=generator, dtype=dtype, device=DEVICE)
    tensors = dict(x=rand(atoms, op.in1_dim), y=rand(graph.num_edges, op.in2_dim),
                   w=rand(graph.num_edges, op.weight_numel), g=rand(atoms, op.out_dim))
    return module, op, graph, tensors, (src, dst)


def whole(op, graph, t):
    out = conv_mod.run_forward(op, t["x"], t["y"], t["w"], graph)
    gx, gy, gw = conv_mod.run_backward(op, t["x"], t["y"], t["w"], t["g"], graph)
    return dict(out=out, gx=gx, gy=gy, gw=gw)


@pytest.mark.parametrize("name,dtype", [("cfg2", torch.float32), ("cfg5", torch.float32), ("cfg2", torch.float64),
                                        ("fixture", torch.float32)])
def test_destination_ranges_add_up(name, dtype):
    module, op, graph, t, _ = problem(name, dtype)
    ref = whole(op, graph, t)
    nodes = graph.num_nodes
    out = torch.full_like(ref["out"], float("nan"))
    gy, gw = torch.full_like(ref["gy"], float("nan")), torch.full_like(ref["gw"], float("nan"))
    gx = torch.zeros_like(ref["gx"])
    covered = 0
    for begin, end in ((0, 17), (17, 17), (17, 150), (150, nodes)):  # uneven, one empty
        piece, e0, e1 = graph.destination_range(begin, end)
        assert piece.num_nodes == end - begin and piece.num_edges == e1 - e0 and piece.source_rows == nodes
        covered += e1 - e0
        conv_mod.run_forward(op, t["x"], t["y"][e0:e1], t["w"][e0:e1], piece, out=out[begin:end])
        conv_mod.run_backward(op, t["x"], t["y"][e0:e1], t["w"][e0:e1], t["g"][begin:end], piece,
                              out=(gx, gy[e0:e1], gw[e0:e1]), add_gx=True)
    op.check_status()
    assert covered == graph.num_edges
    assert torch.equal(out, ref["out"]) and torch.equal(gy, ref["gy"]) and torch.equal(gw, ref["gw"])
    assert_close(gx, ref["gx"].cpu(), dtype, f"{name} gx summed over pieces")
    assert graph.destination_range(17, 150)[0] is graph.destination_range(17, 150)[0]  # cached


@pytest.mark.parametrize("cuts,same", [((0, 1600, 3200), True), ((0, 800, 1600, 2400, 3200), False)])
def test_pieces_of_a_graph_that_hands_out_tiles(cuts, same, monkeypatch):
    """With two warps per CTA a whole graph of 165,000 edges hands out tiles; so do its halves, and then every row of ``out`` is
    the same to the bit.  Its quarters are cut into equal parts of their edges, and sum rows in another order."""
    monkeypatch.setenv("LUNA_B200_MAXW", "2")
    module, op, graph, t, _ = problem("cfg5", torch.float32, atoms=3200)
    teams = 2 * torch.cuda.get_device_properties(DEVICE).multi_processor_count
    assert graph.num_edges > 256 * teams
    ref = whole(op, graph, t)
    for begin, end in zip(cuts[:-1], cuts[1:]):
        piece, e0, e1 = graph.destination_range(begin, end)
        assert (e1 - e0 > 256 * teams) == same
        out = conv_mod.run_forward(op, t["x"], t["y"][e0:e1], t["w"][e0:e1], piece)
        _, gy, gw = conv_mod.run_backward(op, t["x"], t["y"][e0:e1], t["w"][e0:e1], t["g"][begin:end], piece,
                                          (False, True, True))
        assert torch.equal(gy, ref["gy"][e0:e1]) and torch.equal(gw, ref["gw"][e0:e1])
        assert_close(out, ref["out"][begin:end].cpu(), torch.float32, f"rows {begin} to {end}")
        assert not same or torch.equal(out, ref["out"][begin:end])
    op.check_status()


# Ten teams fit the shared memory in FP64, and eight, twelve or two at other widths: a row's parts do not depend on how many rows
# a graph has, up to three per SM, as long as it has enough edges for them.
@pytest.mark.parametrize("mul,degree,dtype", [(64, 2, torch.float64), (96, 2, torch.float64), (48, 2, torch.float32),
                                              (96, 3, torch.float32), (48, 1, torch.float64)])
def test_pieces_of_few_rows(mul, degree, dtype):
    out, ref = _rows_of_pieces(mul, degree, dtype, 400, 400 * 36, (0, 30, 148, 149, 400))
    assert torch.equal(out, ref)


# With two edges per row every launch hands out tiles, however few the rows.
@pytest.mark.parametrize("mul,degree,dtype", [(48, 2, torch.float32), (96, 2, torch.float64), (32, 2, torch.float32)])
def test_pieces_of_a_sparse_graph(mul, degree, dtype):
    out, ref = _rows_of_pieces(mul, degree, dtype, 3000, 6000, (0, 24, 400, 1500, 3000))
    assert torch.equal(out, ref)


def _rows_of_pieces(mul, degree, dtype, nodes, edges, cuts):
    features = "+".join(f"{mul}x{l}{'eo'[l % 2]}" for l in range(degree + 1))
    attributes = "+".join(f"1x{l}{'eo'[l % 2]}" for l in range(degree + 1))
    op = luna.TensorProductConv(features, attributes, features, all_paths(features, attributes, features),
                                internal_weights=False, shared_weights=False, dtype=dtype).op
    generator = torch.Generator().manual_seed(nodes + mul)
    exact = edges // nodes if edges >= 36 * nodes else None  # rows of one length: their groups are the same in all pieces
    src, dst = random_graph(nodes, edges, generator, exact_degree=exact)
    graph = luna.make_graph(src.to(DEVICE), dst.to(DEVICE), nodes)
    rand = lambda *shape: torch.randn(*shape, generator=generator, dtype=torch.float64).to(dtype).to(DEVICE)
    x, y, w = rand(nodes, op.in1_dim), rand(edges, op.in2_dim), rand(edges, op.weight_numel)
    ref = conv_mod.run_forward(op, x, y, w, graph)
    out = torch.full_like(ref, float("nan"))
    for begin, end in zip(cuts[:-1], cuts[1:]):
        piece, e0, e1 = graph.destination_range(begin, end)
        conv_mod.run_forward(op, x, y[e0:e1], w[e0:e1], piece, out=out[begin:end])
    op.check_status()
    return out, ref


def test_add_gx_needs_a_tensor_and_out_shapes_are_checked():
    module, op, graph, t, _ = problem("cfg5", torch.float32, atoms=60)
    with pytest.raises(ValueError, match="add_gx"):
        conv_mod.run_backward(op, t["x"], t["y"], t["w"], t["g"], graph, add_gx=True)
    with pytest.raises(ValueError, match="out must be"):
        conv_mod.run_forward(op, t["x"], t["y"], t["w"], graph, out=torch.empty(3, 3, device=DEVICE))
    with pytest.raises(ValueError, match="outside"):
        graph.destination_range(5, graph.num_nodes + 1)


@pytest.mark.parametrize("name,dtype,chunks", [("cfg2", torch.float32, 5), ("cfg5", torch.float32, 1),
                                                ("cfg2", torch.float64, 3)])
def test_host_streamed_step_matches_one_call(name, dtype, chunks):
    module, op, graph, t, _ = problem(name, dtype, atoms=300)
    ref = whole(op, graph, t)
    host = {k: v.cpu().pin_memory() for k, v in t.items()}
    streamed = HostStreamedConv(op, graph, chunks=chunks)
    assert 1 <= len(streamed.pieces) <= chunks
    for _ in range(2):  # buffers and host outputs are reused from step to step
        out, gx, gy, gw = streamed.step(host["x"], host["y"], host["w"], host["g"])
    op.check_status()
    assert out.device.type == "cpu" and gw.shape == ref["gw"].shape
    assert torch.equal(out, ref["out"].cpu()) and torch.equal(gy, ref["gy"].cpu())
    assert torch.equal(gw, ref["gw"].cpu())
    assert_close(gx, ref["gx"].cpu(), dtype, f"{name} streamed gx")
    # node features already on the device: gx stays there
    out2, gx_device, _, _ = streamed.step(t["x"], host["y"], host["w"], t["g"])
    assert gx_device.is_cuda and torch.equal(gx_device.cpu(), gx) and torch.equal(out2, ref["out"].cpu())
    with pytest.raises(ValueError, match="host tensor"):
        streamed.step(host["x"], t["y"], host["w"], host["g"])


@pytest.mark.parametrize("rank", [0, 1, 2])
def test_overlapped_step_on_one_rank_of_a_partition(rank):
    """The piece schedule of the overlapped step (interior, then the two ends; ends first in the backward), with the
    halo rows supplied by hand in place of the exchange, against plain calls on the shard's graph."""
    dtype = torch.float32
    module, op, _, t, (src, dst) = problem("cfg2", dtype, atoms=300)
    counts = (110, 50, 140)
    begin = sum(counts[:rank])
    mine = (dst >= begin) & (dst < begin + counts[rank])
    shard = sharded.make_graph_shard(src[mine], dst[mine], counts, rank, exchange=False)
    lo, hi = shard.interior
    assert 0 <= lo <= hi <= counts[rank]
    remote = shard.graph.src.long() >= counts[rank]
    touched = torch.unique(shard.graph.dst[remote].long())
    assert not ((touched >= lo) & (touched < hi)).any()  # interior destinations read owned rows only
    x_local, halo = t["x"][begin:begin + counts[rank]], t["x"][shard.halo_ids]
    y, w, g = t["y"][mine], t["w"][mine], t["g"][begin:begin + counts[rank]]
    x_full = torch.cat([x_local, halo])
    ref_out = conv_mod.run_forward(op, x_full, y, w, shard.graph)
    ref_gx, ref_gy, ref_gw = conv_mod.run_backward(op, x_full, y, w, g, shard.graph)
    events = [torch.cuda.Event(enable_timing=True) for _ in range(5)]
    out, gx_full, gy, gw = sharded.overlapped_step(op, x_local, y, w, g, shard, halo_rows=halo, events=events)
    torch.cuda.synchronize()
    op.check_status()
    assert events[0].elapsed_time(events[4]) > 0
    assert torch.equal(out, ref_out) and torch.equal(gy, ref_gy) and torch.equal(gw, ref_gw)
    assert_close(gx_full, ref_gx.cpu(), dtype, f"rank {rank} gx of the compact buffer")


def test_host_streamed_step_on_tiny_and_empty_graphs():
    in1, in2, out, instructions, _ = config("fixture")
    dtype = torch.float32
    module = luna.TensorProductConv(in1, in2, out, instructions, internal_weights=False, shared_weights=False,
                                    dtype=dtype)
    op = module.op
    nodes = 7
    dst = torch.tensor([0, 0, 1, 1, 1, 4, 4, 4, 4, 6], device=DEVICE)  # destinations 2, 3, 5 have no edge
    src = torch.tensor([1, 6, 0, 2, 3, 4, 5, 0, 1, 2], device=DEVICE)
    graph = luna.make_graph(src, dst, nodes)
    generator = torch.Generator(device=DEVICE).manual_seed(2)
    rand = lambda *shape: torch.randn(*shape, generator=generator, dtype=dtype, device=DEVICE)
    t = dict(x=rand(nodes, op.in1_dim), y=rand(10, op.in2_dim), w=rand(10, op.weight_numel), g=rand(nodes, op.out_dim))
    ref = whole(op, graph, t)
    streamed = HostStreamedConv(op, graph, chunks=16)  # more chunks than nodes
    assert 1 <= len(streamed.pieces) <= nodes
    host = {k: v.cpu() for k, v in t.items()}  # pageable memory works too
    out_rows, gx, gy, gw = streamed.step(host["x"], host["y"], host["w"], host["g"])
    assert torch.equal(out_rows, ref["out"].cpu()) and torch.equal(gy, ref["gy"].cpu())
    assert torch.equal(gw, ref["gw"].cpu())
    assert_close(gx, ref["gx"].cpu(), dtype, "tiny graph gx")
    assert not out_rows[[2, 3, 5]].any()

    empty = luna.make_graph(src[:0], dst[:0], 4)
    streamed = HostStreamedConv(op, empty, chunks=3)
    out_rows, gx, gy, gw = streamed.step(host["x"][:4], host["y"][:0], host["w"][:0], host["g"][:4])
    assert out_rows.shape == (4, op.out_dim) and not out_rows.any() and not gx.any()
    assert gy.shape == (0, op.in2_dim) and gw.shape == (0, op.weight_numel)
