"""Kernels that are launched before the one ahead of them has ended: chains of launches give the same bits as with a
synchronisation after every one.

``test_chains_without_synchronisation`` is what a program does, through autograd: the tables, the harmonics and the forward
kernels follow one another, and torch's own kernels, which let nobody start early, run before every backward kernel.  In
``test_edge_kernels_behind_one_another`` forward and backward kernels follow one another directly, to second order."""

import ctypes

import pytest
import torch

import lunaequivariance_b200 as luna
from lunaequivariance_b200 import _native
from lunaequivariance_b200 import conv as conv_mod
from tests.helpers import all_paths, random_graph

pytestmark = pytest.mark.gpu


def _chain(graph_of, module, harmonics, vectors, x, w, steps, sync):
    """Features become outputs and outputs features, in buffers that the allocator hands on from step to step."""
    results = []
    for step in range(steps):
        graph = graph_of()
        vec = vectors.detach().requires_grad_(True)
        weights = w.detach().requires_grad_(True)
        features = x.detach().requires_grad_(True)
        y = harmonics(vec)
        sync()
        out = module(features, y, weights, graph=graph)
        sync()
        grads = torch.autograd.grad(out, (features, vec, weights), torch.ones_like(out) * (1.0 / (step + 1)))
        sync()
        x = out.detach() / out.detach().abs().max()
        w = w + 1e-3 * grads[2] / (1 + grads[2].abs().max())
        vectors = vectors + 1e-3 * grads[1] / (1 + grads[1].abs().max())
        results.append((out.detach().clone(), *(g.clone() for g in grads)))
    return results


# few rows (shared by teams), equal parts and tiles; one edge and two at a time
@pytest.mark.parametrize("nodes,degree,mul", [(40, 30, 64), (700, 12, 64), (700, 12, 32), (9_000, 60, 32)])
@pytest.mark.parametrize("side_stream", [False, True])
def test_chains_without_synchronisation(nodes, degree, mul, side_stream):
    irreps = f"{mul}x0e+{mul}x1o+{mul}x2e"
    attributes = "1x0e+1x1o+1x2e"
    instructions = [(i, j, k, "uvu", True) for i in range(3) for j in range(3) for k in range(3)
                    if (i + j + k) % 2 == 0 and abs(i - j) <= k <= i + j]
    module = luna.TensorProductConv(irreps, attributes, irreps, instructions, internal_weights=False, shared_weights=False,
                                    dtype=torch.float32)
    harmonics = luna.o3.SphericalHarmonics(luna.Irreps(attributes), normalize=True, normalization="component",
                                           dtype=torch.float32)
    generator = torch.Generator(device="cuda").manual_seed(nodes)
    src = torch.randint(nodes, (nodes * degree,), generator=generator, device="cuda")
    dst = torch.arange(nodes, device="cuda").repeat_interleave(degree)
    vectors = torch.randn(src.numel(), 3, generator=generator, device="cuda")
    x = torch.randn(nodes, module.op.in1_dim, generator=generator, device="cuda")
    w = torch.randn(src.numel(), module.op.weight_numel, generator=generator, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        graph = module.create_graph(src, dst, nodes)
        args = (module, harmonics, vectors, x, w, 6)
        want = _chain(lambda: graph, *args, torch.cuda.synchronize)
        got = _chain(lambda: graph, *args, lambda: None)
        fresh = _chain(lambda: module.create_graph(src, dst, nodes), *args, lambda: None)  # tables straight before
    torch.cuda.synchronize()
    module.op.check_status()
    for step, (a, b, c) in enumerate(zip(want, got, fresh)):
        for p, q, r in zip(a, b, c):
            assert torch.equal(p, q) and torch.equal(p, r), step


def _back_to_back(op, graph, start, steps, sync):
    """Launches of the edge kernels straight behind one another, in buffers made before: every one reads what the one before it
    wrote, or overwrites or adds to what that read or wrote.  Between steps the values are brought back to the size of one."""
    x, y, w = (t.clone() for t in start)
    gx, gy, gw, part_y, part_w = (torch.empty_like(t) for t in (x, y, w, y, w))
    out = torch.empty(graph.num_nodes, op.out_dim, dtype=x.dtype, device=x.device)
    stream = _native.current_stream(x.device)
    results = []

    def launch(call, *args, **options):
        value = call(op, *args, graph, **options)
        sync()
        return value

    for _ in range(steps):
        launch(conv_mod.run_forward, x, y, w, out=out)
        launch(conv_mod.run_backward, x, y, w, out, out=(gx, gy, gw))
        launch(conv_mod.run_backward, x, gy, gw, out, out=(gx, part_y, part_w), add_gx=True)
        results += [out.clone(), gx.clone(), part_y.clone(), part_w.clone()]
        for t in (out, gx, gy, gw):
            t.div_(t.abs().max())
        launch(conv_mod.run_backward, x, gy, gw, out, needs=(True, False, True), out=(gx, None, part_w))
        launch(conv_mod.run_backward, gx, gy, w, out, needs=(False, True, False), out=(None, y, None))
        launch(conv_mod.run_backward, gx, y, w, out, needs=(False, False, True), out=(None, None, gw))
        # added to in place: read by bulk copies where the launch before wrote by bulk stores
        _native.check(_native.library().luna_uvu_conv_bwd_add_gw(
            op._plan.handle, ctypes.byref(graph.native()), x.data_ptr(), y.data_ptr(), w.data_ptr(), out.data_ptr(), None, None,
            gw.data_ptr(), None, 0, stream))
        sync()
        launch(conv_mod.run_forward, x, y, gw, out=out)  # overwrites the cotangent of the three before
        results += [gx.clone(), y.clone(), gw.clone(), out.clone()]
        for t in (out, gx, y, gw):
            t.div_(t.abs().max())
        # the second order, whose launches add to one another's outputs, on operands of which the last one has just been written
        launch(conv_mod.run_forward, x, y, gw, out=out)
        results += launch(conv_mod.run_double_backward, x, y, w, out, gx, gy, gw)
        _, _, h_w, h_g = launch(conv_mod.run_double_backward, x, y, w, out, None, gy, None, needs=(False, False, True, True))
        results += [h_w, h_g]
        launch(conv_mod.run_backward, x, gy, h_w, h_g, out=(gx, part_y, w))
        results += [gx.clone(), part_y.clone(), w.clone()]
        x, y, w = gx / gx.abs().max(), part_y / part_y.abs().max(), w / w.abs().max()
    return results


# one edge at a time, two (16 and 48 channels), two and three warps per edge, slices; rows shared by teams, equal parts, tiles
@pytest.mark.parametrize("degree,mul,dtype", [
    (2, 64, torch.float32), (2, 16, torch.float32), (1, 48, torch.float32), (1, 160, torch.float32), (1, 352, torch.float32),
    (2, 64, torch.float64), (1, 16, torch.float64), (1, 160, torch.float64)])
@pytest.mark.parametrize("nodes,edges", [(40, 1_200), (700, 8_400), (1_500, 3_000)])
def test_edge_kernels_behind_one_another(degree, mul, dtype, nodes, edges):
    features = "+".join(f"{mul}x{l}{'eo'[l % 2]}" for l in range(degree + 1))
    attributes = "+".join(f"1x{l}{'eo'[l % 2]}" for l in range(degree + 1))
    module = luna.TensorProductConv(features, attributes, features, all_paths(features, attributes, features),
                                    internal_weights=False, shared_weights=False, dtype=dtype)
    op = module.op
    assert op.backward_variant == "row"  # the edge kernels serve the plan
    generator = torch.Generator().manual_seed(nodes + mul)
    src, dst = random_graph(nodes, edges, generator)
    graph = module.create_graph(src.cuda(), dst.cuda(), nodes)
    start = [torch.randn(*shape, generator=generator, dtype=torch.float64).to(dtype).cuda()
             for shape in ((nodes, op.in1_dim), (edges, op.in2_dim), (edges, op.weight_numel))]
    want = _back_to_back(op, graph, start, 2, torch.cuda.synchronize)
    got = _back_to_back(op, graph, start, 2, lambda: None)
    torch.cuda.synchronize()
    op.check_status()
    for at, (a, b) in enumerate(zip(want, got)):
        assert torch.isfinite(a).all() and a.abs().max() > 0 and torch.equal(a, b), at


class _EdgeData(ctypes.Structure):
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


def _early_starts(call):
    """How many of two launches behind one another, captured in a graph, start before the launch ahead of them has ended."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
        call()
    sources, targets, data, edges = (ctypes.c_void_p * 8)(), (ctypes.c_void_p * 8)(), (_EdgeData * 8)(), ctypes.c_size_t(8)
    error = ctypes.CDLL("libcudart.so.12").cudaGraphGetEdges_v2(ctypes.c_void_p(graph.raw_cuda_graph()), sources, targets, data,
                                                                ctypes.byref(edges))
    assert error == 0 and edges.value == 1  # two nodes
    return sum(data[edge].type == 1 for edge in range(edges.value))  # cudaGraphDependencyTypeProgrammatic


# 128 MB of weights and a little more
@pytest.mark.parametrize("edges,early", [(47_662, 1), (47_663, 0)])
def test_large_weight_gradients_start_in_order(edges, early):
    irreps, attributes = "64x0e+64x1o+64x2e", "1x0e+1x1o+1x2e"
    module = luna.TensorProductConv(irreps, attributes, irreps, all_paths(irreps, attributes, irreps), internal_weights=False,
                                    shared_weights=False, dtype=torch.float32)
    op, nodes = module.op, 2_000
    src, dst = random_graph(nodes, edges, torch.Generator().manual_seed(5))
    graph = module.create_graph(src.cuda(), dst.cuda(), nodes)
    x, y, w, g = (torch.zeros(*shape, device="cuda")
                  for shape in ((nodes, op.in1_dim), (edges, op.in2_dim), (edges, op.weight_numel), (nodes, op.out_dim)))
    out, gw = torch.empty_like(g), torch.empty_like(w)
    assert _early_starts(lambda: conv_mod.run_forward(op, x, y, w, graph, out=out)) == 1
    assert _early_starts(lambda: conv_mod.run_backward(op, x, y, w, g, graph, (False, False, True), out=(None, None, gw))) == early
