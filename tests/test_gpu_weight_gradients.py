"""The weights' gradient where two orders of differentiation meet in it (force training), for weights large enough that the
backward kernel adds to the second order's result in place: values, and who else may hold or ask for them."""

import pytest
import torch

import lunaequivariance_b200 as luna
from oracle import uvu_conv as oracle_conv
from tests.helpers import all_paths, assert_close, random_graph

pytestmark = pytest.mark.gpu
MUL, NODES = 128, 600
CASES = {  # irreps, dtype, edges: weights of 32 MiB and a little more
    "vector": ((f"{MUL}x1o", "1x1o", f"{MUL}x0e"), torch.float64, 32_771),
    "scalars": ((f"{MUL}x0e", "1x0e+1x1o", f"{MUL}x0e+{MUL}x1o"), torch.float32, 32_769),
}


def energy_of(out, linear, scale):
    return (out * scale).sum() if linear else out.square().sum()


def steps(conv, x, y, w, scale, wanted, linear=False):
    out = conv(x, y, w)
    (gy,) = torch.autograd.grad(energy_of(out, linear, scale), y, create_graph=True)
    return torch.autograd.grad(gy.square().sum(), wanted)


class Problem:
    def __init__(self, name, seed=3):
        irreps, dtype, edges = CASES[name]
        instructions = all_paths(*irreps)
        self.module = luna.TensorProductConv(*irreps, instructions, internal_weights=False, shared_weights=False, dtype=dtype)
        self.meta = oracle_conv.build_specs(*irreps, instructions)
        generator = torch.Generator().manual_seed(seed)
        self.src, self.dst = random_graph(NODES, edges, generator)
        rand = lambda *shape: torch.randn(*shape, generator=generator, dtype=dtype)
        self.cpu = [rand(NODES, self.meta["in1_dim"]), rand(edges, self.meta["in2_dim"]), rand(edges, self.meta["weight_numel"])]
        self.scale = rand(NODES, self.meta["out_dim"])
        self.dtype = dtype
        self.graph = self.module.create_graph(self.src.cuda(), self.dst.cuda(), NODES)
        self.conv = lambda x, y, w: self.module(x, y, w, graph=self.graph)
        assert self.cpu[2].nbytes >= 32 << 20

    def device(self):
        return [t.cuda().requires_grad_(True) for t in self.cpu] + [self.scale.cuda()]

    def reference(self, wanted, linear=False):
        x, y, w = (t.double().requires_grad_(True) for t in self.cpu)
        conv = lambda x, y, w: oracle_conv.conv_forward(self.meta, x, y, w, self.src, self.dst, NODES)
        return steps(conv, x, y, w, self.scale.double(), [(x, y, w)[i] for i in wanted], linear)


@pytest.mark.parametrize("linear", [False, True])
@pytest.mark.parametrize("name", CASES)
def test_both_orders(name, linear):
    p = Problem(name)
    want = p.reference((0, 2), linear)
    x, y, w, scale = p.device()
    for got, ref in zip(steps(p.conv, x, y, w, scale, (x, w), linear), want):
        assert_close(got, ref, p.dtype, f"{name} linear={linear}")
    (gw,) = steps(p.conv, x, y, w, scale, (w,), linear)
    assert_close(gw, want[1], p.dtype, f"{name} linear={linear} weights alone")
    p.module.op.check_status()


def test_saved_tensor_hooks_and_a_second_graph_through_the_gradient():
    p = Problem("scalars")
    (want,) = p.reference((2,))
    x, y, w, scale = p.device()
    with torch.autograd.graph.save_on_cpu():
        (gw,) = steps(p.conv, x, y, w, scale, (w,))
    assert_close(gw, want, p.dtype, "saved on the CPU")
    out = p.conv(x, y, w)
    (gy,) = torch.autograd.grad(out.square().sum(), y, create_graph=True)
    (gw,) = torch.autograd.grad(gy.square().sum(), w, create_graph=True)
    assert gw.requires_grad
    assert_close(gw, want, p.dtype, "with a graph")


def test_a_gradient_somebody_holds_is_not_added_to():
    p = Problem("vector")
    x, y, w, scale = p.device()
    (second,) = steps(p.conv, x, y, w, scale, (w,), linear=True)  # the second order alone
    out = p.conv(x, y, w)
    held = []
    out.grad_fn.register_prehook(lambda grads: held.append(grads))
    energy = (out * scale).sum()
    (gy,) = torch.autograd.grad(energy, y, create_graph=True)
    held.clear()
    (gw,) = torch.autograd.grad(gy.square().sum() + energy, w)
    assert len(held) == 1 and torch.equal(held[0][1], second)
    x2, y2, w2 = (t.double().requires_grad_(True) for t in p.cpu)
    first = oracle_conv.conv_forward(p.meta, x2, y2, w2, p.src, p.dst, NODES)
    (first,) = torch.autograd.grad((first * p.scale.double()).sum(), w2)
    assert_close(gw, second.cpu().double() + first, p.dtype, "held")


def test_weights_nobody_asks_for_cost_nothing():
    p = Problem("scalars")
    (want,) = p.reference((0,))
    x, y, w, scale = p.device()
    out = p.conv(x, y, w)
    (gy,) = torch.autograd.grad(out.square().sum(), y, create_graph=True)
    loss = gy.square().sum()
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    (gx,) = torch.autograd.grad(loss, x)
    assert torch.cuda.max_memory_allocated() - before < w.nbytes // 2
    assert_close(gx, want, p.dtype, "features alone")


def test_weights_changed_after_the_call_are_noticed():
    p = Problem("vector")
    x, y, w, scale = p.device()
    out = p.conv(x, y, w)
    with torch.no_grad():
        w.add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out.square().sum(), x)
