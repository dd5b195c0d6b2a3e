"""The weights' gradient where two orders of differentiation meet in it (force training), for weights large enough that the
backward kernel adds to the second order's result in place: values, who else may hold or ask for them, and that hooks and
passes of their own find the same autograd graph as with smaller weights."""

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
BOTH_SIDES = pytest.mark.parametrize("edges", [1_500, None], ids=["small", "large"])  # of the 32 MiB


def energy_of(out, linear, scale):
    return (out * scale).sum() if linear else out.square().sum()


def steps(conv, x, y, w, scale, wanted, linear=False):
    out = conv(x, y, w)
    (gy,) = torch.autograd.grad(energy_of(out, linear, scale), y, create_graph=True)
    return torch.autograd.grad(gy.square().sum(), wanted)


class Problem:
    def __init__(self, name, seed=3, edges=None):
        irreps, dtype, all_edges = CASES[name]
        edges, large = edges or all_edges, edges is None
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
        assert (self.cpu[2].nbytes >= 32 << 20) == large

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
    out = p.conv(x, y, w)
    held = []
    energy = out.square().sum()
    (gy,) = torch.autograd.grad(energy, y, create_graph=True)
    gy.grad_fn.next_functions[2][0].register_prehook(lambda grads: held.append(grads[0]))
    (gw,) = torch.autograd.grad(gy.square().sum(), w)
    assert len(held) == 1
    seen = held[0].clone()
    (alone,) = torch.autograd.grad(torch.autograd.grad(p.conv(x, y, w), y, 2 * out.detach(), create_graph=True)[0].square().sum(), w)
    assert_close(seen, alone.cpu().double(), p.dtype, "the second order's, without the first order's")
    assert_close(gw, p.reference((2,))[0], p.dtype, "held")


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


def first_order(p, factor=1.0):
    """The weights' gradient of the linear energy."""
    x, y, w = (t.double().requires_grad_(True) for t in p.cpu)
    out = oracle_conv.conv_forward(p.meta, x, y, w, p.src, p.dst, NODES)
    return torch.autograd.grad((out * p.scale.double()).sum() * factor, w)[0]


@BOTH_SIDES
def test_hooks_of_the_output_and_its_node_see_the_output_alone(edges):
    p = Problem("vector", edges=edges)
    x, y, w, scale = p.device()
    (second,) = p.reference((2,), linear=True)
    out = p.conv(x, y, w)
    out.register_hook(lambda grad: grad * 2.0)  # a gradient that is not there is no tensor
    (gy,) = torch.autograd.grad((out * scale).sum(), y, create_graph=True)
    (gw,) = torch.autograd.grad(gy.square().sum(), w)  # nothing of it reaches the output
    assert_close(gw, 4.0 * second, p.dtype, "hook of the output")
    out = p.conv(x, y, w)
    counts = []

    def twice(grads):
        counts.append(len(grads))
        return (grads[0] * 2.0,)

    out.grad_fn.register_prehook(twice)
    (gw,) = torch.autograd.grad((out * scale).sum(), w)
    assert counts == [1]
    assert_close(gw, first_order(p, 2.0), p.dtype, "prehook of the node")


@BOTH_SIDES
def test_what_the_first_order_returns_is_its_own_part(edges):
    p = Problem("vector", edges=edges)
    x, y, w, scale = p.device()
    seen = []
    out = p.conv(x, y, w)
    out.grad_fn.register_hook(lambda grad_inputs, grad_outputs: seen.append((len(grad_outputs), grad_inputs[2])))
    energy = out.square().sum()
    (gy,) = torch.autograd.grad(energy, y, create_graph=True)
    seen.clear()
    (gw,) = torch.autograd.grad(gy.square().sum(), w)
    assert len(seen) == 1 and seen[0][0] == 1
    (want,) = p.reference((2,))
    assert_close(gw, want, p.dtype, "both orders")
    assert float((seen[0][1].cpu().double() - want).norm()) > 0.1 * float(want.norm())


@BOTH_SIDES
def test_the_two_orders_in_passes_of_their_own(edges):
    """The force loss first, which reaches the weights but not the output, then the energy through the same graph."""
    p = Problem("vector", edges=edges)
    x, y, w, scale = p.device()
    (second,) = p.reference((2,), linear=True)
    energy = (p.conv(x, y, w) * scale).sum()
    (gy,) = torch.autograd.grad(energy, y, create_graph=True)
    gy.square().sum().backward(inputs=[w])
    assert_close(w.grad, second, p.dtype, "second order")
    energy.backward(inputs=[w])
    assert_close(w.grad, second + first_order(p), p.dtype, "both")


@BOTH_SIDES
def test_one_loss_of_an_energy_that_is_linear_and_of_its_forces(edges):
    """Nothing orders the two contributions; also twice through one graph, and with a graph of its own in between."""
    p = Problem("vector", edges=edges)
    x, y, w, scale = p.device()
    want = p.reference((2,), linear=True)[0] + first_order(p)
    energy = (p.conv(x, y, w) * scale).sum()
    (gy,) = torch.autograd.grad(energy, y, create_graph=True)
    loss = gy.square().sum() + energy
    for create_graph in (False, True, False):
        (gw,) = torch.autograd.grad(loss, w, retain_graph=True, create_graph=create_graph)
        assert_close(gw, want, p.dtype, f"create_graph={create_graph}")


@pytest.mark.parametrize("wanted", [(2,), (0, 1, 2)], ids=["weights", "all"])
@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("linear,energy_too", [(False, False), (False, True), (True, True)])
def test_the_sum_is_made_in_place(name, linear, energy_too, wanted):
    """Whichever order comes first, a second tensor of the weights' size is never there."""
    p = Problem(name)

    def step(conv, x, y, w, scale):
        energy = energy_of(conv(x, y, w), linear, scale)
        (gy,) = torch.autograd.grad(energy, y, create_graph=True)
        return gy.square().sum() + (energy if energy_too else 0.0)

    tensors = p.device()
    loss = step(p.conv, *tensors)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = torch.autograd.grad(loss, [tensors[i] for i in wanted])
    assert torch.cuda.max_memory_allocated() - before < 1.5 * tensors[2].nbytes
    cpu = [t.double().requires_grad_(True) for t in p.cpu]
    conv = lambda x, y, w: oracle_conv.conv_forward(p.meta, x, y, w, p.src, p.dst, NODES)
    want = torch.autograd.grad(step(conv, *cpu, p.scale.double()), [cpu[i] for i in wanted])
    for value, ref, i in zip(got, want, wanted):
        assert_close(value, ref, p.dtype, f"{name} {linear} {energy_too} {i}")


@pytest.mark.parametrize("energy_first", [True, False])
def test_two_force_losses_through_one_graph(energy_first):
    """Two second orders, of which one at most meets the first order; alone, and in one loss."""
    p = Problem("vector")
    cpu = [t.double().requires_grad_(True) for t in p.cpu]
    reference = lambda x, y, w: oracle_conv.conv_forward(p.meta, x, y, w, p.src, p.dst, NODES)

    def losses(conv, x, y, w, scale):
        energy = (conv(x, y, w) * scale).sum()
        (gy,) = torch.autograd.grad(energy, y, create_graph=True)
        (gx,) = torch.autograd.grad(energy, x, create_graph=True)
        a, b = gy.square().sum(), gx.square().sum()
        return (energy + a, energy + b, energy + a + b) if energy_first else (a + energy, b + energy, a + b + energy)

    tensors = p.device()
    for got, want in zip(losses(p.conv, *tensors), losses(reference, *cpu, p.scale.double())):
        (value,) = torch.autograd.grad(got, tensors[2], retain_graph=True)
        assert_close(value, torch.autograd.grad(want, cpu[2], retain_graph=True)[0], p.dtype, "two losses")


def test_passes_after_one_that_failed():
    """The second order's gradient has been set aside when a pass ends with an error; the next ones have their own."""
    p = Problem("vector")
    x, y, w, scale = p.device()
    out = p.conv(x, y, w)
    fail = [True]

    def stop(grad):
        if fail[0]:
            raise ValueError("stop")

    z = out * 1.0
    z.register_hook(stop)
    fail[0] = False
    (gy,) = torch.autograd.grad(z.square().sum(), y, create_graph=True)
    fail[0] = True
    loss = gy.square().sum()
    with pytest.raises(ValueError, match="stop"):
        torch.autograd.grad(loss, w, retain_graph=True)
    fail[0] = False
    for _ in range(2):
        (gw,) = torch.autograd.grad(loss, w, retain_graph=True)
        assert_close(gw, p.reference((2,))[0], p.dtype, "after a failed pass")
