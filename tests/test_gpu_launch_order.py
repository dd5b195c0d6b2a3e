"""Kernels that are launched before the one ahead of them has ended: chains in which every launch reads what the one before it
wrote, and overwrites what it read, give the same bits as with a synchronisation after every step."""

import pytest
import torch

import lunaequivariance_b200 as luna

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
