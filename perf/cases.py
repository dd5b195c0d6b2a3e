"""The work users of this package have it do, as cases that can be timed and compared.

A case is one call pattern of a program that uses the package: a convolution layer in inference, in training and in a
force step, first and second order, the spherical harmonics on their own, and the preparation of a new topology.
``prepare`` makes what the program holds before the call, ``run`` is one pass through the public entry points.

A convolution case names its layer by three degrees: features ``0..in_l``, edge harmonics ``0..sh_l``, outputs
``0..out_l``, ``mul`` channels of every degree, every parity-allowed ``uvu`` path.  ``in_l = 0`` is the first layer of a
network (scalars in), ``out_l = 0`` the last one (scalars out).  Edges are destination-sorted.
"""

from __future__ import annotations

import math
from functools import lru_cache

import torch

import lunaequivariance_b200 as luna

DENSITY = 0.1  # atoms per cubic Angstrom
DTYPES = {"float32": torch.float32, "float64": torch.float64}


def listed():
    return [
        # The smallest convolution the package is tested with, one step of it in double precision: launches and host
        # time are what it costs.
        _conv("vector_1k_f64", "backward", 1, 1, 0, 32, 1_000, 16.0, graph="random", dtype="float64", only_l1=True),
        # One molecule in inference: every atom neighbours every other, 552 edges.
        _conv("molecule_24", "forward", 2, 2, 2, 64, 24, 23.0, graph="complete"),
        # A molecular-dynamics step of a protein-sized system (2,083 atoms, 85,876 edges): harmonics of the edge
        # vectors, convolution, and the gradients that forces need.
        _conv("dynamics_2k", "forces", 2, 2, 2, 64, 2_083, 85_876 / 2_083),
        # First layer of a network, scalars in, in training.
        _conv("first_layer_20k", "backward", 0, 3, 3, 128, 20_000, 52.3),
        # Inference of a layer whose channel count is no multiple of 32.
        _conv("inference_48ch_10k", "forward", 2, 2, 2, 48, 10_001, 52.3),
        # Training step of the 128-channel interaction layer: 50,000 atoms with 52 neighbours (2.6 M edges).
        _conv("interaction_50k", "backward", 2, 3, 3, 128, 50_000, 52.3),
        # All degrees to 3, and sources without any locality: 40 random incoming edges per node.
        _conv("random_40k", "backward", 3, 3, 3, 64, 40_000, 40.0, graph="random"),
        # Training step of a 64-channel layer on one GPU's share of a large system (5.2 M edges).
        _conv("share_100k", "backward", 2, 2, 2, 64, 100_000, 52.3),
        # Force training in double precision: energy, forces, loss, gradient of the weights through both orders.
        _conv("force_training_f64_20k", "force_training", 2, 3, 3, 128, 20_000, 52.3, dtype="float64"),
        # Force training of an interior layer in single precision on a batch of small structures: the features need
        # their gradient too.
        _conv("force_training_4k", "force_training", 2, 2, 2, 32, 4_003, 52.3, features=True),
        # Spherical harmonics to degree 6 of 4 M vectors, values and gradient.
        {"name": "harmonics_4m", "kind": "harmonics", "items": 4_000_000, "lmax": 6, "dtype": "float32"},
        # A new neighbour list: the tables every layer of the network then shares.
        {"name": "topology_20k", "kind": "topology", "nodes": 20_000, "degree": 52.3, "graph": "radius"},
    ]


def _conv(name, kind, in_l, sh_l, out_l, mul, nodes, degree, *, graph="radius", dtype="float32", features=False,
          only_l1=False):
    case = {"kind": kind, "in_l": in_l, "sh_l": sh_l, "out_l": out_l, "mul": mul, "nodes": nodes, "degree": degree,
            "graph": graph, "dtype": dtype, "features": features, "only_l1": only_l1}
    return dict(case, name=name) if name else case


# First, interior and last layers of networks with edge harmonics to degree 1, 2 or 3.
LAYERS = ((0, 1, 1), (0, 2, 2), (0, 3, 3), (1, 1, 1), (2, 2, 2), (3, 3, 3), (2, 3, 3), (1, 1, 0), (2, 2, 0), (3, 3, 0))


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("forward", "forward", "backward", "backward", "backward", "forces", "forces", "force_training",
                       "force_training", "harmonics", "topology"))
    if kind == "harmonics":
        dtype = rng.choice(("float32", "float32", "float64"))
        return {"kind": kind, "items": _log_uniform(rng, 500, 4_000_000 if dtype == "float32" else 2_000_000),
                "lmax": rng.randint(1, 6), "dtype": dtype}
    graph = rng.choice(("radius", "radius", "radius", "random"))
    degree = round(rng.uniform(12.0, 52.0), 1) if graph == "radius" else float(rng.randint(4, 48))
    if kind == "topology":
        return {"kind": kind, "nodes": _log_uniform(rng, 200, 50_000), "degree": degree, "graph": graph}
    in_l, sh_l, out_l = rng.choice(LAYERS)
    mul = rng.choice((16, 32, 48, 64, 64, 96, 128, 128))
    dtype = rng.choice(("float32", "float32", "float32", "float64"))
    case = _conv(None, kind, in_l, sh_l, out_l, mul, 0, degree, graph=graph, dtype=dtype,
                 features=bool(in_l) and rng.random() < 0.5)
    # as many nodes as keep the per-edge weights, the bulk of the bytes, within what the large listed cases hold
    bytes_per_node = degree * mul * _path_count(in_l, sh_l, out_l) * (8 if dtype == "float64" else 4)
    most = {"forward": 8e9, "backward": 6e9, "forces": 6e9, "force_training": 3e9}[kind]
    case["nodes"] = _log_uniform(rng, 160, max(320, min(100_000, int(most / bytes_per_node))))
    return case


def _path_count(in_l, sh_l, out_l):
    return sum((a + b + c) % 2 == 0 and abs(a - b) <= c <= a + b
               for a in range(in_l + 1) for b in range(sh_l + 1) for c in range(out_l + 1))


# ------------------------------------------------------------------------------------------------ layers and graphs


def _irreps(mul, degrees):
    return "+".join(f"{mul}x{l}{'o' if l % 2 else 'e'}" for l in degrees)


@lru_cache(maxsize=None)
def _layer(in_l, sh_l, out_l, mul, dtype, only_l1):
    """The module and its harmonics: a program makes them once and calls them with every new structure."""
    lowest = 1 if only_l1 else 0
    in1, in2 = _irreps(mul, range(lowest, in_l + 1)), _irreps(1, range(lowest, sh_l + 1))
    out = _irreps(mul, range(out_l + 1))
    a, b, c = (list(luna.Irreps(text)) for text in (in1, in2, out))
    instructions = [(i, j, k, "uvu", True) for i, (_, p) in enumerate(a) for j, (_, q) in enumerate(b)
                    for k, (_, r) in enumerate(c) if r in p * q]
    conv = luna.TensorProductConv(in1, in2, out, instructions, internal_weights=False, shared_weights=False,
                                  dtype=DTYPES[dtype])
    harmonics = luna.o3.SphericalHarmonics(luna.Irreps(in2), normalize=True, normalization="component",
                                           dtype=DTYPES[dtype])
    return conv, harmonics


def _layer_of(case):
    return _layer(case["in_l"], case["sh_l"], case["out_l"], case["mul"], case["dtype"], case["only_l1"])


def _edge_count(case):
    return int(round(case["nodes"] * case["degree"]))


def _edges(case, generator):
    """``src``, ``dst`` (int64, sorted by ``dst``) and edge vectors (float64) of the case's topology.

    The structure belongs to the case; the generator moves it through its periodic box, or relabels its nodes.  Node
    numbers and edge order then change, and the sizes of the tables made from them do not.
    """
    nodes, device = case["nodes"], generator.device
    if case["graph"] == "radius":
        return _radius_edges(nodes, _edge_count(case), generator)
    if case["graph"] == "complete":
        pairs = ~torch.eye(nodes, dtype=torch.bool, device=device)
        dst, src = pairs.nonzero(as_tuple=True)
        position = torch.rand(nodes, 3, generator=generator, device=device, dtype=torch.float64) * 6.0
        return src, dst, position[src] - position[dst]
    degree = int(case["degree"])
    fixed = torch.Generator(device=device).manual_seed(nodes)
    dst = torch.arange(nodes, device=device).repeat_interleave(degree)
    src = torch.randint(nodes - 1, (dst.numel(),), generator=fixed, device=device)
    src = src + (src >= dst).long()
    label = torch.randperm(nodes, generator=generator, device=device)
    src = label[src].view(nodes, degree)[torch.argsort(label)].flatten()
    return src, dst, torch.randn(dst.numel(), 3, generator=generator, device=device, dtype=torch.float64)


def _radius_edges(nodes, edges, generator, chunk=8192):
    """The ``edges`` shortest directed pairs of a periodic cube of uniformly placed atoms, atoms numbered cell by cell:
    a neighbour list whose cutoff is the one that gives this many edges."""
    device = generator.device
    box = (nodes / DENSITY) ** (1.0 / 3.0)
    margin = 1.02 + 9.0 / math.sqrt(edges)  # pairs within a radius scatter by about sqrt(2 / edges)
    cutoff = (margin * edges / nodes / DENSITY / (4.0 / 3.0 * math.pi)) ** (1.0 / 3.0)
    cells = max(1, int(box / cutoff))
    fixed = torch.Generator(device=device).manual_seed(nodes)
    position = torch.rand(nodes, 3, generator=fixed, device=device, dtype=torch.float64) * box
    position = (position + torch.rand(3, generator=generator, device=device, dtype=torch.float64) * box) % box
    side = box / cells
    index = (position / side).long().clamp_(max=cells - 1)
    order = torch.argsort((index[:, 0] * cells + index[:, 1]) * cells + index[:, 2], stable=True)
    position, index = position[order], index[order]
    cell = (index[:, 0] * cells + index[:, 1]) * cells + index[:, 2]
    count = torch.bincount(cell, minlength=cells ** 3)
    first = count.cumsum(0) - count
    width = int(count.max())
    if cells >= 3:
        near = torch.tensor([(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)], device=device)
    else:  # fewer cells than the stencil is wide: look at each of them once
        near = torch.tensor([(a, b, c) for a in range(cells) for b in range(cells) for c in range(cells)],
                            device=device)
    slot = torch.arange(width, device=device)
    parts = []
    for begin in range(0, nodes, chunk):
        end = min(nodes, begin + chunk)
        neighbour = (index[begin:end, None, :] + near) % cells if cells >= 3 else near.expand(end - begin, -1, 3)
        neighbour = (neighbour[..., 0] * cells + neighbour[..., 1]) * cells + neighbour[..., 2]
        candidate = first[neighbour][..., None] + slot
        valid = slot < count[neighbour][..., None]
        candidate = torch.where(valid, candidate, 0)
        vector = position[candidate] - position[begin:end, None, None, :]
        vector -= box * torch.round(vector / box)
        length = vector.square().sum(-1)
        valid &= (length < cutoff * cutoff) & (candidate != torch.arange(begin, end, device=device)[:, None, None])
        d, o, k = valid.nonzero(as_tuple=True)
        parts.append((candidate[d, o, k], d + begin, vector[d, o, k], length[d, o, k]))
    src, dst, vector, length = (torch.cat(p) for p in zip(*parts))
    if src.numel() < edges:
        raise RuntimeError(f"{src.numel()} pairs within the cutoff, {edges} wanted")
    keep = torch.sort(torch.topk(length, edges, largest=False).indices).values
    return src[keep], dst[keep], vector[keep]


# ------------------------------------------------------------------------------------------------ the three functions


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    generator = torch.Generator(device=device).manual_seed(int(seed))
    state = {"kind": case["kind"]}
    if case["kind"] == "topology":
        state["nodes"] = case["nodes"]
        state["src"], state["dst"], _ = _edges(case, generator)
        return state
    dtype = DTYPES[case["dtype"]]

    def normal(*shape):
        return torch.randn(*shape, generator=generator, device=device, dtype=dtype)

    if case["kind"] == "harmonics":
        irreps = _irreps(1, range(case["lmax"] + 1))
        state["harmonics"] = luna.o3.SphericalHarmonics(irreps, normalize=True, normalization="component", dtype=dtype)
        state["vec"] = normal(case["items"], 3).requires_grad_(True)
        state["g"] = normal(case["items"], (case["lmax"] + 1) ** 2)
        return state
    conv, harmonics = _layer_of(case)
    src, dst, vec = _edges(case, generator)
    vec = vec.to(dtype)
    op = conv.op
    state.update(conv=conv, graph=conv.create_graph(src, dst, case["nodes"]), x=normal(case["nodes"], op.in1_dim),
                 w=normal(src.numel(), op.weight_numel), g=normal(case["nodes"], op.out_dim),
                 features=case["features"])
    if case["kind"] in ("forward", "backward"):
        state["y"] = harmonics(vec)
    else:
        state.update(harmonics=harmonics, vec=vec.requires_grad_(True))
    if case["kind"] != "forward":
        state["w"].requires_grad_(True)
        if case["kind"] != "force_training" or case["features"]:
            state["x"].requires_grad_(True)
        if case["kind"] == "backward":
            state["y"].requires_grad_(True)
    return state


def run(state):
    kind = state["kind"]
    if kind == "topology":
        graph = luna.TensorProductConv.create_graph(state["src"], state["dst"], state["nodes"])
        segments = graph.source_segments
        return {"src": graph.src, "dst": graph.dst, "dst_rowptr": graph.dst_rowptr, "src_rowptr": graph.src_rowptr,
                "edge_ids_by_src": graph.edge_ids_by_src, "edge_ids_by_dst": graph.edge_ids_by_dst,
                "node_order": graph.node_order, "source_node_order": graph.source_node_order,
                "node_tiers": graph.node_tiers, "segment_nodes": segments.nodes, "segment_begin": segments.begin,
                "segment_end": segments.end, "segment_rowptr": segments.rowptr, "segment_order": segments.order}
    if kind == "harmonics":
        values = state["harmonics"](state["vec"])
        (grad,) = torch.autograd.grad(values, state["vec"], state["g"])
        return values.detach(), grad
    conv, graph, x, w = state["conv"], state["graph"], state["x"], state["w"]
    if kind == "forward":
        with torch.no_grad():
            return conv(x, state["y"], w, graph=graph)
    if kind == "backward":
        y = state["y"]
        out = conv(x, y, w, graph=graph)
        return out.detach(), *torch.autograd.grad(out, (x, y, w), state["g"])
    vec = state["vec"]
    out = conv(x, state["harmonics"](vec), w, graph=graph)
    if kind == "forces":
        return out.detach(), *torch.autograd.grad(out, (x, vec, w), state["g"])
    energy = out.square().sum()
    (forces,) = torch.autograd.grad(energy, vec, create_graph=True)
    loss = forces.square().sum()
    return forces.detach(), *torch.autograd.grad(loss, (x, w) if state["features"] else (w,))


# ------------------------------------------------------------------------------------------------ what a pass needs


def work(case):
    """Every input of the pass read once, every output written once; multiplications and additions of the non-zero
    coupling terms for each contraction of the pass."""
    if case["kind"] == "topology":
        edges, nodes = _edge_count(case), case["nodes"]
        segments = edges // 32 + nodes
        return {"bytes": 16 * edges + 16 * edges + 4 * (4 * nodes + 2) + 20 * segments, "flops": 0}
    size = 8 if case["dtype"] == "float64" else 4
    if case["kind"] == "harmonics":
        columns = (case["lmax"] + 1) ** 2
        return {"bytes": case["items"] * (3 + columns + columns + 3) * size, "flops": case["items"] * 15 * columns}
    conv, _ = _layer_of(case)
    op, edges, nodes = conv.op, _edge_count(case), case["nodes"]
    X, Y, O, W = op.in1_dim, op.in2_dim, op.out_dim, op.weight_numel
    contraction = edges * sum(s["channels"] * (2 * len(s["terms"]) + 2 * s["l2"] + 1) for s in op.generated_specs)
    tables = 12 * edges + 4 * (2 * nodes + 2)
    if case["kind"] == "forward":
        return {"bytes": edges * (W + Y) * size + nodes * (X + O) * size + tables, "flops": contraction}
    if case["kind"] == "backward":
        return {"bytes": 2 * edges * (W + Y) * size + 2 * nodes * (X + O) * size + tables, "flops": 4 * contraction}
    if case["kind"] == "forces":
        return {"bytes": 2 * edges * (W + 3) * size + 2 * nodes * (X + O) * size + tables, "flops": 4 * contraction}
    # features, vectors and weights in; forces and the gradients of weights (and features) out
    features = 2 if case["features"] else 1
    return {"bytes": 2 * edges * (W + 3) * size + features * nodes * X * size + tables,
            "flops": (8 if case["features"] else 5) * contraction}


def tolerance(case):
    """What the operators are held to everywhere: 1e-5 in single, 1e-12 in double precision; index tables exactly."""
    if case["kind"] == "topology":
        return "exact"
    return {"rel": 1e-12} if case["dtype"] == "float64" else {"rel": 1e-5}
