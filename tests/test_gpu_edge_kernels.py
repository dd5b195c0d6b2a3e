"""The edge kernels at the sizes where they can go wrong, against the CPU oracle: every compiled shape, channel counts
that leave lanes idle or need several warps per edge, rows shared by several teams and rows handed out in tiles."""

import dataclasses
import json
import re

import pytest
import torch

import lunaequivariance_b200 as luna
from lunaequivariance_b200 import conv as conv_mod
from oracle import uvu_conv as oracle_conv
from tests.helpers import all_paths, assert_close, random_problem
from tests.test_gpu_random_shapes import skewed_graph

pytestmark = pytest.mark.gpu
DEVICE = "cuda"
# degrees of x, of the edge attributes and of the output
SHAPES = [((0,), (0, 1), (0, 1)), ((0,), (0, 1, 2), (0, 1, 2)), ((0,), (0, 1, 2, 3), (0, 1, 2, 3)),
          ((0, 1), (0, 1), (0, 1)), ((0, 1, 2), (0, 1, 2), (0, 1, 2)), ((0, 1, 2, 3), (0, 1, 2, 3), (0, 1, 2, 3)),
          ((0, 1, 2), (0, 1, 2, 3), (0, 1, 2, 3)), ((0, 1), (0, 1), (0,)), ((0, 1, 2), (0, 1, 2), (0,)),
          ((0, 1, 2, 3), (0, 1, 2, 3), (0,)), ((1,), (1,), (0,))]


def irreps(mul, degrees):
    return "+".join(f"{mul}x{l}{'o' if l % 2 else 'e'}" for l in degrees)


def check(shape, mul, dtype, nodes, edges, skew, seed):
    in1, in2, out = irreps(mul, shape[0]), irreps(1, shape[1]), irreps(mul, shape[2])
    instructions = all_paths(in1, in2, out)
    module = luna.TensorProductConv(in1, in2, out, instructions, internal_weights=False, shared_weights=False,
                                    dtype=dtype)
    assert module.op.backward_variant == "row"  # the edge kernels serve the plan
    meta = oracle_conv.build_specs(in1, in2, out, instructions)
    generator = torch.Generator().manual_seed(seed)
    src, dst = skewed_graph(nodes, edges, generator, skew)
    p = random_problem((meta["in1_dim"], meta["in2_dim"], meta["out_dim"], meta["weight_numel"]), nodes, src, dtype,
                       generator)
    ref = oracle_conv.conv_derivatives(meta, *(p[k].double() for k in ("x", "y", "w")), src, dst, nodes,
                                       p["g"].double(), *(p[k].double() for k in ("rx", "ry", "rw")))
    graph = module.create_graph(src.to(DEVICE), dst.to(DEVICE), nodes)
    x, y, w, g = (p[k].to(DEVICE).requires_grad_(True) for k in ("x", "y", "w", "g"))
    result = module(x, y, w, graph=graph)
    gx, gy, gw = torch.autograd.grad(result, (x, y, w), g, create_graph=True)
    hx, hy, hw, hg = torch.autograd.grad((gx, gy, gw), (x, y, w, g), tuple(p[k].to(DEVICE) for k in ("rx", "ry", "rw")))
    module.op.check_status()
    for key, value in dict(out=result, gx=gx, gy=gy, gw=gw, hx=hx, hy=hy, hw=hw, hg=hg).items():
        assert_close(value, ref[key], dtype, f"{shape} x{mul} {dtype} {key}")
    return module


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_every_shape(shape, dtype):
    mul = (32, 48, 64)[shape % 3]
    check(SHAPES[shape], mul, dtype, 29, 400, 0.0, shape)  # long rows: shared by teams
    check(SHAPES[shape], mul, dtype, 150, 190, 1.5, shape + 50)  # short rows: tiles, many rows without edges


# idle lanes (4, 12, 16, 48, 80, 96), all lanes (32, 64, 128), several warps per edge (160 and more; FP64: 96 and more)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("mul", [4, 12, 16, 32, 48, 64, 80, 96, 128, 160, 256, 320])
def test_channel_counts(mul, dtype):
    check(SHAPES[3], mul, dtype, 23, 260, 0.0, mul)
    check(SHAPES[4], mul, dtype, 60, 90, 1.0, mul + 1)


# one, two and four channels per lane (FP64: one and two)
@pytest.mark.parametrize("shape,mul,dtype", [
    (3, 352, torch.float32), (3, 576, torch.float32), (3, 864, torch.float32), (4, 544, torch.float32),
    (4, 1024, torch.float32), (5, 640, torch.float32), (5, 704, torch.float32), (6, 352, torch.float32),
    (6, 768, torch.float32), (3, 288, torch.float64), (4, 512, torch.float64), (5, 288, torch.float64),
    (5, 320, torch.float64), (6, 384, torch.float64), (6, 416, torch.float64)])
def test_wide_blocks_in_slices(shape, mul, dtype):
    check(SHAPES[shape], mul, dtype, 7, 120, 0.0, mul)  # long rows: shared by teams
    module = check(SHAPES[shape], mul, dtype, 40, 60, 1.0, mul + 1)  # short rows: tiles
    assert module.op._plan.query(8) == 1  # the slices' parts of dL/dy
    one_gradient_alone(SHAPES[shape], mul, dtype, 40, 90, 1.0, mul + 2)


@pytest.mark.parametrize("knob,shape,mul,dtype", [
    ("LUNA_B200_MAXW=1", 3, 160, torch.float32), ("LUNA_B200_MAXW=1", 6, 128, torch.float64),
    ("LUNA_B200_MAXW=3", 4, 256, torch.float32), ("LUNA_B200_EPW=1", 4, 64, torch.float32)])
def test_tuning_settings(knob, shape, mul, dtype, monkeypatch):
    """Fewer warps than a team would have, and tiles of other sizes, on the same kernels."""
    monkeypatch.setenv(*knob.split("="))
    check(SHAPES[shape], mul, dtype, 23, 260, 0.0, mul)
    check(SHAPES[shape], mul, dtype, 3000, 26000 if mul == 64 else 3100, 0.0, mul + 1)


@pytest.mark.parametrize("nodes,edges", [(1, 1), (1, 2), (1, 77), (2, 9), (3, 1000), (700, 4000), (1300, 5300)])
def test_row_splits(nodes, edges):
    for mul in (16, 128):
        check(SHAPES[3], mul, torch.float32, nodes, edges, 0.0, nodes + edges)


def one_gradient_alone(shape, mul, dtype, nodes, edges, skew, seed):
    in1, in2, out = irreps(mul, shape[0]), irreps(1, shape[1]), irreps(mul, shape[2])
    instructions = all_paths(in1, in2, out)
    module = luna.TensorProductConv(in1, in2, out, instructions, internal_weights=False, shared_weights=False,
                                    dtype=dtype)
    meta = oracle_conv.build_specs(in1, in2, out, instructions)
    generator = torch.Generator().manual_seed(seed)
    src, dst = skewed_graph(nodes, edges, generator, skew)
    p = random_problem((meta["in1_dim"], meta["in2_dim"], meta["out_dim"], meta["weight_numel"]), nodes, src, dtype,
                       generator)
    ref = oracle_conv.conv_derivatives(meta, *(p[k].double() for k in ("x", "y", "w")), src, dst, nodes,
                                       p["g"].double(), p["rx"].double(), p["ry"].double(), None)
    graph = module.create_graph(src.to(DEVICE), dst.to(DEVICE), nodes)
    x, y, w, g = (p[k].to(DEVICE).requires_grad_(True) for k in ("x", "y", "w", "g"))
    result = module(x, y, w, graph=graph)
    (gw,) = torch.autograd.grad(result, w, g, retain_graph=True)
    (gy,) = torch.autograd.grad(result, y, g, retain_graph=True)
    gx, gy_too = torch.autograd.grad(result, (x, y), g, create_graph=True)
    (hw,) = torch.autograd.grad((gx, gy_too), w, (p["rx"].to(DEVICE), p["ry"].to(DEVICE)))
    module.op.check_status()
    for key, value in dict(gw=gw, gy=gy, hw=hw).items():
        assert_close(value, ref[key], dtype, f"{shape} x{mul} {dtype} {key} alone")


# three channels per lane: two edges at a time (48), all lanes (96), idle lanes (66, 72), two warps per edge (102, 144)
@pytest.mark.parametrize("shape,mul,dtype", [
    *((shape, mul, dtype) for shape in range(len(SHAPES)) for mul in (48, 96) for dtype in (torch.float32, torch.float64)),
    (4, 72, torch.float32), (1, 144, torch.float32), (4, 66, torch.float64), (4, 102, torch.float64), (3, 144, torch.float64)])
def test_three_channels_per_lane(shape, mul, dtype):
    check(SHAPES[shape], mul, dtype, 29, 400, 0.0, shape)  # long rows: shared by teams
    one_gradient_alone(SHAPES[shape], mul, dtype, 150, 190, 1.5, shape + 50)  # short rows: tiles, many rows without edges
    one_gradient_alone(SHAPES[shape], mul, dtype, 460, 2100, 0.0, shape + 90)  # equal parts


# three, seven, ten and thirteen teams fit: of a row per CTA, and of two
@pytest.mark.parametrize("shape,mul,dtype", [(5, 128, torch.float32), (4, 96, torch.float64), (4, 64, torch.float64),
                                             (6, 128, torch.float64), (2, 48, torch.float32), (6, 96, torch.float32)])
def test_teams_of_few_rows(shape, mul, dtype):
    check(SHAPES[shape], mul, dtype, 24, 552, 0.0, mul)
    check(SHAPES[shape], mul, dtype, 230, 4100, 0.0, mul + 1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_one_gradient_alone(shape, dtype):
    """dL/dw alone and dL/dy alone, whose rows may be the destinations, and two tangents added into one dL/dw; rows shared
    by teams, and tiles with rows without edges."""
    for mul, nodes, edges, skew in ((32, 29, 400, 0.0), (48, 150, 190, 1.5), (160, 40, 130, 1.0)):
        one_gradient_alone(SHAPES[shape], mul, dtype, nodes, edges, skew, 100 + shape)


def term_by_term(meta, x, y, w, g, src, dst):
    """Output and first derivatives as sums over the non-zero coupling terms: a value that is not finite reaches exactly
    the results it is a factor of (a dense contraction would multiply it by the zeros of the coupling tensors too)."""
    out, gx, gy, gw = (torch.zeros_like(t) for t in (g, x, y, w))
    for spec in meta["specs"]:
        cg = torch.as_tensor(spec["cg"], dtype=torch.float64)
        channel = torch.arange(spec["channels"])
        for i, j, k in cg.nonzero().tolist():
            columns = (spec["x_offset"] + channel * spec["d1"] + i, spec["y_offset"] + j,
                       spec["weight_offset"] + channel * spec["weight_stride"],
                       spec["out_offset"] + channel * spec["d3"] + k)
            a, b, c, d = x[src][:, columns[0]], cg[i, j, k] * y[:, columns[1], None], w[:, columns[2]], g[dst][:, columns[3]]
            out[:, columns[3]] = out[:, columns[3]].index_add(0, dst, a * b * c)
            gx[:, columns[0]] = gx[:, columns[0]].index_add(0, src, b * c * d)
            gy[:, columns[1]] += (cg[i, j, k] * a * c * d).sum(1)
            gw[:, columns[2]] += a * b * d
    return dict(out=out, gx=gx, gy=gy, gw=gw)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("mul", [12, 16, 32, 48, 64, 128, 160])
@pytest.mark.parametrize("shape", [3, 4, 6])
def test_values_that_are_not_finite_stay_where_they_belong(shape, mul, dtype):
    """Infinities and NaN in the last channel, which idle lanes read too, and in single edge attributes, which matrix
    entries made of one attribute must not meet.  Finite results stay finite and right, infinite ones keep their sign; where
    the terms disagree (infinity less infinity) any result that is not finite will do."""
    in1, in2, out = irreps(mul, SHAPES[shape][0]), irreps(1, SHAPES[shape][1]), irreps(mul, SHAPES[shape][2])
    instructions = all_paths(in1, in2, out)
    module = luna.TensorProductConv(in1, in2, out, instructions, internal_weights=False, shared_weights=False,
                                    dtype=dtype)
    assert module.op.backward_variant == "row"
    meta = oracle_conv.build_specs(in1, in2, out, instructions)
    generator = torch.Generator().manual_seed(shape + mul)
    nodes, edges = 9, 40
    src, dst = skewed_graph(nodes, edges, generator, 0.0)
    clean = random_problem((meta["in1_dim"], meta["in2_dim"], meta["out_dim"], meta["weight_numel"]), nodes, src, dtype,
                           generator)
    graph = module.create_graph(src.to(DEVICE), dst.to(DEVICE), nodes)
    inf, nan = float("inf"), float("nan")
    for key, row, column, value in (("x", int(src[3]), mul - 1, -inf), ("w", 5, 2 * mul - 1, inf), ("w", 5, mul - 1, nan),
                                    ("g", int(dst[7]), mul - 1, inf), ("y", 11, 0, inf), ("y", 11, 0, nan), ("y", 11, 2, -inf)):
        p = {k: clean[k].clone() for k in ("x", "y", "w", "g")}
        p[key][row, column] = value
        ref = term_by_term(meta, *(p[k].double() for k in ("x", "y", "w", "g")), src, dst)
        x, y, w, g = (p[k].to(DEVICE).requires_grad_(True) for k in ("x", "y", "w", "g"))
        result = module(x, y, w, graph=graph)
        gx, gy, gw = torch.autograd.grad(result, (x, y, w), g, retain_graph=True)
        (gy_alone,) = torch.autograd.grad(result, y, g, retain_graph=True)
        (gw_alone,) = torch.autograd.grad(result, w, g)
        for name, got in dict(out=result, gx=gx, gy=gy, gw=gw, gy_alone=gy_alone, gw_alone=gw_alone).items():
            want, got = ref[name.removesuffix("_alone")], got.detach().cpu().double()
            what = f"{SHAPES[shape]} x{mul} {dtype} {key}[{row}, {column}] = {value}: {name}"
            finite, infinite = want.isfinite(), want.isinf()
            assert bool((got.isfinite() == finite).all()), what
            assert bool((got[infinite] == want[infinite]).all()), what
            assert_close(got[finite], want[finite], dtype, what)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_two_edges_at_a_time(shape, dtype):
    """16 and 32 channels, a half warp per edge: rows of odd and even lengths, one edge, rows without edges between the two
    edges of a pair, and one gradient alone."""
    for mul in (16, 32):
        module = check(SHAPES[shape], mul, dtype, 31, 403, 0.0, mul + shape)
        if mul == 16 or dtype == torch.float32:
            assert module.op._plan.query(1) == mul // 16  # channels per lane
        check(SHAPES[shape], mul, dtype, 150, 191, 1.5, mul + shape + 50)
        one_gradient_alone(SHAPES[shape], mul, dtype, 150, 191, 1.5, mul + shape + 90)
    for nodes, edges in ((1, 1), (1, 2), (2, 3), (900, 7201), (2500, 2501)):
        check(SHAPES[shape], 16, dtype, nodes, edges, 0.5, nodes + edges)


# one warp per edge, two edges per warp, two warps per edge, slices
@pytest.mark.parametrize("mul,dtype", [(48, torch.float32), (16, torch.float32), (160, torch.float32), (352, torch.float32),
                                       (64, torch.float64), (32, torch.float64)])
def test_equal_parts_of_the_edges(mul, dtype):
    """Rows that many teams share, parts within one row, more CTAs than rows, rows without edges at either end of a part."""
    for nodes, edges, skew in ((1, 500, 0.0), (3, 41, 0.0), (149, 1500, 0.0), (149, 1500, 2.0), (600, 9001, 3.0), (2900, 29007, 0.3)):
        check(SHAPES[3], mul, dtype, nodes, edges, skew, nodes + mul)
    check(SHAPES[4], mul, dtype, 300, 5003, 2.5, mul)
    one_gradient_alone(SHAPES[4], mul, dtype, 300, 5003, 2.5, mul)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_output_and_weight_gradient_of_the_second_order(shape, dtype):
    """The two in one call, as force training asks for them: one launch, or two where that is faster."""
    from lunaequivariance_b200 import conv as conv_mod

    for mul, nodes, edges, skew in ((16, 150, 191, 1.5), (48, 31, 403, 0.0), (128, 60, 90, 1.0), (352, 7, 120, 0.0)):
        in1, in2, out = irreps(mul, SHAPES[shape][0]), irreps(1, SHAPES[shape][1]), irreps(mul, SHAPES[shape][2])
        instructions = all_paths(in1, in2, out)
        module = luna.TensorProductConv(in1, in2, out, instructions, internal_weights=False, shared_weights=False, dtype=dtype)
        meta = oracle_conv.build_specs(in1, in2, out, instructions)
        generator = torch.Generator().manual_seed(shape + mul)
        src, dst = skewed_graph(nodes, edges, generator, skew)
        p = random_problem((meta["in1_dim"], meta["in2_dim"], meta["out_dim"], meta["weight_numel"]), nodes, src, dtype,
                           generator)
        ref = oracle_conv.conv_derivatives(meta, *(p[k].double() for k in ("x", "y", "w")), src, dst, nodes, p["g"].double(),
                                           None, p["ry"].double(), None)
        graph = module.create_graph(src.to(DEVICE), dst.to(DEVICE), nodes)
        x, y, w, g, ry = (p[k].to(DEVICE) for k in ("x", "y", "w", "g", "ry"))
        hx, hy, hw, hg = conv_mod.run_double_backward(module.op, x, y, w, g, None, ry, None, graph, needs=(False, False, True, True))
        module.op.check_status()
        assert hx is None and hy is None
        assert_close(hw, ref["hw"], dtype, f"{SHAPES[shape]} x{mul} {dtype} hw")
        assert_close(hg, ref["hg"], dtype, f"{SHAPES[shape]} x{mul} {dtype} hg")


@pytest.mark.parametrize("shape", [0, 1, 3, 7, 8, 10])
def test_two_edges_at_a_time_with_four_channels_per_lane(shape):
    """64 channels of the shapes whose paths all have a degree of zero; the forward at degree 2 only."""
    module = check(SHAPES[shape], 64, torch.float32, 31, 403, 0.0, shape)
    assert module.op._plan.query(1) == (4 if shape in (1, 8) else 2)
    check(SHAPES[shape], 64, torch.float32, 150, 191, 1.5, shape + 50)
    check(SHAPES[shape], 64, torch.float32, 900, 7201, 0.5, shape + 70)
    one_gradient_alone(SHAPES[shape], 64, torch.float32, 150, 191, 1.5, shape + 90)


@pytest.mark.parametrize("shape,mul", [(3, 32), (3, 16), (8, 64), (10, 16)])
def test_parts_without_edges_behind_the_last_row(shape, mul):
    """Teams without an edge where the last row has begun already, which find no row there; the row tables are views that end
    inside a larger tensor, as a caller's may."""
    in1, in2, out = irreps(mul, SHAPES[shape][0]), irreps(1, SHAPES[shape][1]), irreps(mul, SHAPES[shape][2])
    instructions = all_paths(in1, in2, out)
    module = luna.TensorProductConv(in1, in2, out, instructions, internal_weights=False, shared_weights=False)
    meta = oracle_conv.build_specs(in1, in2, out, instructions)
    generator = torch.Generator().manual_seed(shape + mul)
    for degrees in ([4] * 500, [5] * 450, [16] * 1000 + [200]):
        nodes, dst = len(degrees), torch.arange(len(degrees)).repeat_interleave(torch.tensor(degrees))
        src = torch.randint(nodes, dst.shape, generator=generator)
        p = random_problem((meta["in1_dim"], meta["in2_dim"], meta["out_dim"], meta["weight_numel"]), nodes, src, torch.float32,
                           generator)
        ref = oracle_conv.conv_derivatives(meta, *(p[k].double() for k in ("x", "y", "w")), src, dst, nodes, p["g"].double(),
                                           None, None, None)
        graph = module.create_graph(src.to(DEVICE), dst.to(DEVICE), nodes)
        behind = torch.full((5,), 2**31 - 1, dtype=torch.int32, device=DEVICE)
        graph = dataclasses.replace(graph, dst_rowptr=torch.cat([graph.dst_rowptr, behind])[:nodes + 1],
                                    src_rowptr=torch.cat([graph.src_rowptr, behind])[:nodes + 1])
        x, y, w, g = (p[k].to(DEVICE) for k in ("x", "y", "w", "g"))
        result = conv_mod.run_forward(module.op, x, y, w, graph)
        gx, gy, gw = conv_mod.run_backward(module.op, x, y, w, g, graph)
        module.op.check_status()
        for key, value in dict(out=result, gx=gx, gy=gy, gw=gw).items():
            assert_close(value, ref[key], torch.float32, f"{SHAPES[shape]} x{mul} {nodes} nodes {key}")


def launches(op, dtype, nodes, edges, which, tmp_path):
    """(kernel, channels per lane, warps and shared memory of a block) of the edge kernels that a call launches."""
    src, dst = skewed_graph(nodes, edges, torch.Generator().manual_seed(nodes), 0.0)
    graph = luna.make_graph(src.to(DEVICE), dst.to(DEVICE), nodes)
    x, y, w, g = (torch.zeros(*rows, dtype=dtype, device=DEVICE)
                  for rows in ((nodes, op.in1_dim), (edges, op.in2_dim), (edges, op.weight_numel), (nodes, op.out_dim)))
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as profile:
        if which == "forward":
            conv_mod.run_forward(op, x, y, w, graph)
        else:
            conv_mod.run_backward(op, x, y, w, g, graph, tuple(key in which for key in "xyw"))
        torch.cuda.synchronize()
    profile.export_chrome_trace(str(tmp_path / "trace.json"))
    found = []
    for event in json.loads((tmp_path / "trace.json").read_text())["traceEvents"]:
        match = re.search(r"(edge|pair)_(?:fwd|bwd)_kernel<(?:float|double), (\d)", event.get("name", ""))
        if match and "shared memory" in event.get("args", {}):
            found.append((match[1], int(match[2]), event["args"]["block"][0] // 32, event["args"]["shared memory"]))
    return found


# The kernels of small graphs, of larger ones and of those that hand out tiles: the plan's figure bounds what any launch takes.
@pytest.mark.parametrize("shape,mul,dtype", [(4, 48, torch.float32), (4, 96, torch.float64), (3, 48, torch.float64),
                                             (5, 128, torch.float32), (4, 64, torch.float32), (3, 352, torch.float32)])
def test_shared_memory_of_a_forward_block(shape, mul, dtype, tmp_path):
    in1, in2, out = irreps(mul, SHAPES[shape][0]), irreps(1, SHAPES[shape][1]), irreps(mul, SHAPES[shape][2])
    op = luna.TensorProductConv(in1, in2, out, all_paths(in1, in2, out), internal_weights=False, shared_weights=False,
                                dtype=dtype).op
    for nodes, edges in ((24, 552), (700, 12_000), (900, 1_800)):
        (launch,) = launches(op, dtype, nodes, edges, "forward", tmp_path)
        assert launch[3] <= op._plan.query(3), (nodes, launch)


# Layouts that are slower than the ones beside them are not chosen.
@pytest.mark.parametrize("shape,mul,dtype,which,kernel,lane_channels,warps", [
    # an estimate of registers that is taken to be too high
    (8, 64, torch.float32, "xw", "pair", 4, [12]), (8, 48, torch.float64, "xw", "pair", 3, [8]),
    (2, 80, torch.float32, "y", "edge", 4, [12]), (2, 128, torch.float32, "y", "edge", 4, [16]),
    (4, 48, torch.float64, "forward", "edge", 2, [12]),
    # idle lanes, and states that are too large, of the layout with less work
    (5, 80, torch.float32, "forward", "edge", 4, None), (5, 160, torch.float32, "forward", "edge", 4, None),
    (5, 128, torch.float32, "forward", "edge", 2, None), (5, 192, torch.float64, "y", "edge", 2, None),
    (6, 192, torch.float64, "xw", "edge", 2, None), (6, 192, torch.float64, "w", "edge", 3, None),
    # too many bulk copies under way
    (7, 96, torch.float32, "forward", "edge", 3, [16]), (0, 96, torch.float32, "forward", "edge", 3, [24]),
])
def test_layout_of_a_launch(shape, mul, dtype, which, kernel, lane_channels, warps, tmp_path):
    in1, in2, out = irreps(mul, SHAPES[shape][0]), irreps(1, SHAPES[shape][1]), irreps(mul, SHAPES[shape][2])
    op = luna.TensorProductConv(in1, in2, out, all_paths(in1, in2, out), internal_weights=False, shared_weights=False,
                                dtype=dtype).op
    (launch,) = launches(op, dtype, 700, 12_000, which, tmp_path)
    assert launch[:2] == (kernel, lane_channels) and launch[2] in (warps or [launch[2]]), launch


# One warp per edge and several, rows by source and by destination: the smallest work for a stage of all kernels, whose last read
# comes straight before the row that replaces it.
@pytest.mark.parametrize("shape,mul,nodes,edges", [(2, 224, 2453, 27_901), (9, 128, 3524, 18_953), (9, 60, 1514, 104_166)])
def test_a_stage_is_read_before_it_is_refilled(shape, mul, nodes, edges):
    in1, in2, out = irreps(mul, SHAPES[shape][0]), irreps(1, SHAPES[shape][1]), irreps(mul, SHAPES[shape][2])
    op = luna.TensorProductConv(in1, in2, out, all_paths(in1, in2, out), internal_weights=False, shared_weights=False,
                                dtype=torch.float64).op
    src, dst = skewed_graph(nodes, edges, torch.Generator().manual_seed(5), 0.0)
    graph = luna.make_graph(src.to(DEVICE), dst.to(DEVICE), nodes)
    generator = torch.Generator(device=DEVICE).manual_seed(5)
    x, y, w, g = (torch.randn(*rows, generator=generator, dtype=torch.float64, device=DEVICE)
                  for rows in ((nodes, op.in1_dim), (edges, op.in2_dim), (edges, op.weight_numel), (nodes, op.out_dim)))
    _, want, _ = conv_mod.run_backward(op, x, y, w, g, graph)
    results = [torch.empty_like(want) for _ in range(120)]
    for gy in results:
        conv_mod.run_backward(op, x, y, w, g, graph, (False, True, False), out=(None, gy, None))
    op.check_status()
    assert_close(results[0], want.cpu(), torch.float64, "dL/dy alone")
    assert all(torch.equal(gy, results[0]) for gy in results)
