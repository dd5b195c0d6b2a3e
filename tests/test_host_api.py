"""CPU-only checks: the C-ABI library loads and exports every declared symbol, host-side validation, graph tables
on CPU tensors (the reference's known-answer tests, tests/lunatp/test_make_graph.py:9-55), module surface."""

import os
import re

import pytest
import torch

import lunaequivariance_b200 as luna
from lunaequivariance_b200 import _native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol():
    header = open(os.path.join(ROOT, "include", "luna_b200.h")).read()
    declared = set(re.findall(r"LUNA_API [\w\s\*]+?\b(luna_\w+)\(", header))
    assert declared and declared == set(_native.EXPORTED_SYMBOLS)
    lib = _native.library()
    for name in declared:
        assert getattr(lib, name) is not None
    assert lib.luna_compiled_sm() == 100


def test_plan_creation_and_errors_without_gpu():
    op = luna.prepare_tensor_product("32x0e+32x1o", "1x0e+1x1o", "32x0e+32x1o",
                                     [(0, 0, 0, "uvu", True), (1, 1, 0, "uvu", True), (0, 1, 1, "uvu", True),
                                      (1, 0, 1, "uvu", True)], convolution=True)
    assert op.weight_numel == 128 and op.out_dim == 128 and op.uses_staged_kernels
    odd = luna.prepare_tensor_product("33x0e", "1x0e", "33x0e", [(0, 0, 0, "uvu", True)], convolution=True)
    assert not odd.uses_staged_kernels
    bad = dict(op.meta)
    bad["generated_specs"] = [dict(op.meta["generated_specs"][0], x_offset=10_000)]
    with pytest.raises(ValueError, match="outside its tensor dimension"):
        luna.TensorProductConv(bad, mode="uvu")
    with pytest.raises(ValueError, match="float32 or torch.float64"):
        luna.create_uvu_conv_operator(op.meta, dtype=torch.float16)
    with pytest.raises(ValueError, match='mode="uuu" or mode="uvu"'):
        luna.TensorProductConv(op.meta)
    with pytest.raises(TypeError):
        luna.TensorProductConv("32x0e")
    with pytest.raises(ValueError, match="one connection mode"):
        luna.TensorProductConv("2x0e", "2x0e", "2x0e", [(0, 0, 0, "uvu", True), (0, 0, 0, "uuu", True)],
                               internal_weights=False, shared_weights=False)
    with pytest.raises(ValueError, match="internal_weights=False"):
        luna.TensorProductConv("2x0e", "1x0e", "2x0e", [(0, 0, 0, "uvu", True)])


def test_module_surface():
    conv = luna.TensorProductConv("4x0e+4x1o", "1x0e+1x1o", "4x0e+4x1o",
                                  [(0, 0, 0, "uvu", True), (1, 1, 0, "uvu", True)],
                                  internal_weights=False, shared_weights=False)
    assert conv.mode == "uvu_conv" and conv.weight_numel == 8
    assert str(conv.irreps_in1) == "4x0e+4x1o" and len(conv.instructions) == 2
    assert conv.internal_weights is False and conv.shared_weights is False
    assert conv.op.compute_dtype == torch.float32
    assert conv.double().op.compute_dtype == torch.float64
    meta_conv = luna.TensorProductConv(conv.op.meta, mode="uvu", dtype=torch.float64)
    assert meta_conv.weight_numel == 8
    import pickle

    restored = pickle.loads(pickle.dumps(conv.op))
    assert restored.weight_numel == 8 and restored.compute_dtype == torch.float64


def test_destination_sorted_endpoints_are_preserved():
    src, dst = torch.tensor([2, 0, 1]), torch.tensor([0, 1, 2])
    graph = luna.make_graph(src, dst, 4)
    assert torch.equal(graph.dst, dst.to(graph.dst.dtype)) and torch.equal(graph.src, src.to(graph.src.dtype))
    assert graph.dst_rowptr.tolist() == [0, 1, 2, 3, 3]


def test_invalid_graph_includes_values():
    with pytest.raises(ValueError, match="num_nodes=2.*at least 4"):
        luna.make_graph(torch.tensor([3]), torch.tensor([0]), 2)
    with pytest.raises(ValueError, match="nonnegative"):
        luna.make_graph(torch.tensor([-1]), torch.tensor([0]), 2)
    with pytest.raises(TypeError):
        luna.make_graph(torch.tensor([0.0]), torch.tensor([0.0]), 2)
    with pytest.raises(ValueError, match="equal shape"):
        luna.make_graph(torch.tensor([0, 1]), torch.tensor([0]), 2)


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_generated_graph_tables_and_input_ownership(dtype):
    src = torch.tensor([2, 0, 1, 0], dtype=dtype)
    dst = torch.tensor([0, 1, 1, 2], dtype=dtype)
    graph = luna.make_graph(src, dst, 4)
    assert graph.src_rowptr.tolist() == [0, 2, 3, 4, 4]
    assert graph.dst_rowptr.tolist() == [0, 1, 3, 4, 4]
    assert graph.edge_ids_by_src.sort().values.tolist() == [0, 1, 2, 3]
    assert graph.src[graph.edge_ids_by_src.long()].tolist() == [0, 0, 1, 2]
    assert graph.edge_ids_by_dst.tolist() == [0, 1, 2, 3]
    for rowptr, order in ((graph.dst_rowptr, graph.node_order), (graph.src_rowptr, graph.source_node_order)):
        assert order.sort().values.tolist() == [0, 1, 2, 3]
        assert rowptr.diff()[order.long()].tolist() == [2, 1, 1, 0]
    assert graph.src.data_ptr() != src.data_ptr() and graph.dst.data_ptr() != dst.data_ptr()
    src.zero_()
    dst.zero_()
    assert graph.src.tolist() == [2, 0, 1, 0] and graph.dst.tolist() == [0, 1, 1, 2]
    assert len(graph.table_list()) == 13


def test_spherical_harmonics_argument_handling():
    from lunaequivariance_b200.spherical_harmonics import parse_irreps

    irreps_in, out, degrees = parse_irreps("1x0e+1x1o+1x2e")
    assert str(irreps_in) == "1x1o" and degrees == (0, 1, 2) and out.dim == 9
    assert parse_irreps([3, 1, 3, 0])[2] == (3, 1, 3, 0)
    assert str(parse_irreps("1x1e")[0]) == "1x1e"
    with pytest.raises(ValueError, match="parity"):
        parse_irreps("1x1e", "1o")
    with pytest.raises(NotImplementedError):
        parse_irreps(13)
    with pytest.raises(TypeError):
        luna.SphericalHarmonics("1x0e")
    with pytest.raises(ValueError):
        luna.SphericalHarmonics("1x0e", normalize=True, normalization="bogus")


def test_custom_op_fake_shapes():
    """The shape functions registered for torch.compile run on meta tensors without any kernel."""
    op = luna.prepare_tensor_product("4x0e+4x1o", "1x0e+1x1o", "4x0e+4x1o",
                                     [(0, 0, 0, "uvu", True), (1, 1, 0, "uvu", True)], convolution=True)
    x = torch.empty(5, 16, device="meta")
    y = torch.empty(9, 4, device="meta")
    w = torch.empty(9, 8, device="meta")
    tables = [torch.empty(9, dtype=torch.int32, device="meta")] * 13
    out, l0 = torch.ops.lunatp.uvu_conv_forward(x, y, w, None, tables, 5, False, op.torch_config)
    assert out.shape == (5, 16) and l0 is None
    grads = torch.ops.lunatp.uvu_conv_backward(x, y, w, None, out, None, tables, 5, [True, False, True, False],
                                               op.torch_config)
    assert grads[0].shape == x.shape and grads[1] is None and grads[2].shape == w.shape
    v = torch.empty(7, 3, device="meta")
    from lunaequivariance_b200.spherical_harmonics import SphericalHarmonicsConfig

    desc = SphericalHarmonicsConfig((0, 1, 2), True, "component", torch.float32).descriptor()
    assert torch.ops.lunaeq.spherical_harmonics_forward(v, desc).shape == (7, 9)


def test_canonical_path_lists_are_detected_without_gpu():
    """Full lists of allowed couplings of degrees from 0 on are recognised; lists with gaps or in another order are not."""
    from tests.helpers import config

    expected = {"cfg2": 3, "cfg4": 3, "cfg5": 2, "fixture": 1, "wide": 1, "cfg1": -1, "partial": -1}
    for name, l2 in expected.items():
        in1, in2, out, instructions, options = config(name)
        op = luna.prepare_tensor_product(in1, in2, out, instructions, convolution=True, **options)
        assert op.uses_staged_kernels, name
        assert op.canonical_l2 == l2, (name, op.canonical_l2)
        assert op.uses_compiled_patterns == (l2 >= 0), name
    # the same couplings in another order are not canonical (weight blocks follow the instruction order)
    in1, in2, out, instructions, options = config("fixture")
    shuffled = luna.prepare_tensor_product(in1, in2, out, instructions[::-1], convolution=True)
    assert shuffled.uses_staged_kernels and shuffled.canonical_l2 == -1


def test_launch_path_shares_the_cpp_runtime():
    """A second, static copy of the C++ runtime beside torch's makes error texts crash."""
    from lunaequivariance_b200 import _native

    _native.binding()
    with open(_native.BINDING_PATH, "rb") as module:
        assert b"libstdc++.so" in module.read()


def test_forward_mode_operands_are_refused_by_the_launch_path():
    """The kernels drop the tangent of a dual tensor, which need not require grad: it must not get as far as a launch."""
    import torch.autograd.forward_ad as forward_ad

    from tests.helpers import config

    in1, in2, out, instructions, options = config("small")
    op = luna.prepare_tensor_product(in1, in2, out, instructions, convolution=True, **options)
    src, dst = torch.tensor([0, 1, 1]), torch.tensor([0, 0, 1])
    holder = luna.make_graph(src, dst, 2).native_holder()
    shapes = ((2, op.in1_dim), (3, op.in2_dim), (3, op.weight_numel))
    for dual in range(3):
        with forward_ad.dual_level():
            operands = [torch.ones(shape) for shape in shapes]
            operands[dual] = forward_ad.make_dual(operands[dual], torch.ones(shapes[dual]))
            with pytest.raises(NotImplementedError, match="forward-mode"):  # asked before the device is looked at
                _native.binding().conv(op._plan.op, holder, *operands)


def test_forward_mode_vectors_are_refused_by_the_harmonics():
    import torch.autograd.forward_ad as forward_ad

    from lunaequivariance_b200.spherical_harmonics import SphericalHarmonicsConfig

    holder = SphericalHarmonicsConfig((0, 1, 2), True, "component", torch.float32).holder(torch.float32)
    with forward_ad.dual_level():
        vectors = forward_ad.make_dual(torch.ones(5, 3), torch.ones(5, 3))
        with pytest.raises(NotImplementedError, match="forward-mode"):
            _native.binding().harmonics(holder, vectors)
        constant = SphericalHarmonicsConfig((0,), True, "component", torch.float32).holder(torch.float32)
        with pytest.raises(RuntimeError, match="CUDA is required"):  # not refused: its derivative is zero
            _native.binding().harmonics(constant, vectors)


def test_default_build_leaves_line_tables_out():
    """They made the library and its objects 360 MB, too much for a checkout that is copied about with its build."""
    from lunaequivariance_b200 import build

    assert "-lineinfo" not in build.NVCC_FLAGS
    assert os.path.getsize(_native.LIBRARY_PATH) < 100 << 20


def test_scratch_is_asked_for_only_where_it_is_used(monkeypatch):
    from tests.helpers import all_paths, config

    def plan(in1, in2, out, instructions, dtype):
        op = luna.prepare_tensor_product(in1, in2, out, instructions, convolution=True, dtype=dtype)
        return op, _native.library().luna_uvu_conv_scratch_bytes(op._plan.handle, 100, 1000), op._plan.query(8)

    cfg2 = config("cfg2")[:4]
    wide = ("352x0e+352x1o", "1x0e+1x1o", "352x0e+352x1o")
    op, size, needs = plan(*cfg2, torch.float64)  # one team of warps takes the 128 channels
    assert (op.backward_variant, size, needs) == ("row", 0, 0)
    op, size, needs = plan(*wide, all_paths(*wide), torch.float32)  # eleven slices
    assert (op.backward_variant, size, needs) == ("row", 11 * 1000 * 4 * 4, 1)
    monkeypatch.setenv("LUNA_B200_NO_CANON", "1")
    op, size, needs = plan(*cfg2, torch.float64)  # two channel chunks of the table kernels
    assert (op.backward_variant, size, needs) == ("tables", 2 * 1000 * 16 * 8, 1)


@pytest.mark.parametrize("mul,lmax,dtype,lanes,chunks", [
    (48, 2, torch.float32, 2, 1), (64, 2, torch.float32, 2, 1), (128, 3, torch.float64, 2, 1), (352, 1, torch.float32, 1, 11)])
def test_plan_queries_describe_the_kernels_that_run(mul, lmax, dtype, lanes, chunks):
    from tests.helpers import all_paths

    block = lambda m, top: "+".join(f"{m}x{l}{'eo'[l % 2]}" for l in range(top + 1))
    irreps = (block(mul, lmax), block(1, lmax), block(mul, lmax))
    op = luna.prepare_tensor_product(*irreps, all_paths(*irreps), convolution=True, dtype=dtype)
    assert op.backward_variant == "row" and op.uses_staged_kernels and op.uses_compiled_patterns
    assert (op.canonical_l2, op._plan.query(1), op._plan.query(2)) == (lmax, lanes, chunks)
    row = op.weight_numel // chunks * (8 if dtype == torch.float64 else 4)
    for smem in (op._plan.query(3), op._plan.query(4)):
        assert 2 * row < smem <= 227 * 1024
    # a full list that no kernel has compiled in
    irreps = (block(64, 1), block(1, 2), block(64, 2))
    op = luna.prepare_tensor_product(*irreps, all_paths(*irreps), convolution=True, dtype=dtype)
    assert op.backward_variant == "tables" and op.canonical_l2 == 2 and not op.uses_compiled_patterns


@pytest.mark.parametrize("dtype,rounding", [(torch.float32, 1e-7), (torch.float64, 1e-15)])
def test_compiled_patterns_need_one_coefficient_where_a_degree_is_zero(dtype, rounding):
    """The edge kernels take the coupling of a path with a degree of zero as one number: terms that differ by rounding are
    that, terms that differ by more go to the kernels that read every term."""
    from tests.helpers import all_paths

    irreps = ("64x0e+64x1o", "1x0e+1x1o", "64x0e+64x1o")
    meta = luna.prepare_tensor_product(*irreps, all_paths(*irreps), convolution=True, dtype=dtype).meta
    for factor, variant in ((1 + rounding, "row"), (1.001, "tables")):
        for spec in meta["generated_specs"]:
            if len(spec["terms"]) != 3:
                continue
            i, j, k, c = spec["terms"][1]
            terms = [spec["terms"][0], (i, j, k, c * factor), spec["terms"][2]]
            changed = [dict(s, terms=terms) if s is spec else s for s in meta["generated_specs"]]
            op = luna.create_uvu_conv_operator(dict(meta, generated_specs=changed), dtype=dtype)
            assert op.backward_variant == variant, (spec["l1"], spec["l2"], spec["l3"], factor)
