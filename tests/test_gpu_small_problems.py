"""The paths for small work, at the sizes where they can go wrong."""
import numpy as np
import pytest

from oxionnx_b200 import models
from oxionnx_b200.graph import Graph, Node
from oxionnx_b200.session import Session

pytestmark = pytest.mark.gpu


def test_dispatch_plans_follow_their_operands():
    """A kept single-node plan must not carry anything over from the call before: new lanes, new shapes, re-registered
    weights, more nodes than are kept."""
    from oxionnx_b200.session import CudaContext, try_cuda_dispatch, try_cuda_dispatch_resident
    rng = np.random.default_rng(3)
    ctx = CudaContext(0)
    node = Node("Conv", "c", ["x", "w"], ["y"], {"pads": [1, 1, 1, 1]})
    relu = Node("Relu", "r", ["y"], ["z"], {})
    for rnd in range(3):
        w = (rng.standard_normal((32, 32, 3, 3)) * 0.05).astype(np.float32)
        ctx.register_weights({"w": w})
        for hw in list(range(4, 24)) + [5, 4]:
            x = rng.standard_normal((1, 32, hw, hw)).astype(np.float32)
            y = try_cuda_dispatch_resident(node, {"w": w}, {"x": x}, "device", ctx)
            z = try_cuda_dispatch(relu, {}, {"y": y}, ctx)[0]
            want = try_cuda_dispatch(Node("Conv", "fresh", ["x", "v"], ["y"], {"pads": [1, 1, 1, 1]}), {}, {"x": x, "v": w}, ctx)[0]
            assert np.array_equal(z, np.maximum(want, 0))
            y.release()
    ctx.close()


def _run(graph, weights, feeds, **tuning):
    b = Session.builder()
    if "kernel_path" in tuning:
        b = b.with_kernel_path(tuning.pop("kernel_path"))
    sess = b.with_tuning(**tuning).build_from_graph(graph, weights)
    out = sess.run(feeds)
    kernels = [s["kernel"] for s in sess.steps()]
    sess.close()
    return out, kernels


# batch, channels, height, width, filters, kernel, stride: ragged row and channel tiles, slices of uneven length
SHAPES = [(1, 32, 1, 1, 32, 1, 1), (1, 64, 5, 7, 40, 3, 1), (1, 128, 13, 11, 96, 1, 1), (1, 512, 7, 7, 512, 3, 1), (2, 256, 9, 9, 1000, 1, 1), (1, 2048, 1, 1, 1000, 1, 1),
          (1, 64, 17, 16, 64, 3, 2), (3, 384, 7, 7, 130, 3, 1)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("requant", ["packed", "f64", "union"])
def test_small_integer_convolutions_match_the_direct_kernel(shape, requant):
    n, c, h, w, oc, k, stride = shape
    rng = np.random.default_rng([n, c, h, oc, k])
    weights = {"w": rng.integers(-127, 128, (oc, c, k, k)).astype(np.float32), "ws": rng.uniform(0.001, 0.01, oc).astype(np.float32),
               "wz": np.zeros(oc, np.float32), "b": rng.integers(-1000, 1001, oc).astype(np.float32), "xs": np.float32([0.02]), "z0": np.float32([0]),
               "ys": np.float32([0.05 * np.sqrt(c * k * k)]), "yz": np.float32([0 if requant == "union" else 128])}
    nodes = [Node("QuantizeLinear", "q", ["x", "xs", "z0"], ["xq"], {}),
             Node("QLinearConv", "conv", ["xq", "xs", "z0", "w", "ws", "wz", "ys", "yz", "b"], ["yq"], {"strides": [stride] * 2, "pads": [k // 2] * 4}),
             Node("DequantizeLinear", "dq", ["yq", "ys", "yz"], ["y"], {})]
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["y"])
    feeds = {"x": rng.standard_normal((n, c, h, w)).astype(np.float32)}
    got, kernels = _run(graph, weights, feeds, requant_f64=1 if requant == "f64" else 0)
    assert any("small" in s for s in kernels), kernels
    want, _ = _run(graph, weights, feeds, kernel_path="direct")
    assert np.array_equal(got["y"], want["y"])


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision", ["tf32", "bf16"])
def test_small_float_convolutions_match_the_direct_kernel(shape, precision):
    n, c, h, w, oc, k, stride = shape
    rng = np.random.default_rng([n, c, h, oc, k, 1])
    weights = {"w1": (rng.standard_normal((oc, c, k, k)) / np.sqrt(c * k * k)).astype(np.float32), "b1": rng.standard_normal(oc).astype(np.float32)}
    attrs = {"strides": [stride] * 2, "pads": [k // 2] * 4}
    nodes = [Node("Relu", "pre", ["x"], ["x1"], {}), Node("Conv", "c1", ["x1", "w1", "b1"], ["y"], dict(attrs, activation="relu"))]
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["y"])
    feeds = {"x": rng.standard_normal((n, c, h, w)).astype(np.float32)}
    got, kernels = _run(graph, weights, feeds, float_precision=precision)
    assert any("small" in s for s in kernels), kernels
    want, _ = _run(graph, weights, feeds, kernel_path="direct")
    tol = 2e-3 if precision == "tf32" else 2e-2
    assert np.all(np.abs(got["y"] - want["y"]) <= tol * np.abs(want["y"]) + tol * np.abs(want["y"]).max())


@pytest.mark.parametrize("batch,seq", [(1, 1), (1, 16), (2, 33), (3, 63), (2, 65), (1, 127), (4, 129), (2, 320), (1, 513)])
def test_attention_at_ragged_lengths_is_the_separate_nodes_bit_for_bit(batch, seq):
    graph, weights, feeds, _ = models.build_bert_dynamic_int8(batch=batch, seq=seq, hidden=128, heads=2, ffn=128, layers=2, vocab=100)
    f = feeds()
    f["attention_mask"][:, (seq + 1) // 2:] = 0
    f["attention_mask"][0] = 1
    got, kernels = _run(graph, weights, f)
    assert kernels.count("attention_f32") == 2, kernels
    want, _ = _run(graph, weights, f, keep_intermediates=True)
    assert np.array_equal(got["hidden"], want["hidden"])


# batch, channels, height, width, filters, kernel, pad: ragged tiles of the second pass, the fewest and the most columns
@pytest.mark.parametrize("shape", [(1, 32, 134, 140, 3, 7, 0), (2, 64, 100, 101, 2, 5, 2), (1, 32, 129, 128, 9, 7, 3), (3, 128, 90, 67, 1, 3, 1)])
@pytest.mark.parametrize("activation", ["", "relu"])
def test_row_summed_convolutions_match_the_direct_kernel(shape, activation):
    n, c, h, w, oc, k, pad = shape
    rng = np.random.default_rng([n, c, h, oc, k, 2])
    weights = {"w1": (rng.standard_normal((oc, c, k, k)) / np.sqrt(c * k * k)).astype(np.float32), "b1": rng.standard_normal(oc).astype(np.float32)}
    attrs = {"pads": [pad] * 4}
    if activation:
        attrs["activation"] = activation
    nodes = [Node("Relu", "pre", ["x"], ["x1"], {}), Node("Conv", "c1", ["x1", "w1", "b1"], ["y"], attrs)]
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["y"])
    feeds = {"x": rng.standard_normal((n, c, h, w)).astype(np.float32)}
    got, kernels = _run(graph, weights, feeds)
    assert "row_sums" in kernels, kernels
    want, _ = _run(graph, weights, feeds, kernel_path="direct")
    assert np.all(np.abs(got["y"] - want["y"]) <= 2e-3 * np.abs(want["y"]) + 2e-3 * np.abs(want["y"]).max())


@pytest.mark.parametrize("reader", ["modulators", "other"])
def test_slices_read_in_place_by_the_normalisation(reader):
    n, c, hw = 3, 40, 6
    rng = np.random.default_rng(11)
    weights = {"g": (rng.standard_normal((16, 2 * c)) * 0.3).astype(np.float32), "s0": np.float32([0]), "s1": np.float32([c]), "s2": np.float32([2 * c]),
               "ax": np.float32([1]), "shape": np.float32([n, c, 1, 1])}
    nodes = [Node("MatMul", "mm", ["l", "g"], ["style"], {}), Node("Slice", "sa", ["style", "s0", "s1", "ax"], ["a"], {}),
             Node("Slice", "sb", ["style", "s1", "s2", "ax"], ["b"], {}), Node("Reshape", "ra", ["a", "shape"], ["a4"], {}),
             Node("Reshape", "rb", ["b", "shape"], ["b4"], {}), Node("OxiInstanceNorm", "in", ["x"], ["xn"], {"epsilon": 1e-5}),
             Node("Mul", "mul", ["xn", "a4"], ["xm"], {}), Node("Add", "add", ["xm", "b4"], ["y"], {})]
    outs = ["y"]
    if reader == "other":
        nodes.append(Node("Sigmoid", "sg", ["a"], ["z"], {}))
        outs.append("z")
    graph = Graph(nodes=nodes, input_names=["x", "l"], output_names=outs)
    feeds = {"x": rng.standard_normal((n, c, hw, hw)).astype(np.float32), "l": rng.standard_normal((n, 16)).astype(np.float32)}
    got, kernels = _run(graph, weights, feeds)
    assert kernels.count("slice (read in place)") == (2 if reader == "modulators" else 1), kernels
    want, _ = _run(graph, weights, feeds, keep_intermediates=True)
    assert all(np.array_equal(got[o], want[o]) for o in outs)


@pytest.mark.parametrize("h,w", [(4, 5), (17, 19), (45, 40)])  # planes of both kernels, the largest past shared memory
@pytest.mark.parametrize("mode,plain", [("reflect", True), ("edge", False), ("constant", True)])
def test_normalisation_adds_the_residual_and_pads(h, w, mode, plain):
    n, c = 2, 40 if plain else 42
    rng = np.random.default_rng([h, w, len(mode)])
    weights = {"g": (rng.standard_normal((16, 2 * c)) * 0.3).astype(np.float32), "s0": np.float32([0]), "s1": np.float32([c]), "s2": np.float32([2 * c]),
               "ax": np.float32([1]), "shape": np.float32([n, c, 1, 1]), "pads": np.float32([0, 0, 1, 2, 0, 0, 3, 0]), "fill": np.float32([0.5])}
    nodes = [Node("MatMul", "mm", ["l", "g"], ["style"], {}), Node("Slice", "sa", ["style", "s0", "s1", "ax"], ["a"], {}),
             Node("Slice", "sb", ["style", "s1", "s2", "ax"], ["b"], {}), Node("Reshape", "ra", ["a", "shape"], ["a4"], {}),
             Node("Reshape", "rb", ["b", "shape"], ["b4"], {}), Node("Relu", "rx", ["x"], ["x1"], {}),
             Node("MaxPool", "rr", ["x1"], ["r1"], {"kernel_shape": [3, 3], "strides": [1, 1], "pads": [1] * 4}),
             Node("OxiInstanceNorm", "in", ["r1"], ["xn"], {"epsilon": 1e-5}),
             Node("Mul", "mul", ["xn", "a4"], ["xm"], {}), Node("Add", "add", ["xm", "b4"], ["xa"], {}), Node("Add", "res", ["xa", "r1"], ["xr"], {}),
             Node("Pad", "pad", ["xr", "pads", "fill"] if mode == "constant" else ["xr", "pads"], ["y"], {"mode": mode})]
    outs = ["y"]
    if plain:
        nodes.append(Node("Sigmoid", "sg", ["xr"], ["z"], {}))
        outs.append("z")
    graph = Graph(nodes=nodes, input_names=["x", "l"], output_names=outs)
    feeds = {"x": rng.standard_normal((n, c, h, w)).astype(np.float32), "l": rng.standard_normal((n, 16)).astype(np.float32)}
    got, kernels = _run(graph, weights, feeds)
    assert "instance_norm+adain+residual+pad" in kernels, kernels
    want, _ = _run(graph, weights, feeds, keep_intermediates=True)
    assert all(np.array_equal(got[o], want[o]) for o in outs)


# rows and the three products' widths: all small, the persistent kernel's, split K beside unsplit, one after the other's memory
@pytest.mark.parametrize("rows,k,widths", [(5, 256, (96, 512, 40)), (154, 768, (768, 768, 768)), (3000, 512, (512, 1024, 256)), (64, 2048, (64, 2048, 1000))])
@pytest.mark.parametrize("graph_replay", [False, True])
def test_products_that_run_side_by_side(rows, k, widths, graph_replay):
    rng = np.random.default_rng([rows, k, *widths])
    weights, nodes, outs = {}, [Node("DynamicQuantizeLinear", "q0", ["x"], ["xq", "xs", "xz"], {})], []
    for i, n in enumerate(widths):
        weights[f"w{i}"] = rng.integers(-127, 128, (k, n)).astype(np.float32)
        nodes.append(Node("MatMulInteger", f"mm{i}", ["xq", f"w{i}", "xz"], [f"acc{i}"], {}))
    for i, n in enumerate(widths):
        nodes.append(Node("Relu", f"r{i}", [f"acc{i}"], [f"y{i}"], {}))
        outs.append(f"y{i}")
    graph = Graph(nodes=nodes, input_names=["x"], output_names=outs)
    sess = Session.builder().with_cuda_graph(graph_replay).build_from_graph(graph, weights)
    ref = Session.builder().with_kernel_path("direct").build_from_graph(graph, weights)
    for _ in range(6):
        feeds = {"x": rng.standard_normal((rows, k)).astype(np.float32)}
        got, want = sess.run(feeds), ref.run(feeds)
        assert all(np.array_equal(got[o], want[o]) for o in outs)
    assert sum("umma_i8" in s["kernel"] for s in sess.steps()) == 3
    sess.close()
    ref.close()


# input channels, height, width, filters of the first convolution and of the shortcut: one slice each, unequal slices (four and
# one, eight and four), a last cluster with CTAs too many, ragged tiles
@pytest.mark.parametrize("c,h,w,oc1,oc2", [(64, 9, 7, 64, 256), (1024, 14, 14, 512, 2048), (1024, 14, 14, 512, 968), (2048, 5, 5, 40, 200)])
@pytest.mark.parametrize("kind", ["int8", "tf32", "bf16"])
def test_a_shortcut_beside_its_first_convolution(c, h, w, oc1, oc2, kind):
    rng = np.random.default_rng([c, h, oc1, oc2])
    conv, first, sc = {"strides": [2, 2]}, {"strides": [1, 1]}, {"strides": [2, 2]}
    feeds = {"x": rng.standard_normal((1, c, h, w)).astype(np.float32)}
    if kind == "int8":
        weights = {"s": np.float32([0.02]), "z": np.float32([128]), "z0": np.float32([0]), "j": np.float32([0.04])}
        nodes = [Node("QuantizeLinear", "q", ["x", "s", "z"], ["xq"], {})]
        for name, x, oc, k, attrs in (("c1", "xq", oc1, c, first), ("c2", "c1q", oc2, oc1, conv), ("sc", "xq", oc2, c, sc)):
            weights.update({name + "w": rng.integers(-127, 128, (oc, k, 1, 1)).astype(np.float32), name + "ws": rng.uniform(2e-4, 4e-4, oc).astype(np.float32),
                            name + "b": rng.integers(-1000, 1001, oc).astype(np.float32)})
            nodes.append(Node("QLinearConv", name, [x, "s", "z", name + "w", name + "ws", "z0", "s", "z", name + "b"], [name + "q"], attrs))
        nodes += [Node("DequantizeLinear", "d1", ["c2q", "s", "z"], ["a"], {}), Node("DequantizeLinear", "d2", ["scq", "s", "z"], ["b"], {}),
                  Node("Add", "add", ["a", "b"], ["sum"], {}), Node("Relu", "relu", ["sum"], ["r"], {}), Node("QuantizeLinear", "qj", ["r", "j", "z0"], ["yq"], {}),
                  Node("DequantizeLinear", "dq", ["yq", "j", "z0"], ["y"], {})]
        tuning, tol = {}, 0.0
    else:
        weights, nodes = {}, [Node("Relu", "pre", ["x"], ["x1"], {})]
        for name, x, oc, k, attrs in (("c1", "x1", oc1, c, dict(first, activation="relu")), ("c2", "c1y", oc2, oc1, conv), ("sc", "x1", oc2, c, sc)):
            weights.update({name + "w": (rng.standard_normal((oc, k, 1, 1)) / np.sqrt(k)).astype(np.float32), name + "b": rng.standard_normal(oc).astype(np.float32)})
            nodes.append(Node("Conv", name, [x, name + "w", name + "b"], [name + "y"], attrs))
        nodes += [Node("Add", "add", ["c2y", "scy"], ["sum"], {}), Node("Relu", "relu", ["sum"], ["y"], {})]
        # two products after one another, 11 (TF32) or 8 (bf16) significant bits each
        tuning, tol = {"float_precision": kind}, 4e-3 if kind == "tf32" else 4e-2
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["y"])
    got, kernels = _run(graph, weights, feeds, **tuning)
    beside = [s for s in kernels if "inside the launch of 'c1'" in s]
    assert len(beside) == 1 and ("im2col" in beside[0]), kernels
    want, _ = _run(graph, weights, feeds, kernel_path="direct")
    assert np.all(np.abs(got["y"] - want["y"]) <= tol * np.abs(want["y"]).max())


# storage of the convolution's lanes, of the residual and of the sum: zero points of every sign, with and without Relu
JOINS = {"unsigned relu": (("u8", 128, 0.07622), ("u8", 0, 0.04274), ("u8", 0, 0.05397), True),
         "signed residual": (("u8", 131, 0.05076), ("i8", -3, 0.05087), ("u8", 130, 0.07024), False),
         "signed": (("i8", -7, 0.07615), ("i8", 5, 0.08084), ("i8", -9, 0.06283), False),
         "signed sum relu": (("i8", 11, 0.04367), ("u8", 140, 0.0632), ("i8", -20, 0.04647), True),
         "narrow": (("u8", 3, 0.02), ("i8", 0, 0.9), ("i8", 100, 0.7), False)}  # many sums saturate
# batch, channels, height, width, filters, kernel, CTA pairs, what the kernel has to say: every kernel and staging depth that takes a join,
# ragged rows and channel tiles
JOIN_SHAPES = [(1, 64, 9, 7, 96, 1, "auto", "small"), (1, 512, 7, 7, 160, 1, "auto", "small"), (1, 128, 13, 11, 64, 3, "auto", "small"),
               (1, 64, 61, 43, 288, 1, "always", "cta-pair"), (1, 512, 61, 43, 544, 1, "always", "cta-pair"), (2, 64, 30, 31, 256, 3, "always", "cta-pair"),
               (1, 64, 139, 137, 256, 1, "never", "residual-buffers=4"), (1, 512, 137, 137, 384, 1, "never", "residual-buffers=3"),
               (1, 1024, 137, 137, 256, 1, "never", "residual-buffers=2"), (2, 64, 139, 137, 32, 3, "never", "residual-buffers"),
               # whole groups of 64 filters (the fragment epilogue) with a ragged last channel tile in a CTA pair, and 32 more than that (the
               # general epilogue) at every depth of the staging
               (1, 64, 61, 43, 320, 1, "always", "cta-pair fragments"), (1, 512, 61, 43, 448, 1, "always", "cta-pair fragments"),
               (1, 64, 139, 137, 288, 1, "never", "residual-buffers=4"), (1, 512, 137, 137, 352, 1, "never", "residual-buffers=3"),
               (1, 1024, 137, 137, 224, 1, "never", "residual-buffers=2")]


@pytest.mark.parametrize("shape", JOIN_SHAPES, ids=str)
@pytest.mark.parametrize("join", JOINS)
def test_quantised_joins_in_the_epilogue_are_the_separate_nodes(shape, join):
    n, c, h, w, oc, k, pairs, says = shape
    (a_st, a_z, a_s), (b_st, b_z, b_s), (y_st, y_z, y_s), relu = JOINS[join]
    rng = np.random.default_rng([n, c, h, oc, k])
    kinds = {"u8": np.uint8, "i8": np.int8}
    peak = min(127, (1 << 24) // (300 * c * k * k))  # accumulators that convert exactly
    weights = {"w": rng.integers(-peak, peak + 1, (oc, c, k, k)).astype(np.float32), "wz": np.int8([0]), "xs": np.float32([0.02]), "xz": np.uint8([121 if k == 1 else 0]),
               "bias": rng.integers(-1000, 1001, oc).astype(np.float32), "one": np.float32([1]), "rz": kinds[b_st]([128 if b_st == "u8" else 0]),
               "as": np.float32([a_s]), "az": kinds[a_st]([a_z]), "bs": np.float32([b_s]), "bz": kinds[b_st]([b_z]), "ys": np.float32([y_s]), "yz": kinds[y_st]([y_z])}
    # a standard deviation of about sixty lanes in front of the first saturation
    spread = 60 / (50 * peak / np.sqrt(3) * np.sqrt(c * k * k))
    weights["ws"] = (rng.uniform(0.7, 1.4, oc) * spread * a_s / 0.02).astype(np.float32)
    nodes = [Node("QuantizeLinear", "qx", ["x", "xs", "xz"], ["xq"], {}), Node("QuantizeLinear", "qr", ["r", "one", "rz"], ["rq"], {}),
             Node("QLinearConv", "conv", ["xq", "xs", "xz", "w", "ws", "wz", "as", "az", "bias"], ["aq"], {"pads": [k // 2] * 4}),
             Node("DequantizeLinear", "da", ["aq", "as", "az"], ["a"], {}), Node("DequantizeLinear", "db", ["rq", "bs", "bz"], ["b"], {}),
             Node("Add", "add", ["a", "b"], ["sum"], {})]
    if relu:
        nodes.append(Node("Relu", "relu", ["sum"], ["s"], {}))
    nodes += [Node("QuantizeLinear", "qy", ["s" if relu else "sum", "ys", "yz"], ["yq"], {}), Node("DequantizeLinear", "dy", ["yq", "ys", "yz"], ["y"], {})]
    graph = Graph(nodes=nodes, input_names=["x", "r"], output_names=["y"])
    feeds = {"x": rng.standard_normal((n, c, h, w)).astype(np.float32),
             "r": (rng.integers(0, 256, (n, oc, h, w)) - 128).astype(np.float32)}
    got, kernels = _run(graph, weights, feeds, cta_pairs=pairs)
    joined = [s for s in kernels if s.endswith("+join")]
    assert len(joined) == 1 and says in joined[0], kernels
    # the persistent kernel joins whole groups of 64 filters in its fragment epilogue, everything else in its general one
    assert ("fragments" in joined[0]) == (says != "small" and oc % 64 == 0), joined
    want, apart = _run(graph, weights, feeds, cta_pairs=pairs, keep_intermediates=True)
    assert not any("+join" in s for s in apart)
    assert np.array_equal(got["y"], want["y"])
    assert np.unique(want["y"]).size > 20  # not only the ends of the range


# a 1x1 filter whose outputs are a few more, or a few fewer, than 64 Mi: images, channels, filters, a Relu on the lane itself, joined or not
SHORT_JOINS = [(56, 64, 96, False, False), (55, 64, 96, False, True), (56, 32, 96, False, True), (84, 64, 64, False, True), (84, 64, 64, True, False), (83, 64, 64, True, True)]


@pytest.mark.parametrize("images, c, oc, lane_relu, joins", SHORT_JOINS)
def test_short_joins_past_l2_are_fused_where_the_fragments_take_them(images, c, oc, lane_relu, joins):
    rng = np.random.default_rng([images, oc])
    weights = {"xs": np.float32([0.02]), "xz": np.uint8([0]), "as": np.float32([0.07615]), "az": np.int8([0]), "bs": np.float32([0.08084]), "bz": np.int8([5]),
               "ys": np.float32([0.06283]), "yz": np.int8([-9]), "z0": np.float32([0])}
    nodes = [Node("QuantizeLinear", "qx", ["x", "xs", "xz"], ["xq"], {})]
    for name, scale, zp in (("b", "bs", "bz"), ("a", "as", "az")):
        weights[name + "w"] = rng.integers(-127, 128, (oc, c, 1, 1)).astype(np.float32)
        weights[name + "ws"] = (rng.uniform(0.7, 1.4, oc) * 0.003).astype(np.float32)
        weights[name + "bias"] = rng.integers(-1000, 1001, oc).astype(np.float32)
        nodes.append(Node("QLinearConv", "conv_" + name, ["xq", "xs", "xz", name + "w", name + "ws", "z0", scale, zp, name + "bias"], [name + "q"], {}))
    if lane_relu:
        nodes.append(Node("Relu", "lane", ["aq"], ["ar"], {}))
    nodes += [Node("DequantizeLinear", "da", ["ar" if lane_relu else "aq", "as", "az"], ["a"], {}), Node("DequantizeLinear", "db", ["bq", "bs", "bz"], ["b"], {}),
              Node("Add", "add", ["a", "b"], ["sum"], {}), Node("QuantizeLinear", "qy", ["sum", "ys", "yz"], ["yq"], {}),
              Node("DequantizeLinear", "dy", ["yq", "ys", "yz"], ["y"], {}), Node("GlobalAveragePool", "gap", ["y"], ["z"], {})]
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["z"])
    feeds = {"x": np.abs(rng.standard_normal((images, c, 112, 112), dtype=np.float32))}
    got, kernels = _run(graph, weights, feeds)
    assert any(s.endswith("+join") for s in kernels) == joins and any(s.startswith("residual_requant") for s in kernels) != joins, kernels
    want, _ = _run(graph, weights, feeds, keep_intermediates=True)
    assert np.array_equal(got["z"], want["z"])


def test_side_by_side_products_are_one_launch():
    rng = np.random.default_rng(5)
    weights, nodes, outs = {}, [Node("DynamicQuantizeLinear", "q0", ["x"], ["xq", "xs", "xz"], {})], []
    for i in range(5):  # more than one launch takes
        weights[f"w{i}"] = rng.integers(-127, 128, (256, 96)).astype(np.float32)
        nodes.append(Node("MatMulInteger", f"mm{i}", ["xq", f"w{i}", "xz"], [f"acc{i}"], {}))
    for i in range(5):
        nodes.append(Node("Relu", f"r{i}", [f"acc{i}"], [f"y{i}"], {}))
        outs.append(f"y{i}")
    sess = Session.builder().build_from_graph(Graph(nodes=nodes, input_names=["x"], output_names=outs), weights)
    feeds = {"x": rng.standard_normal((33, 256)).astype(np.float32)}
    sess.run(feeds)
    before = sess.cuda_cache_counters()["umma_launches"]
    sess.run(feeds)
    assert sess.cuda_cache_counters()["umma_launches"] - before == 2
    sess.close()


@pytest.mark.parametrize("channels,h,w,scale", [(128, 5, 7, 2.0), (132, 9, 33, 1.5), (320, 1, 70, 3.0)])
@pytest.mark.parametrize("coord", ["half_pixel", "align_corners", "asymmetric"])
def test_linear_resize_of_many_channels_is_the_one_of_few(channels, h, w, scale, coord):
    rng = np.random.default_rng([channels, h, w])
    weights = {"s": np.float32([1, 1, scale, scale])}
    nodes = [Node("Relu", "r", ["x"], ["x1"], {}), Node("Resize", "up", ["x1", "", "s"], ["y"], {"mode": "linear", "coordinate_transformation_mode": coord})]
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["y"])
    x = rng.standard_normal((2, channels, h, w)).astype(np.float32)
    got, _ = _run(graph, weights, {"x": x})
    for c in range(0, channels, 64):
        want, _ = _run(graph, weights, {"x": np.ascontiguousarray(x[:, c:c + 64])})
        assert np.array_equal(got["y"][:, c:c + 64], want["y"])
