"""Whole-graph parity on the B200 through the planned, device-resident session
(oxb200_session_plan + oxb200_run): the five benchmark topologies at sizes the CPU oracle
finishes in seconds, per node and end to end, plus size-independent properties at full size."""
import numpy as np
import pytest

import oracle
from oxionnx_b200 import models
from oxionnx_b200.session import Session

pytestmark = pytest.mark.gpu

RTOL = 2e-3


def close_tf32(got, want, scale=1.0):
    want = np.asarray(want, np.float32)
    atol = RTOL * scale * float(np.max(np.abs(want)))
    return bool(np.all(np.abs(got.astype(np.float64) - want) <= atol + RTOL * scale * np.abs(want)))


def run_both(graph, weights, feeds, **builder):
    b = Session.builder().with_keep_intermediates(True)
    if builder.get("kernel_path"):
        b = b.with_kernel_path(builder["kernel_path"])
    sess = b.build_from_graph(graph, weights)
    out = sess.run(feeds)
    oracle.set_threads(8)
    ref = oracle.run_graph(graph, weights, feeds)
    return sess, out, ref


@pytest.mark.parametrize("spelling", ["qlinearconv", "qlinearmatmul"])
@pytest.mark.parametrize("path", ["auto", "direct"])
def test_int8_mlp_small_bit_exact_per_node(spelling, path):
    graph, weights, feeds, _ = models.build_int8_mlp(rows=24, dims=(128, 256, 192, 64), spelling=spelling)
    sess, out, ref = run_both(graph, weights, feeds(), kernel_path=path)
    for name in ("q0", "q1", "q2", "q3", "y"):
        assert np.array_equal(sess.fetch_value(name), ref[name]), name
    assert np.array_equal(out["y"], ref["y"])
    sess.close()


def test_int8_mlp_full_size_bit_exact():
    """Config 1 at its real size: 64 x (1024 -> 4096 -> 4096 -> 1024)."""
    graph, weights, feeds, _ = models.build_int8_mlp()
    sess, out, ref = run_both(graph, weights, feeds())
    for name in ("q0", "q1", "q2", "q3"):
        assert np.array_equal(sess.fetch_value(name), ref[name]), name
    assert np.array_equal(out["y"], ref["y"])
    kernels = [s["kernel"] for s in sess.steps() if s["op"] == "QLinearConv"]
    assert all(k.startswith("umma_i8") for k in kernels), kernels
    sess.close()


@pytest.mark.parametrize("rows,dims", [(64, (256, 512, 384, 128)), (1, (128, 256, 200, 72)), (37, (512, 1024, 1024, 1024, 256)),
                                       (64, (128, 256, 256, 256, 256, 256, 128))])
def test_int8_mlp_chain_kernel_matches_oracle_and_separate_kernels(rows, dims):
    """Consecutive quantised linear layers over at most 64 rows run as one cooperative kernel (weights as the 128-row
    MMA operand, K slices summed by integer reductions, one grid barrier per layer).  Every layer's rows must equal the
    oracle's and those of the one-kernel-per-layer plan (split_k_max = 1 keeps the layers apart); channel counts that
    are not multiples of the 128-channel tile, a single row, a layer whose K keeps it out of the chain, and six layers
    (two chains) are covered;
    a replayed CUDA graph gives the same lanes."""
    graph, weights, feeds, _ = models.build_int8_mlp(rows=rows, dims=dims)
    sess, out, ref = run_both(graph, weights, feeds())
    names = [f"q{i}" for i in range(len(dims))]
    for name in names:
        assert np.array_equal(sess.fetch_value(name), ref[name]), name
    assert np.array_equal(out["y"], ref["y"])
    kernels = [s["kernel"] for s in sess.steps() if s["op"] == "QLinearConv"]
    assert kernels[0].startswith("umma_i8_chain rows="), kernels
    assert sum(k.startswith("umma_i8_chain rows=") for k in kernels) == (2 if len(dims) == 7 else 1), kernels
    launches_chain = sess.cuda_cache_counters()["umma_launches"]
    sess.close()
    apart = Session.builder().with_tuning(split_k_max=1).build_from_graph(graph, weights)
    got = apart.run(feeds())
    assert np.array_equal(got["y"], out["y"])
    assert not any("chain" in s["kernel"] for s in apart.steps())
    assert apart.cuda_cache_counters()["umma_launches"] > launches_chain
    apart.close()
    replay = Session.builder().with_cuda_graph().build_from_graph(graph, weights)
    for i in range(4):
        f = {"x": feeds()["x"] * (1.0 + 0.5 * i)}
        want = oracle.run_graph(graph, weights, f)["y"]
        assert np.array_equal(replay.run(f)["y"], want), i
    # without kept intermediates the QuantizeLinear in front of the chain and the DequantizeLinear behind it run inside it
    steps = replay.steps()
    fused = [s["kernel"] for s in steps if s["op"] in ("QuantizeLinear", "DequantizeLinear")]
    assert len(fused) == 2 and fused[0].startswith("umma_i8_chain (inside"), [(s["op"], s["kernel"]) for s in steps]
    chain_desc = [s["kernel"] for s in steps if s["kernel"].startswith("umma_i8_chain rows=")]
    assert "+quantize" in chain_desc[0], chain_desc
    if dims[-2] % 128 == 0:
        assert fused[1].startswith("umma_i8_chain (inside") and "+dequantize" in chain_desc[-1], (fused, chain_desc)
    replay.close()


def test_int8_mlp_chain_accumulators_beyond_24_bits_take_the_f64_requantisation():
    """The chain kernel requantises with one float FMA where the accumulator converts exactly (below 2^24) and with the
    reference's f64 operations elsewhere: all-127 weights over K = 2048 and saturated inputs give 127 * 127 * 2048 = 33 M."""
    rows, dims = 16, (2048, 256, 128)
    graph, weights, feeds, _ = models.build_int8_mlp(rows=rows, dims=dims)
    weights = dict(weights)
    weights["w0"] = np.full_like(weights["w0"], 127.0)
    weights["w0"][::3] = -127.0
    weights["w0_scale"] = np.full_like(weights["w0_scale"], 4e-6)
    x = feeds()["x"]
    x[:8] = 100.0   # saturates the input quantiser at 255
    x[8:12] = -100.0
    sess, out, ref = run_both(graph, weights, {"x": x})
    assert any("umma_i8_chain rows=" in s["kernel"] for s in sess.steps())
    q1 = sess.fetch_value("q1")
    assert np.array_equal(q1, ref["q1"]) and np.array_equal(out["y"], ref["y"])
    assert 0 < q1.min() and q1.max() < 255 and len(np.unique(q1)) > 2  # inside the range: the rounding itself is compared
    sess.close()


@pytest.mark.parametrize("rows,k,n,gelu", [(200, 256, 200, True), (128, 128, 96, False), (37, 384, 1000, True)])
def test_contraction_hands_its_extrema_to_the_next_dynamic_quantize_linear(rows, k, n, gelu):
    """A tensor-core contraction that writes f32 lanes merges their minimum and maximum into the keys of the
    DynamicQuantizeLinear that reads them, which then skips its own first pass.  Row counts that are not a multiple
    of the 128-row tile and channel counts that are not a multiple of the 32-channel run must not leak padding
    lanes into the extrema: scale, zero point and every quantised lane equal those of a session that keeps its
    intermediates (where nothing is handed over) and the oracle's."""
    from oxionnx_b200.graph import Graph, Node
    rng = np.random.default_rng(977 + rows)
    w = {"w": np.clip(np.rint(rng.standard_normal((k, n)) * 40.0), -127, 127).astype(np.float32),
         "ws": rng.uniform(0.0005, 0.002, n).astype(np.float32), "bias": (rng.standard_normal(n) * 0.5 + 0.8).astype(np.float32)}
    nodes = [Node("DynamicQuantizeLinear", "q0", ["x"], ["xq", "xs", "xz"], {}),
             Node("MatMulInteger", "mmi", ["xq", "w", "xz"], ["acc"], {}), Node("Cast", "cast", ["acc"], ["accf"], {"to": 1}),
             Node("Mul", "scales", ["xs", "ws"], ["sc"], {}), Node("Mul", "rescale", ["accf", "sc"], ["scaled"], {}),
             Node("Add", "addb", ["scaled", "bias"], ["lin"], {})]
    last = "lin"
    if gelu:
        nodes.append(Node("Gelu", "act", ["lin"], ["act_out"], {}))
        last = "act_out"
    nodes.append(Node("DynamicQuantizeLinear", "q1", [last], ["yq", "ys", "yz"], {}))
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["yq", "ys", "yz"])
    feeds = {"x": (rng.standard_normal((rows, k)) * 2 + 0.3).astype(np.float32)}
    handed = Session.builder().build_from_graph(graph, w)
    got = handed.run(feeds)
    kernels = {s["node"]: s["kernel"] for s in handed.steps()}
    assert "extrema from the producer" in kernels["q1"], kernels
    handed.close()
    kept = Session.builder().with_keep_intermediates(True).build_from_graph(graph, w)
    want = kept.run(feeds)
    assert "extrema from the producer" not in {s["node"]: s["kernel"] for s in kept.steps()}["q1"]
    kept.close()
    ref = oracle.run_graph(graph, w, feeds)
    for name in ("ys", "yz", "yq"):
        assert np.array_equal(np.ravel(got[name]), np.ravel(want[name])), name
    assert float(np.ravel(got["yz"])[0]) == float(np.ravel(ref["yz"])[0])
    assert np.isclose(float(np.ravel(got["ys"])[0]), float(np.ravel(ref["ys"])[0]), rtol=1e-6)
    assert np.max(np.abs(got["yq"].astype(np.int32) - ref["yq"].astype(np.int32))) <= 1  # the oracle's Gelu may differ in the last place


def _gelu_arguments(n):
    """n values for the exact Gelu: those around the end of a binade of its polynomial's denominator (1 + 0.3275911 |y| / sqrt 2
    = 2), the ends of the range, and a dense rest."""
    f = np.float32
    special = np.arange(f(4.3165).view(np.int32), f(4.3175).view(np.int32), dtype=np.int32).view(f)
    d = f(1) + special * f(0.70710678118654752440) * f(0.3275911)
    assert d[0] < 2 < d[-1]
    ends = np.float32([0.0, 1e-45, 1e-38, 1e-20, 1e-7, 14.3, 14.5, 18.0, 40.0, 1e10, 1e30, 3.4e38])
    rest = np.random.default_rng(8).uniform(0, 15, n // 2 - special.size - ends.size).astype(f)
    half = np.concatenate([special, ends, rest])
    return np.concatenate([half, -half])


@pytest.mark.parametrize("pairs", ["auto", "always"])  # the small-problem kernel, the persistent one
def test_gelu_in_the_epilogue_is_the_separate_node_at_its_hardest_arguments(pairs):
    """The bias carries the argument (every weight is zero), so each is met exactly."""
    from oxionnx_b200.graph import Graph, Node
    n, k = 30000, 64
    y = _gelu_arguments(n)
    w = {"w": np.zeros((k, n), np.float32), "ws": np.full(n, 0.01, np.float32), "bias": y}
    nodes = [Node("DynamicQuantizeLinear", "q0", ["x"], ["xq", "xs", "xz"], {}), Node("MatMulInteger", "mmi", ["xq", "w", "xz"], ["acc"], {}),
             Node("Cast", "cast", ["acc"], ["accf"], {"to": 1}), Node("Mul", "scales", ["xs", "ws"], ["sc"], {}),
             Node("Mul", "rescale", ["accf", "sc"], ["scaled"], {}), Node("Add", "addb", ["scaled", "bias"], ["lin"], {}),
             Node("Gelu", "act", ["lin"], ["y"], {}), Node("Relu", "keep", ["y"], ["r"], {}), Node("Sub", "neg", ["y", "r"], ["m"], {})]
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["r", "m"])
    feeds = {"x": np.random.default_rng(9).standard_normal((2, k)).astype(np.float32)}
    fused = Session.builder().with_tuning(cta_pairs=pairs).build_from_graph(graph, w)
    got = fused.run(feeds)
    kernels = [s["kernel"] for s in fused.steps()]
    assert any(s.startswith("umma_i8") and "+dequant" in s and ("small" in s) == (pairs == "auto") for s in kernels), kernels
    fused.close()
    apart = Session.builder().with_keep_intermediates(True).build_from_graph(graph, w)
    want = apart.run(feeds)
    assert np.array_equal(apart.fetch_value("lin")[1], y)
    apart.close()
    for name in ("r", "m"):
        assert np.array_equal(got[name], want[name])


@pytest.mark.parametrize("shape", [(5, 37, 768), (64, 96), (3, 130, 1024)])
def test_layer_norm_absorbs_the_residual_add_in_front_of_it(shape):
    """Add -> LayerNormalization with the sum read by nothing else is one kernel (the sum is never written); the
    lanes are those of the two separate kernels bit for bit (one rounded sum per lane, then the same arithmetic)."""
    from oxionnx_b200.graph import Graph, Node
    rng = np.random.default_rng(41 + shape[-1])
    w = {"g": rng.uniform(0.5, 1.5, shape[-1]).astype(np.float32), "b": rng.standard_normal(shape[-1]).astype(np.float32)}
    nodes = [Node("Add", "res", ["x", "y"], ["sum"], {}), Node("LayerNormalization", "ln", ["sum", "g", "b"], ["out"], {"axis": -1, "epsilon": 1e-12}),
             Node("Mul", "use_y", ["y", "out"], ["out2"], {})]
    graph = Graph(nodes=nodes, input_names=["x", "y"], output_names=["out", "out2"])
    feeds = {"x": (rng.standard_normal(shape) * 3).astype(np.float32), "y": (rng.standard_normal(shape) + 0.5).astype(np.float32)}
    fused = Session.builder().build_from_graph(graph, w)
    got = fused.run(feeds)
    kernels = [s["kernel"] for s in fused.steps()]
    assert "add+layer_norm_rows" in kernels and kernels.count("binary") == 1, kernels  # the Mul stays; the Add is gone
    fused.close()
    apart = Session.builder().with_keep_intermediates(True).build_from_graph(graph, w)
    want = apart.run(feeds)
    assert "layer_norm_rows" in [s["kernel"] for s in apart.steps()]
    apart.close()
    assert np.array_equal(got["out"], want["out"]) and np.array_equal(got["out2"], want["out2"])
    ref = oracle.run_graph(graph, w, feeds)
    assert np.max(np.abs(got["out"] - ref["out"])) <= 1e-4


def test_resnet_f32_small_per_node_and_final():
    graph, weights, feeds, _ = models.build_resnet50_f32(batch=3, image=64, base=16, classes=40)
    sess, out, ref = run_both(graph, weights, feeds(3))
    # teacher-free run: per-node error stays inside the TF32 tolerance relative to the tensor's magnitude
    worst = 0.0
    for node in graph.nodes:
        name = node.outputs[0]
        if not sess.has_value(name):
            continue  # fused into its producer
        got, want = sess.fetch_value(name), ref[name]
        assert got.shape == want.shape, name
        err = float(np.max(np.abs(got - want)) / (np.max(np.abs(want)) + 1e-30))
        worst = max(worst, err)
        assert err <= 2.5 * RTOL, f"{name}: relative-to-max error {err}"
    assert close_tf32(out["logits"], ref["logits"], scale=2.5), worst
    used = {s["kernel"].split()[0] for s in sess.steps()}
    assert any(k.startswith("umma_tf32") for k in used), used
    sess.close()


def test_resnet_f32_arena_reuse_matches_private_slots():
    graph, weights, feeds, _ = models.build_resnet50_f32(batch=2, image=64, base=16, classes=40)
    f = feeds(2)
    a = Session.builder().with_keep_intermediates(True).build_from_graph(graph, weights)
    b = Session.builder().build_from_graph(graph, weights)
    ya, yb = a.run(f)["logits"], b.run(f)["logits"]
    assert np.array_equal(ya, yb)
    ca, cb = a.cuda_cache_counters(), b.cuda_cache_counters()
    assert cb["arena_bytes"] < ca["arena_bytes"] and cb["arena_slots"] < ca["arena_slots"]
    # without the per-node copies the residual Add (+Relu) of every block runs inside a convolution's epilogue,
    # with the same two roundings: the logits above are bit-identical to the node-by-node session's
    kb = [s["kernel"] for s in b.steps()]
    assert sum(k.endswith("+residual") for k in kb) == 16 and not any(k.startswith("binary") for k in kb), kb
    assert sum(s["kernel"].startswith("binary") for s in a.steps()) == 16
    # a second run re-uploads activations only: weights stay resident, one fence per run
    before = b.cuda_cache_counters()
    yb2 = b.run(f)["logits"]
    after = b.cuda_cache_counters()
    assert np.array_equal(yb, yb2)
    assert after["weight_uploads"] == before["weight_uploads"]
    assert after["uploads"] - before["uploads"] == 1 and after["downloads"] - before["downloads"] == 1
    assert after["fences"] - before["fences"] == 1
    a.close()
    b.close()


@pytest.mark.parametrize("path", ["auto", "direct"])
def test_resnet_qlinear_small_bit_exact_per_node(path):
    graph, weights, feeds, _ = models.build_resnet50_qlinear(batch=3, image=64, base=32, classes=48)
    sess, out, ref = run_both(graph, weights, feeds(3), kernel_path=path)
    checked = 0
    for node in graph.nodes:
        name = node.outputs[0]
        if not sess.has_value(name):
            continue
        got, want = sess.fetch_value(name), ref[name]
        assert np.array_equal(got, want), f"{node.op} {name}: {np.sum(got != want)} of {want.size} lanes differ"
        checked += 1
    assert checked > 60
    assert np.array_equal(out["logits"], ref["logits"])
    if path == "auto":
        fams = [s["kernel"].split()[0] for s in sess.steps() if s["op"] == "QLinearConv"]
        assert sum(k.startswith("umma_i8") for k in fams) >= len(fams) - 1, fams  # all but the 3-channel stem
    sess.close()


def test_resnet_qlinear_fused_session_equals_the_oracle_bit_for_bit():
    """The session a user gets (no per-node copies): QuantizeLinear inside the stem packing, the residual chains as
    one kernel each, DequantizeLinear inside GlobalAveragePool; the logits must still be the oracle's, lane for lane."""
    graph, weights, feeds, _ = models.build_resnet50_qlinear(batch=3, image=64, base=32, classes=48)
    sess = Session.builder().build_from_graph(graph, weights)
    f = feeds(3)
    out = sess.run(f)
    oracle.set_threads(8)
    ref = oracle.run_graph(graph, weights, f)
    assert np.array_equal(out["logits"], ref["logits"])
    kernels = [s["kernel"] for s in sess.steps()]
    assert "dequantize+global_avg_pool" in kernels and "quantize+s2d_window_pack" in kernels, kernels
    assert not any(k == "global_avg_pool" for k in kernels)
    sess.close()


def test_full_size_properties_resnet_qlinear():
    """At the benchmark's per-image size the oracle is too slow for a full comparison, so the
    run is pinned through size-independent properties: the tensor-core path and the direct
    path agree bit for bit on every value, and batch sharding is exact (each image's logits
    do not depend on its neighbours)."""
    graph, weights, feeds, _ = models.build_resnet50_qlinear(batch=4, image=224)
    f = feeds(4)
    a = Session.builder().build_from_graph(graph, weights)
    ya = a.run(f)["logits"]
    one = a.run({"input": f["input"][1:2]})["logits"]
    assert np.array_equal(one[0], ya[1])
    a.close()
    b = Session.builder().with_kernel_path("direct").build_from_graph(graph, weights)
    yb = b.run({"input": f["input"][:2]})["logits"]
    assert np.array_equal(yb, ya[:2])
    b.close()
    assert np.unique(ya).size > 100


RESIDUAL_SETS = [
    # a storage, a (scale, zp), b storage, b (scale, zp), y (scale, zp or None), relu
    ("u8", (0.02, 0), "u8", (0.05, 0), (0.02, 0), True),           # the ResNet blocks
    ("u8", (0.031, 128), "i8", (0.0173, -3), (0.043, 131), False),  # mixed storage, odd scales, no Relu
    ("i8", (0.5, 0), "i8", (0.25, 5), (0.125, -7), True),           # powers of two: every quotient is exact, many ties
    ("u8", (3.1e-7, 7), "u8", (2.9e-7, 0), (4.4e-7, None), False),  # scales outside the proven range: general kernel
]


@pytest.mark.parametrize("case", RESIDUAL_SETS, ids=[str(i) for i in range(len(RESIDUAL_SETS))])
def test_residual_requantisation_chain_bit_exact(case):
    """DequantizeLinear x2 -> Add -> [Relu] -> QuantizeLinear is planned as one kernel; its
    division-free form is used only for parameter sets proven pair by pair on the host.  Both
    forms must reproduce the node-by-node reference (oxionnx-ops src/indexing/quantize.rs)."""
    from oxionnx_b200.graph import Graph, Node
    a_st, (a_s, a_z), b_st, (b_s, b_z), (y_s, y_z), relu = case
    rng = np.random.default_rng(5)
    shape = (2, 48, 9, 7)
    rng_of = {"u8": (0, 256), "i8": (-128, 128)}
    a = rng.integers(*rng_of[a_st], shape).astype(np.float32)
    b = rng.integers(*rng_of[b_st], shape).astype(np.float32)
    # every pair of lanes at least once
    grid = np.stack(np.meshgrid(np.arange(*rng_of[a_st]), np.arange(*rng_of[b_st]), indexing="ij"), 0).astype(np.float32)
    weights = {"as": np.float32([a_s]), "az": np.float32([a_z]), "bs": np.float32([b_s]), "bz": np.float32([b_z]), "ys": np.float32([y_s]),
               "one": np.float32([1.0])}
    q_in = ["r", "ys"]
    if y_z is not None:
        weights["yz"] = np.float32([y_z])
        q_in.append("yz")
    # the operands reach the chain as 8-bit device tensors: quantise them with scale 1 first
    weights["azq"] = np.float32([128 if a_st == "u8" else 0])
    weights["bzq"] = np.float32([128 if b_st == "u8" else 0])
    nodes = [Node("QuantizeLinear", "qa", ["a", "one", "azq"], ["aq"], {}), Node("QuantizeLinear", "qb", ["b", "one", "bzq"], ["bq"], {}),
             Node("DequantizeLinear", "da", ["aq", "as", "az"], ["af"], {}), Node("DequantizeLinear", "db", ["bq", "bs", "bz"], ["bf"], {}),
             Node("Add", "add", ["af", "bf"], ["s"], {})]
    if relu:
        nodes.append(Node("Relu", "relu", ["s"], ["r"], {}))
    else:
        q_in[0] = "s"
    nodes += [Node("QuantizeLinear", "q", q_in, ["yq"], {}), Node("DequantizeLinear", "dq", ["yq", "ys"] + (["yz"] if y_z is not None else []), ["y"], {})]
    graph = Graph(nodes=nodes, input_names=["a", "b"], output_names=["y"])
    off_a, off_b = weights["azq"][0], weights["bzq"][0]
    for feeds in ({"a": a - off_a, "b": b - off_b}, {"a": grid[0].reshape(1, 256, 16, 16) - off_a, "b": grid[1].reshape(1, 256, 16, 16) - off_b}):
        sess, out, ref = run_both(graph, weights, feeds)
        assert any(s["kernel"].startswith("residual_requant") for s in sess.steps()), [s["kernel"] for s in sess.steps()]
        assert np.array_equal(sess.fetch_value("yq"), ref["yq"]), f"{np.sum(sess.fetch_value('yq') != ref['yq'])} lanes differ"
        assert np.array_equal(out["y"], ref["y"])
        sess.close()


def test_inswapper_f32_small_per_node_and_final():
    """Config 3 at reduced width: reflect Pad, pad-free 3x3 convolutions, OxiInstanceNorm with per-sample
    Mul/Add modulation from Gemm + Slice heads, residual joins, Resize x2 decoder, 7x7 + Tanh."""
    graph, weights, feeds, _ = models.build_inswapper_f32(batch=3, size=32, widths=(32, 64, 96, 128), blocks=2, latent=64)
    sess, out, ref = run_both(graph, weights, feeds(3))
    for node in graph.nodes:
        name = node.outputs[0]
        if not sess.has_value(name):
            continue
        got, want = sess.fetch_value(name), ref[name]
        assert got.shape == want.shape, name
        err = float(np.max(np.abs(got - want)) / (np.max(np.abs(want)) + 1e-30))
        # teacher-free drift: TF32 rounding of every layer before it compounds, and each instance normalisation
        # rescales it; the bound is 2.5x the per-operator tolerance inside the network and 5x (1e-2 of the
        # tensor's magnitude) behind the last, heavily cancelling 7x7 convolution
        bound = (5.0 if name in ("out_conv_out", "image") else 2.5) * RTOL
        assert err <= bound, f"{name}: relative-to-max error {err}"
    assert close_tf32(out["image"], ref["image"], scale=5.0)
    kernels = [s["kernel"] for s in sess.steps()]
    assert any(k.startswith("umma_tf32") for k in kernels) and any(k.startswith("instance_norm") for k in kernels), kernels
    sess.close()
    # the planned-for-speed session (no per-node copies, residual joins inside the convolutions) gives the same image
    fast = Session.builder().build_from_graph(graph, weights)
    assert close_tf32(fast.run(feeds(3))["image"], ref["image"], scale=5.0)
    fast.close()


def test_bert_dynamic_int8_small_per_node_and_teacher_forced():
    """Config 4 at reduced size.  Float nodes: relative-to-max error within the float tolerance, teacher-free.
    A dynamically quantised tensor may differ from the oracle's by one step in a few lanes when its f32 input
    differs in the last bits, so the integer nodes are checked teacher-forced: fed the oracle's own inputs
    through the operator boundary they must match bit for bit."""
    from oxionnx_b200.graph import Node
    from oxionnx_b200 import session as S
    graph, weights, feeds, _ = models.build_bert_dynamic_int8(batch=3, seq=32, hidden=128, heads=4, ffn=256, layers=2, vocab=500)
    f = feeds(3)
    sess, out, ref = run_both(graph, weights, f)
    worst = {}
    for node in graph.nodes:
        for name in node.outputs:
            if not sess.has_value(name):
                continue
            got, want = sess.fetch_value(name), ref[name]
            assert got.shape == want.shape, name
            if node.op == "DynamicQuantizeLinear":
                # teacher-free, the lanes themselves are not comparable (a zero point that rounds the other way moves
                # every lane by one): compare what they stand for, (q - zp) * scale, once per node
                if name.endswith("_q"):
                    stem = name[:-2]
                    dq_got = (got - sess.fetch_value(stem + "_z")) * sess.fetch_value(stem + "_s")
                    dq_want = (want - ref[stem + "_z"]) * ref[stem + "_s"]
                    assert float(np.max(np.abs(dq_got - dq_want)) / np.max(np.abs(dq_want))) <= 5e-2, name
                continue
            err = float(np.max(np.abs(got - want)) / (np.max(np.abs(want)) + 1e-30))
            worst[node.op] = max(worst.get(node.op, 0.0), err)
            # teacher-free drift: a requantisation point turns a last-bit difference into a whole step, and the softmax
            # turns an absolute error of the TF32 attention logits into a relative error of the probabilities; 5e-2 of
            # the tensor's magnitude inside the network, the same on the final hidden state (every dynamically quantised linear
            # re-amplifies any float difference to its own quantisation-noise level, about half a per cent of the range)
            assert err <= 5e-2, f"{name} ({node.op}): relative-to-max error {err}"
    assert float(np.max(np.abs(out["hidden"] - ref["hidden"])) / np.max(np.abs(ref["hidden"]))) <= 5e-2, worst
    kernels = {s["kernel"].split()[0] for s in sess.steps()}
    assert {"umma_i8", "layer_norm_rows", "softmax_rows", "gather_rows", "transpose_perm"} <= kernels, kernels
    # the planned-for-speed session runs Cast, both Mul, Add (and Gelu) of every linear inside the contraction's
    # epilogue with the same roundings: its hidden state is bit-identical to the node-by-node session's
    fast = Session.builder().build_from_graph(graph, weights)
    hidden_fast = fast.run(f)["hidden"]
    fused = [s["kernel"] for s in fast.steps()]
    assert sum(k.endswith("+dequant") for k in fused) == 12 and not any(k.startswith("cast") for k in fused), fused
    assert sum(k == "softmax_rows+scale+mask" for k in fused) == 2, fused
    # a DynamicQuantizeLinear behind a LayerNormalization takes its extrema from that kernel (one pass saved)
    assert sum(k.startswith("dynamic_quantize_linear (extrema") for k in fused) >= 2, fused
    assert np.array_equal(hidden_fast, out["hidden"])
    fast.close()
    sess.close()
    # teacher-forced: every integer node on the oracle's inputs, bit-exact
    ctx = S.CudaContext(0)
    for node in graph.nodes:
        if node.op not in ("DynamicQuantizeLinear", "MatMulInteger"):
            continue
        inter = {n: (weights[n] if n in weights else ref[n]) for n in node.inputs}
        got = S.try_cuda_dispatch(Node(node.op, node.name, node.inputs, node.outputs, node.attrs), {}, inter, ctx)
        assert got is not None, ctx.last_error()
        for g_, name in zip(got, node.outputs):
            assert np.array_equal(g_, ref[name]), f"{node.name}: {name} differs on the oracle's own inputs"
    ctx.close()


def test_bert_attention_on_the_tensor_cores():
    """With 128-token sequences the two attention products run as batched TF32 tensor-core products that read the
    heads of Q, K and V straight out of the [tokens, hidden] outputs of their linears (no head-split transposes for
    Q and K, one for V) and write the context back in that layout."""
    graph, weights, feeds, _ = models.build_bert_dynamic_int8(batch=2, seq=128, hidden=64, heads=2, ffn=128, layers=2, vocab=300)
    f = feeds(2)
    oracle.set_threads(8)
    ref = oracle.run_graph(graph, weights, f)
    fast = Session.builder().build_from_graph(graph, weights)
    hidden = fast.run(f)["hidden"]
    kernels = [s["kernel"] for s in fast.steps()]
    assert sum(k.startswith("umma_tf32 batched") for k in kernels) == 4, kernels
    assert sum(k.startswith("transpose_perm") for k in kernels) == 2 and not any(k.startswith("matmul_f32_direct") for k in kernels), kernels
    rel = lambda a, b: float(np.max(np.abs(a - b)) / np.max(np.abs(b)))
    assert rel(hidden, ref["hidden"]) <= 5e-2
    slow = Session.builder().with_keep_intermediates(True).build_from_graph(graph, weights)
    assert rel(slow.run(f)["hidden"], hidden) <= 5e-2
    for name in ("l0_scores", "l0_probs", "l0_ctx"):
        got, want = slow.fetch_value(name), ref[name]
        assert float(np.max(np.abs(got - want)) / np.max(np.abs(want))) <= 1e-2, name
    fast.close()
    slow.close()


def _round_tf32(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x1000) & 0xFFFFE000).astype(np.uint32).view(np.float32)  # round to nearest, ties away, as cvt.rna


@pytest.mark.parametrize("batch,heads,merge,masked", [(3, 2, True, True), (2, 5, False, True), (1, 3, True, False)])
def test_attention_scores_softmax_and_context_in_one_kernel(batch, heads, merge, masked):
    """MatMul(Q, K^T) -> Mul(scale) -> Add(mask) -> Softmax -> MatMul(., V) [-> head merge] over 128 positions and heads of
    64 lanes is one tensor-core kernel whose scores and probabilities stay on the SM.  Its context equals that of the
    separate kernels (a session that keeps intermediates runs those) to within what one TF32 rounding of a probability
    can move, and the oracle's within the TF32 tolerance; rows that are masked out carry no weight."""
    from oxionnx_b200.graph import Graph, Node
    S_, D = 128, 64
    rng = np.random.default_rng(5 + batch * 10 + heads)
    hd = heads * D
    w = {"heads_shape": np.float32([batch, S_, heads, D]), "rows_shape": np.float32([batch * S_, hd]), "att_scale": np.float32([1.0 / 8.0])}
    nodes = []
    def split(name, perm):
        nodes.append(Node("Reshape", f"{name}_split", [name, "heads_shape"], [f"{name}4r"], {}))
        nodes.append(Node("Transpose", f"{name}_t", [f"{name}4r"], [f"{name}4"], {"perm": perm}))
        return f"{name}4"
    # a projection in front of each operand makes it a device value, as in an encoder layer
    for name in ("q", "k", "v"):
        w[f"{name}_w"] = _round_tf32(rng.standard_normal((hd, hd)) / np.sqrt(hd))
        nodes.append(Node("MatMul", f"{name}_proj", [f"{name}_in", f"{name}_w"], [name], {}))
    q4, k4, v4 = split("q", [0, 2, 1, 3]), split("k", [0, 2, 3, 1]), split("v", [0, 2, 1, 3])
    nodes.append(Node("MatMul", "qk", [q4, k4], ["scores"], {}))
    nodes.append(Node("Mul", "scale", ["scores", "att_scale"], ["scaled"], {}))
    nodes.append(Node("Add", "mask_add", ["scaled", "mask"], ["masked"], {}))
    nodes.append(Node("Softmax", "softmax", ["masked"], ["probs"], {"axis": -1}))
    nodes.append(Node("MatMul", "av", ["probs", v4], ["ctx4"], {}))
    out = "ctx4"
    if merge:
        nodes.append(Node("Transpose", "merge_t", ["ctx4"], ["ctx_t"], {"perm": [0, 2, 1, 3]}))
        nodes.append(Node("Reshape", "merge", ["ctx_t", "rows_shape"], ["ctx"], {}))
        out = "ctx"
    graph = Graph(nodes=nodes, input_names=["q_in", "k_in", "v_in", "mask"], output_names=[out])
    mask = np.zeros((batch, 1, 1, S_), np.float32)
    if masked:
        mask[0, :, :, 100:] = -10000.0
        mask[-1, :, :, ::3] = -10000.0
    feeds = {n: _round_tf32(rng.standard_normal((batch * S_, hd)) * 1.5) for n in ("q_in", "k_in", "v_in")}
    feeds["mask"] = mask
    fused = Session.builder().build_from_graph(graph, w)
    got = fused.run(feeds)[out]
    kernels = [s["kernel"] for s in fused.steps()]
    assert sum(k.startswith("umma_attention") for k in kernels) == 1 and not any(k.startswith("softmax_rows") or "batched" in k for k in kernels), kernels
    fused.close()
    apart = Session.builder().with_keep_intermediates(True).build_from_graph(graph, w)
    want = apart.run(feeds)[out]
    assert not any(s["kernel"].startswith("umma_attention") for s in apart.steps())
    apart.close()
    ref = oracle.run_graph(graph, w, feeds)[out]
    top = float(np.max(np.abs(ref)))
    assert got.shape == ref.shape
    assert float(np.max(np.abs(got - want))) <= 1e-3 * top, float(np.max(np.abs(got - want))) / top
    assert float(np.max(np.abs(got - ref))) <= 4e-3 * top, float(np.max(np.abs(got - ref))) / top


def test_pipelined_runs_match_synchronous_runs():
    """oxb200_run_submit / oxb200_run_collect: three different batches with two in flight give, in order, exactly
    what the synchronous call gives for each; the same when the input's address is built into a tensor map (one
    input buffer, no overlap) and when a caller mixes both forms."""
    graph, weights, feeds, _ = models.build_resnet50_qlinear(batch=2, image=32, base=8, classes=10)
    sess = Session.builder().build_from_graph(graph, weights)
    batches = [feeds(2, f"pipe{i}") for i in range(3)]
    want = [sess.run(b)["logits"].copy() for b in batches]
    got = sess.run_pipelined(batches)
    for g_, w_ in zip(got, want):
        assert np.array_equal(g_["logits"], w_)
    assert np.array_equal(sess.run(batches[1])["logits"], want[1])
    assert not np.array_equal(want[0], want[1])
    sess.close()
    # a float GEMM straight on the graph input: the tensor map holds the input's address
    g2, w2, f2, _ = models.build_int8_mlp(rows=64, dims=(256, 512, 512, 128))
    s2 = Session.builder().build_from_graph(g2, w2)
    b2 = [{"x": f2()["x"] * (1.0 + 0.25 * i)} for i in range(3)]
    want2 = [s2.run(b)["y"].copy() for b in b2]
    for g_, w_ in zip(s2.run_pipelined(b2), want2):
        assert np.array_equal(g_["y"], w_)
    s2.close()


def test_cuda_graph_replay_is_bit_identical_and_counted():
    """OXIONNX_CUDA_GRAPH (oxionnx-cuda src/graph_cache.rs; tests/graph_cache_gpu.rs checks replays bit for bit):
    the first run on a set of input addresses launches the ordinary way, the second records, later ones replay;
    every run gives exactly the lanes of a session without graphs; launch counters advance as if each step had
    been launched; pipelined runs record one graph per input buffer; with shadow verification on nothing is
    recorded."""
    graph, weights, feeds, _ = models.build_resnet50_qlinear(batch=2, image=32, base=8, classes=10)
    batches = [feeds(2, f"graph{i}") for i in range(4)]
    plain = Session.builder().build_from_graph(graph, weights)
    want = [plain.run(b)["logits"].copy() for b in batches]
    per_run = plain.cuda_cache_counters()["kernel_launches"] // len(batches)
    plain.close()

    sess = Session.builder().with_cuda_graph().build_from_graph(graph, weights)
    for b, w in zip(batches, want):
        assert np.array_equal(sess.run(b)["logits"], w)
    c = sess.cuda_cache_counters()
    assert (c["graph_captures"], c["graph_replays"], c["graph_poisoned"]) == (1, 3, 0)
    assert c["kernel_launches"] == per_run * len(batches)
    for g_, w_ in zip(sess.run_pipelined(batches), want):
        assert np.array_equal(g_["logits"], w_)
    c = sess.cuda_cache_counters()
    assert c["graph_poisoned"] == 0 and c["graph_captures"] in (1, 2) and c["graph_replays"] >= 5
    sess.upload(batches[2])
    sess.run_resident(3)
    assert np.array_equal(sess.download()["logits"], want[2])
    sess.close()

    # float graph with tensor-core steps launched as programmatic dependents
    g2, w2, f2, _ = models.build_resnet50_f32(batch=2, image=32, base=16, classes=10)
    feeds2 = f2(2, "graph-f32")
    s_plain = Session.builder().build_from_graph(g2, w2)
    want2 = s_plain.run(feeds2)["logits"].copy()
    s_plain.close()
    s_graph = Session.builder().with_cuda_graph().build_from_graph(g2, w2)
    for _ in range(4):
        assert np.array_equal(s_graph.run(feeds2)["logits"], want2)
    assert s_graph.cuda_cache_counters()["graph_replays"] == 3
    s_graph.close()

    verified = Session.builder().with_cuda_graph().with_verify().build_from_graph(graph, weights)
    for b, w in zip(batches, want):
        assert np.array_equal(verified.run(b)["logits"], w)
    c = verified.cuda_cache_counters()
    assert (c["graph_captures"], c["graph_replays"]) == (0, 0)
    verified.close()


def test_split_k_is_used_and_agrees_with_the_unsplit_kernel():
    """Layers with few output tiles and a long K run as several K slices per tile that meet in a workspace.  The
    integer form must equal the unsplit kernel bit for bit; the float form adds the slices in a fixed order, so
    it is reproducible run to run and agrees with the unsplit kernel within the TF32 tolerance."""
    from oxionnx_b200.graph import Graph, Node
    rng = np.random.default_rng(77)
    wq = {"w": rng.integers(-127, 128, (256, 1024, 3, 3)).astype(np.float32), "ws": rng.uniform(0.001, 0.01, 256).astype(np.float32),
          "wz": np.zeros(256, np.float32), "b": rng.integers(-1000, 1000, 256).astype(np.float32), "xs": np.float32([0.02]), "z0": np.float32([0]),
          "z128": np.float32([128]), "ys": np.float32([2.0]), "qs": np.float32([0.02])}
    gq = Graph(nodes=[Node("QuantizeLinear", "q", ["x", "qs", "z0"], ["xq"], {}),
                      Node("QLinearConv", "conv", ["xq", "xs", "z0", "w", "ws", "wz", "ys", "z128", "b"], ["yq"], {"pads": [1, 1, 1, 1]}),
                      Node("DequantizeLinear", "dq", ["yq", "ys", "z128"], ["y"], {})], input_names=["x"], output_names=["y"])
    xq = np.abs(rng.standard_normal((2, 1024, 7, 7))).astype(np.float32)
    wf = {"w": (rng.standard_normal((512, 256, 3, 3)) * 0.02).astype(np.float32), "b": rng.standard_normal(512).astype(np.float32)}
    gf = Graph(nodes=[Node("Relu", "pre", ["x"], ["x1"], {}), Node("Conv", "conv", ["x1", "w", "b"], ["y"], {"pads": [1, 1, 1, 1], "activation": "relu"})],
               input_names=["x"], output_names=["y"])
    xf = rng.standard_normal((2, 256, 7, 7)).astype(np.float32)
    results = {}
    for mode in ("split", "unsplit"):
        for name, graph, weights, x in (("int8", gq, wq, xq), ("f32", gf, wf, xf)):
            sess = Session.builder().with_tuning(split_k_max=8 if mode == "split" else 1).build_from_graph(graph, weights)
            first = sess.run({"x": x})["y"].copy()
            again = sess.run({"x": x})["y"].copy()
            assert np.array_equal(first, again), "a split-K sum must not depend on the arrival order"
            kernel = [s_["kernel"] for s_ in sess.steps() if s_["node"] == "conv" and s_["kernel"].startswith("umma")][0]
            assert ("splitK" in kernel) == (mode == "split"), kernel
            results[(mode, name)] = first
            sess.close()
    assert np.array_equal(results[("split", "int8")], results[("unsplit", "int8")])
    assert np.unique(results[("split", "int8")]).size > 8
    assert close_tf32(results[("split", "f32")], results[("unsplit", "f32")])
