"""The fragment epilogues of the persistent integer kernel (csrc/umma_epilogue8.cuh): every tile width, ragged rows and
channel tiles, weights in the ring and resident, every bound of the saturation, activations with a zero point and without.
The same layers through the general epilogue, or their nodes one by one, are the reference.  Joins with a residual are covered
by test_quantised_joins_in_the_epilogue_are_the_separate_nodes, which says for each which epilogue it takes."""
import numpy as np
import pytest

from oxionnx_b200.graph import Graph, Node
from oxionnx_b200.session import Session

pytestmark = pytest.mark.gpu


def _run(graph, weights, feeds, **tuning):
    sess = Session.builder().with_tuning(**tuning).build_from_graph(graph, weights)
    out = sess.run(feeds)
    kernels = [s["kernel"] for s in sess.steps()]
    sess.close()
    return out, kernels


# batch, channels, height, width, filters, kernel, CTA pairs: one to five channel tiles, the last of them ragged, few and many K blocks
SHAPES = [(1, 64, 211, 199, 64, 1, "never"), (1, 32, 211, 199, 64, 3, "never"), (1, 256, 150, 151, 128, 1, "never"), (1, 64, 150, 151, 192, 1, "never"),
          (1, 64, 139, 137, 256, 1, "never"), (1, 128, 139, 137, 320, 1, "never"), (1, 64, 100, 101, 1088, 1, "never"), (2, 64, 61, 43, 320, 3, "always"),
          (1, 512, 61, 43, 448, 1, "always")]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("relu, y_zp", [(True, 0), (False, -3), (False, 131)])
def test_fragment_requantisation_is_the_general_epilogues(shape, relu, y_zp):
    n, c, h, w, oc, k, pairs = shape
    rng = np.random.default_rng([n, c, h, oc, k, y_zp + 3])
    weights = {"w": rng.integers(-127, 128, (oc, c, k, k)).astype(np.float32), "wz": np.zeros(oc, np.float32), "b": rng.integers(-1000, 1001, oc).astype(np.float32),
               "xs": np.float32([0.02]), "z0": np.float32([0]), "yz": np.int8([y_zp]) if y_zp < 0 else np.uint8([y_zp]), "ys": np.float32([0.35])}
    # a standard deviation of some sixty lanes: ties, saturation on both sides and everything between
    spread = 60 * 0.35 / (0.02 * 70 * 40 * np.sqrt(c * k * k))
    weights["ws"] = (spread * rng.uniform(0.7, 1.4, oc)).astype(np.float32)
    nodes = [Node("QuantizeLinear", "q", ["x", "xs", "z0"], ["xq"], {}),
             Node("QLinearConv", "conv", ["xq", "xs", "z0", "w", "ws", "wz", "ys", "yz", "b"], ["yq"], {"pads": [k // 2] * 4})]
    if relu:
        nodes.append(Node("Relu", "r", ["yq"], ["yr"], {}))
    nodes.append(Node("DequantizeLinear", "dq", ["yr" if relu else "yq", "ys", "yz"], ["y"], {}))
    graph = Graph(nodes=nodes, input_names=["x"], output_names=["y"])
    feeds = {"x": np.abs(rng.standard_normal((n, c, h, w))).astype(np.float32)}
    got, kernels = _run(graph, weights, feeds, cta_pairs=pairs)
    assert any("fragments" in s and ("cta-pair" in s) == (pairs == "always") for s in kernels), kernels
    want, general = _run(graph, weights, feeds, cta_pairs=pairs, requant_f64=1)
    assert not any("fragments" in s for s in general), general
    assert np.array_equal(got["y"], want["y"]), f"{np.sum(got['y'] != want['y'])} of {want['y'].size} lanes differ"
    assert np.unique(want["y"]).size > 100, "degenerate test vector"


# rows, K, outputs
LINEARS = [(20001, 64, 192, False), (4099, 256, 1088, True), (9001, 768, 320, False), (20001, 768, 256, False)]


@pytest.mark.parametrize("rows, k, n, gelu", LINEARS)
@pytest.mark.parametrize("pairs", ["never", "always"])
@pytest.mark.parametrize("zero_point", [True, False])
def test_fragment_dequantisation_is_the_separate_nodes(rows, k, n, gelu, pairs, zero_point):
    if pairs == "always" and n < 256:
        pytest.skip("a pair shares a 256-wide tile")
    rng = np.random.default_rng([rows, k, n])
    w = {"w": np.clip(np.rint(rng.standard_normal((k, n)) * 40.0), -127, 127).astype(np.float32),
         "ws": rng.uniform(0.0005, 0.002, n).astype(np.float32), "bias": (rng.standard_normal(n) * 0.5 + 0.8).astype(np.float32)}
    nodes = [Node("DynamicQuantizeLinear", "q0", ["x"], ["xq", "xs", "xz"], {}),
             Node("MatMulInteger", "mmi", ["xq", "w"] + ["xz"] * zero_point, ["acc"], {}), Node("Cast", "cast", ["acc"], ["accf"], {"to": 1}),
             Node("Mul", "scales", ["xs", "ws"], ["sc"], {}), Node("Mul", "rescale", ["accf", "sc"], ["scaled"], {}),
             Node("Add", "addb", ["scaled", "bias"], ["lin"], {})]
    if gelu:
        nodes.append(Node("Gelu", "act", ["lin"], ["act_out"], {}))
    last = nodes[-1].outputs[0]
    nodes.append(Node("DynamicQuantizeLinear", "q1", [last], ["yq", "ys", "yz"], {}))
    graph = Graph(nodes=nodes, input_names=["x"], output_names=[last, "yq", "ys", "yz"])
    feeds = {"x": (rng.standard_normal((rows, k)) * 2 + 0.3).astype(np.float32)}
    got, kernels = _run(graph, w, feeds, cta_pairs=pairs)
    assert any("fragments +dequant" in s and ("cta-pair" in s) == (pairs == "always") for s in kernels), kernels
    want, _ = _run(graph, w, feeds, keep_intermediates=True)
    for name in graph.output_names:
        assert np.array_equal(got[name], want[name]), name


@pytest.mark.parametrize("pairs", ["never", "always"])
@pytest.mark.parametrize("zero_point", [True, False])
def test_values_transposed_by_their_linear(pairs, zero_point):
    """V leaves its linear in the layout that the attention kernel reads, unless somebody else reads it too.  Copies of two
    sentences have the extrema of the two, so every copy is the small batch's, where V is transposed by a launch of its own."""
    from oxionnx_b200 import models
    rng = np.random.default_rng(5)
    ids, mask = rng.integers(0, 500, (2, 128)).astype(np.float32), np.ones((2, 128), np.float32)
    mask[1, 90:] = 0
    out = {}
    for batch, other_reader in ((2, False), (42, False), (42, True)):
        graph, weights, _, _ = models.build_bert_dynamic_int8(batch=batch, seq=128, hidden=768, heads=12, ffn=768, layers=2, vocab=500)
        if not zero_point:
            for node in graph.nodes:
                if node.name in ("l0_v_mmi", "l1_v_mmi"):
                    node.inputs = node.inputs[:2]
        if other_reader:
            graph = Graph(nodes=graph.nodes, input_names=graph.input_names, output_names=graph.output_names + ["l0_v_out"])
        got, kernels = _run(graph, weights, {"input_ids": np.tile(ids, (batch // 2, 1)), "attention_mask": np.tile(mask, (batch // 2, 1))},
                            cta_pairs=pairs if batch > 2 else "never")
        if batch > 2:
            values = [s for s in kernels if s.endswith("fragments +dequant") and "N=768 K=768" in s]
            assert values and all(("cta-pair" in s) == (pairs == "always") for s in values), kernels
        assert sum("umma_attention" in s for s in kernels) == 2, kernels
        assert sum(s.startswith("transpose") for s in kernels) == (2 if batch == 2 else int(other_reader)), kernels
        out[batch, other_reader] = got["hidden"].reshape(batch // 2, 2, 128, 768)
    for copies in ((42, False), (42, True)):
        assert all(np.array_equal(c, out[2, False][0]) for c in out[copies]), copies


def test_transposed_values_are_fetched_in_order():
    """A value that its linear left transposed is handed out in its logical order, by its own name and by a view's."""
    from oxionnx_b200 import models
    rng = np.random.default_rng(6)
    graph, weights, _, _ = models.build_bert_dynamic_int8(batch=42, seq=128, hidden=768, heads=12, ffn=768, layers=1, vocab=500)
    upto = [n.name for n in graph.nodes].index("l0_ctx_merge") + 1
    graph = Graph(nodes=graph.nodes[:upto], input_names=graph.input_names, output_names=["l0_ctx"])
    feeds = {"input_ids": rng.integers(0, 500, (42, 128)).astype(np.float32), "attention_mask": np.ones((42, 128), np.float32)}
    got = {}
    for keep in (False, True):
        sess = Session.builder().with_keep_intermediates(keep).build_from_graph(graph, weights)
        sess.run(feeds)
        assert any(s["kernel"].startswith("transpose") for s in sess.steps()) == keep
        got[keep] = [sess.fetch_value(name) for name in ("l0_v_out", "l0_v4r")]
        sess.close()
    for plain, kept in zip(got[False], got[True]):
        assert plain.shape == kept.shape and np.unique(kept).size > 1000
        # the lanes that a TF32 product reads are rounded to eleven bits by their producer where it knows of the product
        assert np.all(np.abs(plain - kept) <= 2.0**-11 * np.abs(kept))
