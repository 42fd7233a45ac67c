"""Split K of the persistent kernel: the slices' exchange through owners, counters and the workspace."""
import numpy as np
import pytest

from oxionnx_b200.graph import Graph, Node
from oxionnx_b200.session import Session

pytestmark = pytest.mark.gpu

# batch, channels, height, filters, kernel: two to eight slices of 128 and 256 columns, ragged rows, a ragged channel tile
SHAPES = [(32, 256, 14, 256, 3), (8, 512, 7, 512, 3), (32, 512, 7, 512, 3), (29, 2048, 7, 480, 1), (7, 512, 7, 200, 3)]

UNSPLIT_16 = [SHAPES[0]]  # half the K blocks in 16 bits: whole sums there; the others meet in the workspace (SHAPES[2]) or within a cluster


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("precision", ["tf32", "bf16"])
def test_slices_meet_in_the_order_of_their_index(shape, precision):
    n, c, h, oc, k = shape
    rng = np.random.default_rng([n, c, h, oc, k])
    weights = {"w": (rng.standard_normal((oc, c, k, k)) / np.sqrt(c * k * k)).astype(np.float32), "b": rng.standard_normal(oc).astype(np.float32)}
    graph = Graph(nodes=[Node("Relu", "pre", ["x"], ["x1"], {}), Node("Conv", "conv", ["x1", "w", "b"], ["y"], {"pads": [k // 2] * 4})], input_names=["x"], output_names=["y"])
    feeds = {"x": rng.standard_normal((n, c, h, h)).astype(np.float32)}
    out = {}
    for most in (0, 1):
        session = Session.builder().with_tuning(split_k_max=most, float_precision=precision).build_from_graph(graph, weights)
        runs = [session.run(feeds)["y"].copy() for _ in range(4)]
        assert all(np.array_equal(r, runs[0]) for r in runs), "the sum depends on who arrived when"
        kernels = [s["kernel"] for s in session.steps()]
        split = most == 0 and not (precision == "bf16" and shape in UNSPLIT_16)
        assert any("splitK" in s for s in kernels) == split, kernels
        session.close()
        out[most] = runs[0]
    # the same exact products, added in f32 in another order: K additions of terms of 1 / sqrt(K), 2^-24 each
    assert np.max(np.abs(out[0] - out[1])) <= 4 * np.sqrt(c * k * k) * 2.0**-24 * np.abs(out[1]).max()


# batch, channels, height, filters: slices of the persistent kernel behind a 3x3 filter of 81 K blocks and more, where the small-problem
# kernel takes no slice; whole and ragged channel tiles, ragged rows
INTEGER_SHAPES = [(32, 1152, 7, 256), (11, 1280, 13, 160), (29, 1152, 7, 512)]


@pytest.mark.parametrize("shape", INTEGER_SHAPES, ids=str)
@pytest.mark.parametrize("behind", ["requantisation", "join"])
def test_integer_slices_are_the_unsplit_sum(shape, behind):
    n, c, h, oc = shape
    rng = np.random.default_rng([n, c, h, oc])
    peak = (1 << 24) // (300 * c * 9)  # accumulators that convert exactly
    weights = {"w": rng.integers(-peak, peak + 1, (oc, c, 3, 3)).astype(np.float32), "wz": np.int8([0]), "xs": np.float32([0.02]), "z0": np.uint8([0]),
               "bias": rng.integers(-1000, 1001, oc).astype(np.float32), "as": np.float32([0.07622]), "az": np.uint8([128]), "one": np.float32([1]),
               "bs": np.float32([0.04274]), "ys": np.float32([0.05397])}
    # a standard deviation of about thirty lanes, so that no accumulator can leave the int16 range
    weights["ws"] = (rng.uniform(0.7, 1.4, oc) * 30 / (40 * peak / np.sqrt(3) * np.sqrt(9 * c)) * 0.07622 / 0.02).astype(np.float32)
    nodes = [Node("QuantizeLinear", "qx", ["x", "xs", "z0"], ["xq"], {}),
             Node("QLinearConv", "conv", ["xq", "xs", "z0", "w", "ws", "wz", "as", "az", "bias"], ["aq"], {"pads": [1] * 4})]
    feeds = {"x": np.abs(rng.standard_normal((n, c, h, h))).astype(np.float32)}
    if behind == "join":
        nodes += [Node("QuantizeLinear", "qr", ["r", "one", "az"], ["rq"], {}), Node("DequantizeLinear", "da", ["aq", "as", "az"], ["a"], {}),
                  Node("DequantizeLinear", "db", ["rq", "bs", "z0"], ["b"], {}), Node("Add", "add", ["a", "b"], ["sum"], {}), Node("Relu", "relu", ["sum"], ["s"], {}),
                  Node("QuantizeLinear", "qy", ["s", "ys", "z0"], ["yq"], {}), Node("DequantizeLinear", "dy", ["yq", "ys", "z0"], ["y"], {})]
        # the residual's producer stands in front of the convolution
        nodes.insert(0, nodes.pop(2))
        feeds["r"] = (rng.integers(0, 256, (n, oc, h, h)) - 128).astype(np.float32)
    else:
        nodes.append(Node("DequantizeLinear", "dy", ["aq", "as", "az"], ["y"], {}))
    graph = Graph(nodes=nodes, input_names=list(feeds), output_names=["y"])
    out = {}
    for most in (0, 1):
        session = Session.builder().with_tuning(split_k_max=most).build_from_graph(graph, weights)
        runs = [session.run(feeds)["y"].copy() for _ in range(4)]
        assert all(np.array_equal(r, runs[0]) for r in runs)
        kernel = [s["kernel"] for s in session.steps() if s["node"] == "conv" and s["kernel"].startswith("umma")][0]
        assert ("splitK" in kernel) == (most == 0) and "small" not in kernel and kernel.endswith("+join") == (behind == "join"), kernel
        session.close()
        out[most] = runs[0]
    assert np.array_equal(out[0], out[1])
    assert np.unique(out[0]).size > 60


def test_layers_of_a_session_share_one_workspace():
    """Two and ten layers of the same filters, each of whose slices fill a workspace of several MB: the longer session holds no more of them."""
    import torch
    rng = np.random.default_rng(3)
    weights = {"w": (rng.standard_normal((512, 512, 3, 3)) / np.sqrt(9 * 512)).astype(np.float32), "b": np.zeros(512, np.float32)}
    feeds = {"x": rng.standard_normal((32, 512, 7, 7)).astype(np.float32)}
    held = {}
    for layers in (2, 10):
        nodes = [Node("Relu", "pre", ["x"], ["x0"], {})]
        nodes += [Node("Conv", f"c{i}", [f"x{i}", "w", "b"], [f"x{i + 1}"], {"pads": [1] * 4, "activation": "relu"}) for i in range(layers)]
        graph = Graph(nodes=nodes, input_names=["x"], output_names=[f"x{layers}"])
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        session = Session.builder().build_from_graph(graph, weights)
        session.run(feeds)
        held[layers] = before - torch.cuda.mem_get_info()[0]
        split = [s["kernel"] for s in session.steps() if "splitK" in s["kernel"]]
        session.close()
        assert len(split) == layers and not any("small" in s for s in split), split
    tile = [int(v) for v in split[0].split("tile=")[1].split("x")[:2]]
    workspace = -(-32 * 49 // tile[0]) * (512 // tile[1]) * int(split[0].split("splitK=")[1].split()[0]) * tile[0] * tile[1] * 4
    assert workspace >= 4 << 20
    assert held[10] - held[2] < 2 * workspace, (held, workspace)
