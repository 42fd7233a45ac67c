"""Split K of the persistent kernel: the slices' exchange through owners, counters and the workspace."""
import numpy as np
import pytest

from oxionnx_b200.graph import Graph, Node
from oxionnx_b200.session import Session

pytestmark = pytest.mark.gpu

# batch, channels, height, filters, kernel: two to eight slices of 128 and 256 columns, ragged rows, a ragged channel tile
SHAPES = [(32, 256, 14, 256, 3), (8, 512, 7, 512, 3), (32, 512, 7, 512, 3), (29, 2048, 7, 480, 1), (7, 512, 7, 200, 3)]


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
        if precision == "tf32":
            assert any("splitK" in s for s in kernels) == (most == 0), kernels
        session.close()
        out[most] = runs[0]
    # the same exact products, added in f32 in another order: K additions of terms of 1 / sqrt(K), 2^-24 each
    assert np.max(np.abs(out[0] - out[1])) <= 4 * np.sqrt(c * k * k) * 2.0**-24 * np.abs(out[1]).max()
