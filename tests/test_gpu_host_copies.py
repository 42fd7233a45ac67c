"""Host lanes in and out of a planned session at the sizes where the copy path changes: the session's staging
memory (up to 256 KB), the driver's staging, and the piecewise copies (512 KB pieces; uploads from 16 MB on)."""
import numpy as np
import pytest

from oxionnx_b200.graph import Graph, Node
from oxionnx_b200.session import Session

pytestmark = pytest.mark.gpu

KB = 256  # lanes per KB


@pytest.mark.parametrize("lanes", [1, 256 * KB - 1, 256 * KB, 256 * KB + 1, 512 * KB + 1, 1024 * KB, 16 * 1024 * KB - 1, 16 * 1024 * KB, 17 * 1024 * KB + 5])
def test_feeds_and_fetches_arrive_whole(lanes):
    graph = Graph(nodes=[Node("Relu", "relu", ["x"], ["y"], {})], input_names=["x"], output_names=["y"])
    sess = Session.builder().build_from_graph(graph, {})
    for seed in range(2):  # the second run meets buffers that the first has filled
        x = np.random.default_rng(seed).standard_normal(lanes).astype(np.float32)
        want = np.maximum(x, 0)
        assert np.array_equal(sess.run({"x": x})["y"], want)
        for got in sess.run_pipelined([{"x": x}, {"x": -x}]):
            assert np.array_equal(got["y"], want)
            want = np.maximum(-x, 0)
    sess.close()
