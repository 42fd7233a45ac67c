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
