"""Memory that a context holds only for reuse is there for whoever needs it when the device is nearly full."""
import numpy as np
import pytest

from oxionnx_b200.graph import Node
from oxionnx_b200.session import CudaContext, try_cuda_dispatch, try_cuda_dispatch_resident

pytestmark = pytest.mark.gpu

MB = 1 << 20
RELU = Node("Relu", "r", ["x"], ["y"], {})


@pytest.fixture
def leave_free():
    """leave_free(n): takes all of the device's memory but about n bytes; given back when the test ends."""
    import torch
    taken = []

    def take(n):
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        assert free > n
        taken.append(torch.empty(free - n, dtype=torch.uint8, device="cuda"))

    yield take
    taken.clear()
    torch.cuda.empty_cache()


def _relu(ctx, x, placement):
    return try_cuda_dispatch_resident(RELU, {}, {"x": x}, placement, ctx)


def _fill_pool(ctx):
    """Five released device tensors of 48 MB."""
    x = np.full(12 * MB, -1.0, np.float32)
    for t in [_relu(ctx, x, "device") for _ in range(5)]:
        t.release()


def _fill_plans(ctx):
    """Five kept plans of 48 MB (an input and an output of 24 MB each)."""
    for i in range(5):
        x = np.full(6 * MB - i, -1.0, np.float32)
        assert not try_cuda_dispatch(RELU, {}, {"x": x}, ctx)[0].any()


@pytest.mark.parametrize("held", [_fill_pool, _fill_plans])
def test_a_new_plan_takes_what_is_held_for_reuse(leave_free, held):
    ctx = CudaContext(0)
    held(ctx)
    leave_free(300 * MB)
    x = np.linspace(-1, 1, 32 * MB).astype(np.float32)  # operand, result and the tensor handed out: three times 128 MB
    y = _relu(ctx, x, "device")
    assert np.array_equal(y.read_back(), np.maximum(x, 0))
    y.release()
    ctx.close()


def test_a_kept_plan_outlives_the_others_while_it_runs(leave_free):
    ctx = CudaContext(0)
    _fill_plans(ctx)
    x = np.linspace(-1, 1, 6 * MB).astype(np.float32)
    tensors = [_relu(ctx, x, "device")]
    leave_free(16 * MB)  # not enough for another tensor of this size
    tensors.append(_relu(ctx, x, "device"))  # the plan of this very call is among the kept ones
    tensors.append(_relu(ctx, x, "device"))
    for t in tensors:
        assert np.array_equal(t.read_back(), np.maximum(x, 0))
        t.release()
    ctx.close()
