"""The one-call dispatch of a lazy graph (rt_graph_resolve) and the staged download of small results."""
import numpy as np
import pytest

import ratchet_b200 as rb
from ratchet_b200 import Device, DeviceRequest, Tensor

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    return Device.request_device(DeviceRequest.GPU)


def test_a_diamond_resolves_each_node_once_and_in_order(gpu):
    """Small integers: every product and sum is exact, so the results are equal and not merely close."""
    rng = np.random.default_rng(3)
    a, b, c = (rng.integers(-2, 3, size=(16, 16)).astype(np.float32) for _ in range(3))
    ta, tb, tc = (Tensor.from_data(v, gpu) for v in (a, b, c))
    ab = ta.matmul(tb)
    left, right = ab.matmul(tc), tc.matmul(ab)
    top = left.matmul(right)
    assert list(map(id, (t for t in top.execution_order() if t.op))) == list(map(id, (ab, left, right, top)))
    ab.resolve()
    held = ab.storage
    top.resolve()
    assert ab.storage is held  # already resolved: not computed again
    assert np.array_equal(top.to(Device.CPU).to_numpy(), (a @ b @ c) @ (c @ (a @ b)))
    assert np.array_equal(right.to(Device.CPU).to_numpy(), c @ (a @ b))


def test_an_operand_on_the_host_is_refused_before_anything_is_launched(gpu):
    dev, host = Tensor.from_data(np.ones((4, 4), np.float32), gpu), Tensor.from_data(np.ones((4, 4), np.float32))
    first = dev.matmul(dev)
    top = host.gemm(first, None, False, False, False)
    with pytest.raises(rb.RatchetError, match="operand on"):
        top.resolve()
    assert not first.resolved() and not top.resolved()


@pytest.mark.parametrize("nbytes", [16, 4096, (256 << 10) - 4, 256 << 10, (256 << 10) + 4])
def test_downloads_around_the_staging_area(gpu, nbytes):
    data = np.random.default_rng(nbytes).integers(0, 1 << 32, size=nbytes // 4, dtype=np.uint32)
    t = Tensor.from_data(data, gpu)
    pinned = rb.PinnedArray((nbytes // 4,), np.uint32)
    t.to(Device.CPU, out=pinned.array)
    assert np.array_equal(t.to(Device.CPU).to_numpy(), data) and np.array_equal(pinned.array, data)
