"""Weight gradients of training steps whose points do not fill their 64-point stages: the tcgen05 and
mma.sync kernels agree bit for bit, and a step's gradient is the sum of its shares' gradients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradient(it, point0, count, moments, total):
    it.flow_step_moments(point0, count)
    return it.flow_step_gradient(moments, total)[0].cpu().numpy().astype(np.float64)


@pytest.fixture(scope="module")
def flow():
    import cupythia_b200 as cp
    it = cp.Integrator()
    it.integrate(4, 1 << 16, alpha=1.5)
    it.flow_init(7)
    it.flow_train(8, 4096, lr=8e-3)      # non-zero output layers, so every gradient is non-zero
    yield it
    it.close()


@pytest.mark.parametrize("count", [1, 7, 31, 33, 63, 64, 65, 127, 1000, 4097, 65536 + 24])
def test_gradient_of_ragged_steps(flow, count):
    it = flow
    m = it.flow_step_moments(0, count)
    whole = {}
    for kernel in ("tcgen05", "mma"):
        it.flow_kernel(kernel)
        whole[kernel] = _gradient(it, 0, count, m, count)
    it.flow_kernel("tcgen05")
    assert np.array_equal(whole["tcgen05"], whole["mma"])
    g = whole["tcgen05"]
    assert np.linalg.norm(g) > 0
    if count > 1:
        a = count // 3 + 1
        parts = _gradient(it, 0, a, m, count) + _gradient(it, a, count - a, m, count)
        # the same products in another order of FP32 additions (1024 points a slot, 64 slots)
        scale = np.abs(_gradient(it, 0, a, m, count)) + np.abs(_gradient(it, a, count - a, m, count))
        assert np.linalg.norm(g - parts) <= 1024 * 2.0 ** -24 * np.linalg.norm(scale) + 1e-12
