"""Training that production passes interrupt: the buffers they gave back are made anew with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_training_goes_on_after_production_passes():
    import cupythia_b200 as cp

    got = []
    for produce in (False, True):
        with cp.Integrator() as it:
            it.integrate(3, 1 << 16)
            it.flow_init(7)
            it.set_wmax(1e-3)
            a = it.flow_train(3, 4096 + 32)
            if produce:
                for _ in range(9):
                    it.unweight(5000)
            b = it.flow_train(3, 4096 + 32)
            m = it.flow_step_moments(0, 1000)
            if produce:
                for _ in range(9):
                    it.unweight(5000)
            g, loss = it.flow_step_gradient(m, 1000)
            got.append((a, b, g.cpu().numpy(), loss, it.flow_params))
    for x, y in zip(*got):
        assert np.array_equal(x, y)
