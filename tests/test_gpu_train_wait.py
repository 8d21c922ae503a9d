"""The training kernels' bounded wait for their weights, let run out by the test hook (no copy is started): the call
reports it, and training from the saved state gives the undisturbed run's result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [64, 65536])
def test_expired_weight_wait_is_reported_and_recoverable(batch):
    import cupythia_b200 as cp

    with cp.Integrator() as it:
        it.integrate(2, 1 << 16)
        it.flow_init(7)
        it.flow_train(2, batch)
        state, updates = it.flow_state()
        ref = it.flow_train(3, batch)
        params = it.flow_params
        it.lib.cp_flow_test_stall(it.h, 1)
        with pytest.raises(cp.CpError) as e:
            it.flow_train(1, batch)
        assert e.value.code == cp._lib.CP_ERR_TIMEOUT
        with pytest.raises(cp.CpError) as e:
            it.flow_loss_grad(batch, 3)
        assert e.value.code == cp._lib.CP_ERR_TIMEOUT
        it.lib.cp_flow_test_stall(it.h, 0)
        it.flow_restore(state, updates)
        assert np.array_equal(it.flow_train(3, batch), ref) and np.array_equal(it.flow_params, params)
