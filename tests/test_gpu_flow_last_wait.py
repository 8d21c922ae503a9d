"""A tensor-core wait that expires in one warp only, at its tiles' end: the warps that are through by then must not hide
it.  The test hook lets the last warp of each warpgroup wait about a second for an arrival that does not come."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 128, 4096, 148 * 5 * 128 + 1])
def test_one_warp_s_expired_last_wait_is_reported(n):
    import cupythia_b200 as cp

    with cp.Integrator() as it:
        it.flow_init(7)
        ref = it.flow_sample(0, n, 3, 0).cpu().numpy()
        it.lib.cp_flow_test_stall(it.h, 2)
        with pytest.raises(cp.CpError) as e:
            it.flow_sample(0, n, 3, 0)
        assert e.value.code == cp._lib.CP_ERR_TIMEOUT
        it.lib.cp_flow_test_stall(it.h, 0)
        assert np.array_equal(it.flow_sample(0, n, 3, 0).cpu().numpy(), ref)


def test_the_same_in_fused_production():
    import cupythia_b200 as cp

    with cp.Integrator() as it:
        it.integrate(2, 1 << 16)
        it.flow_init(7)
        it.flow_enable(True)
        it.flow_fuse_production(True)
        it.set_wmax(1e-3)
        ref = cp.events_view(it.unweight(5000, iteration=4)[0]).tobytes()
        it.lib.cp_flow_test_stall(it.h, 2)
        with pytest.raises(cp.CpError) as e:
            it.unweight(5000, iteration=4)
        assert e.value.code == cp._lib.CP_ERR_TIMEOUT
        it.lib.cp_flow_test_stall(it.h, 0)
        assert cp.events_view(it.unweight(5000, iteration=4)[0]).tobytes() == ref
