"""Passes with so few points that most blocks of the iteration-end cluster have no slot to load and go straight to
the first block's shared memory: the records and grids of many of them, against the separate kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 255, 256, 257, 1024])
def test_one_slot_iterations_match_accumulate_and_refine(n):
    import cupythia_b200 as cp

    with cp.Integrator(n_bins=50) as a, cp.Integrator(n_bins=50) as b:
        per, _ = a.integrate(50, n, alpha=0.3)
        for k, r in enumerate(per):
            assert r == b.refine(b.accumulate(n, k), n, 0.3)
        assert np.asarray(a.grid).tobytes() == np.asarray(b.grid).tobytes()
