"""The end of an iteration in one cluster launch against the separate reduction and refinement kernels.

Both add the block slots in one order and share the refinement, so the record and the grid have the same bytes,
over bin counts that do and do not fill the column groups and passes of one block to all of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [2, 3, 31, 50, 65, 128])
@pytest.mark.parametrize("n", [2, 257, 33 * 256 + 1, 300_001])
def test_iteration_matches_accumulate_and_refine(nb, n):
    import cupythia_b200 as cp

    with cp.Integrator(n_bins=nb) as a, cp.Integrator(n_bins=nb) as b:
        for k, alpha in enumerate((1.5, 0.7)):
            ra = a.iteration(n, k, alpha)
            rb = b.refine(b.accumulate(n, k), n, alpha)
            assert ra == rb
            assert np.asarray(a.grid).tobytes() == np.asarray(b.grid).tobytes()


@pytest.mark.parametrize("n_iter", [1, 2, 3])
def test_weight_histogram_is_the_last_pass_s(n_iter):
    import cupythia_b200 as cp

    n = 70_001
    with cp.Integrator() as a, cp.Integrator() as b:
        a.iteration(5000, 9)     # leaves a histogram behind
        a.grid = b.grid
        a.integrate(n_iter, n)
        for k in range(n_iter):
            b.iteration(n, k)
        assert np.asarray(a.grid).tobytes() == np.asarray(b.grid).tobytes()
        h = a.weight_histogram().cpu().numpy()
        assert (h == b.weight_histogram().cpu().numpy()).all() and 0 < h.sum() <= n
