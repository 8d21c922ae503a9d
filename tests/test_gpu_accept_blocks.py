"""Production passes at the sizes where the accept kernel's blocks, the offset scan and the cleared
range totals have edges: the accepted set is {u w_max < w}, in point order, whatever ran before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def production():
    import cupythia_b200 as cp
    it = cp.Integrator()
    it.integrate(5, 1 << 18, alpha=1.5)
    it.iteration(1 << 18, 9, alpha=0.0)
    it.wmax = it.weight_quantile(0.999)
    yield it
    it.close()


def _accepted(it, n, iteration):
    w = it.point_weights(0, n, iteration).cpu().numpy()
    words = it.philox_words(it.cfg.seed, 0, n, iteration, 0)
    u = (words[:, 3] >> 8).astype(np.float32) * np.float32(2.0 ** -24)
    return np.nonzero(u * np.float32(it.wmax) < w)[0], w


@pytest.mark.parametrize("n", [2, 31, 33, 127, 129, 1023, 1025, 16383, 16385, 300007, 1000003, 5 << 20])
def test_accepted_points_in_order(production, n):
    import cupythia_b200 as cp
    it = production
    points, w = _accepted(it, n, 4)
    rec, stats = it.unweight(n, iteration=4)
    ev = cp.events_view(rec)
    assert np.array_equal(ev["point"], points.astype(np.uint32))
    assert stats["n_accepted"] == len(points)
    assert stats["w_max_seen"] == w.max()
    assert abs(stats["sigma"] / w.astype(np.float64).mean() - 1) < 1e-6


def test_passes_do_not_see_each_other(production):
    """A pass after a larger one, after one without records and after one that overflowed."""
    import cupythia_b200 as cp
    import torch
    it = production
    ref = cp.events_view(it.unweight(20011, iteration=4)[0]).copy()
    it.unweight(1 << 20, iteration=5)
    small = torch.empty((10, 64), dtype=torch.uint8, device=it.device)
    with pytest.raises(cp.CpError):
        it.unweight(50000, iteration=6, records=small)
    it.unweight(50000, iteration=6, records=torch.empty((50000, 64), dtype=torch.uint8, device=it.device))
    assert np.array_equal(cp.events_view(it.unweight(20011, iteration=4)[0]), ref)
