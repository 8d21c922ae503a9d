"""Scale-variation ratios at the sizes where their kernel's mapping has edges (one record, one beyond a
block of points, several chunks): every record's ratios are those of the same event in a larger pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def production():
    import cupythia_b200 as cp
    it = cp.Integrator()
    it.integrate(5, 1 << 18, alpha=1.5)
    it.iteration(1 << 18, 9, alpha=0.0)
    it.weight_quantile(0.999)
    yield it
    it.close()


@pytest.mark.parametrize("n", [2, 33, 127, 129, 1025, 50021, (1 << 24) + 77])
def test_ratios_follow_their_records(production, n):
    import cupythia_b200 as cp
    it = production
    it.set_point_offset(0)
    rec, w, st = it.unweight_scale_weights(n, iteration=4)
    ev = cp.events_view(rec)
    w = w.cpu().numpy()
    assert w.shape == (st["n_accepted"], 6) and np.all(np.isfinite(w)) and np.all(w > 0)
    assert np.allclose(w[:, 4], w[:, 0] * w[:, 2], rtol=1e-6) and np.allclose(w[:, 5], w[:, 1] * w[:, 3], rtol=1e-6)
    # the last events again, from a pass that starts at another point: other blocks, ranges and chunks
    start = max(0, n - 4099) | 1 if n > 4099 else 0
    it.set_point_offset(start)
    try:
        rec2, w2, _ = it.unweight_scale_weights(max(2, n - start), iteration=4)
    finally:
        it.set_point_offset(0)
    ev2, w2 = cp.events_view(rec2), w2.cpu().numpy()
    tail = ev["point"] >= start
    assert np.array_equal(ev[tail], ev2[:tail.sum()])
    assert np.array_equal(w[tail], w2[:tail.sum()])


def test_ratios_stop_at_the_capacity(production):
    import cupythia_b200 as cp
    import torch
    it = production
    small = torch.empty((10, 64), dtype=torch.uint8, device=it.device)
    with pytest.raises(cp.CpError):
        it.unweight_scale_weights(50000, iteration=6, records=small)
    rec, w, _ = it.unweight_scale_weights(50000, iteration=6)
    assert np.array_equal(cp.events_view(rec[:10]), cp.events_view(small))
