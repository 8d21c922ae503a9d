"""The record builder's windows over the accept masks: nearly all points accepted, the usual share, almost none.

Whether a point is accepted and its record depend on the point alone, so the records of a pass are the front of a
longer pass's, however both were split over warps and windows."""
import pytest

pytestmark = pytest.mark.gpu

LONG = 1_300_021


@pytest.fixture(scope="module", params=[1e-3, 1.0, 300.0])
def passes(request):
    import torch

    import cupythia_b200 as cp

    it = cp.Integrator()
    it.integrate(4, 1 << 18)
    it.set_wmax(it.weight_quantile(0.99) * request.param)
    rec, st = it.unweight(LONG, iteration=7)
    assert st["n_accepted"] == len(rec)
    torch.cuda.synchronize()
    return it, rec.clone()


@pytest.mark.parametrize("n", [2, 31, 33, 1023, 1025, 32 * 4736 - 1, 32 * 4736 + 17, 300_001, 1_200_003])
def test_records_are_the_front_of_a_longer_pass(passes, n):
    it, ref = passes
    rec, st = it.unweight(n, iteration=7)
    m = st["n_accepted"]
    assert len(rec) == m <= len(ref) and (rec == ref[:m]).all().item()


@pytest.mark.parametrize("capacity", [1, 40, 1000])
def test_records_beyond_the_capacity_are_not_stored(passes, capacity):
    import torch

    import cupythia_b200 as cp

    it, ref = passes
    n = 300_001
    m = it.unweight(n, iteration=7)[1]["n_accepted"]
    buf = torch.zeros((capacity + 8, 64), dtype=torch.uint8, device=ref.device)
    if m > capacity:
        with pytest.raises(cp.CpError, match="too small"):
            it.unweight(n, iteration=7, records=buf[:capacity])
    else:
        it.unweight(n, iteration=7, records=buf[:capacity])
    k = min(capacity, m)
    assert (buf[:k] == ref[:k]).all().item() and (buf[k:] == 0).all().item()
