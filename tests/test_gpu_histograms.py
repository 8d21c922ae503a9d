"""Per-bin sums of the VEGAS and adjoint passes against plain FP64 sums over the same points, at the
sizes where the warp adds can go wrong: part of a warp, one point beyond a warp or block, few bins
(every lane of a warp in one of two bins) and the most bins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bins(it, n, iteration):
    words = it.philox_words(it.cfg.seed, 0, n, iteration, 0)
    m = (words[:, :3] >> 8).astype(np.uint64) * it.nb
    return (m >> 24).astype(np.int64)


@pytest.mark.parametrize("nb", [2, 3, 50, 128])
@pytest.mark.parametrize("n", [2, 31, 33, 257, 5000])
def test_vegas_bin_sums(nb, n):
    import cupythia_b200 as cp
    with cp.Integrator(n_bins=nb) as it:
        w = it.point_weights(0, n, 3).cpu().numpy()
        w2 = (w * w).astype(np.float64)   # squared in FP32, as the pass does (tiny squares underflow)
        h = it.last_histogram()["hist"]
        b = _bins(it, n, 3)
        for d in range(3):
            ref = np.bincount(b[:, d], weights=w2, minlength=nb)
            # at most 256 FP32 additions of non-negative terms per block and bin
            assert np.all(np.abs(h[d] - ref) <= 257 * 2.0 ** -24 * ref), (d, nb, n)


@pytest.mark.parametrize("params", [True, False])
@pytest.mark.parametrize("nb,n", [(2, 33), (3, 31), (50, 129), (128, 5000)])
def test_adjoint_bin_sums(nb, n, params):
    """The lower- and upper-edge sums add up to the x-derivative sums of their bin: per dimension
    lo + hi = sum of df/dx J over the bin's points, and every histogram is the sum of one-point
    passes (point offset p, one point each)."""
    import cupythia_b200 as cp
    with cp.Integrator(n_bins=nb) as it:
        it.adjoint_parameter_tangents(params)
        whole = it.adjoint_accumulate(n, iteration=5).cpu().numpy()
        parts = np.zeros_like(whole)
        size = np.zeros_like(whole)
        for p in range(0, n, 7):
            it.set_point_offset(p)
            s = it.adjoint_accumulate(min(7, n - p), iteration=5).cpu().numpy()
            s[8] = 0.0
            parts += s
            size += np.abs(s)
        whole[8] = 0.0
        # FP32 adds of at most n terms in either order, against the sum of the terms' magnitudes
        assert np.all(np.abs(whole - parts) <= 2 * (min(n, 300) + 7) * 2.0 ** -24 * size + 1e-30)
