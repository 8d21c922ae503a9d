"""The partonic g g -> g g kernel's matrix element and draws at the ends of its ranges, against the
closed form (9/2)(3 - tu/s^2 - su/t^2 - st/u^2) in extended precision at the kernel's own cos theta."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _element(c):
    """(9/2) x the form at cos theta = c (double) in long double, 64-bit mantissa."""
    c = c.astype(np.longdouble)
    t, u = -(1 - c) / 2, -(1 + c) / 2
    return 4.5 * (3 - t * u - u / t ** 2 - t / u ** 2)


def _scale(s, aS, cmax, conv):
    return np.longdouble(np.pi) / s ** 2 * aS ** 2 * 0.5 * (2 * cmax) * (s / 2) * conv


@pytest.mark.parametrize("cmax", [1e-3, 0.5, 0.9, 0.999, 1 - 2.0 ** -30])
def test_weights_against_extended_precision(integ, cmax):
    n = 5000
    w = integ.partonic_weights(77, n, cmax=cmax).cpu().numpy()
    words = integ.philox_words(42, 77, n, 0, 0).astype(np.uint64)
    u = (((words[:, 1] << np.uint64(32)) | words[:, 0]) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
    ref = _element((2 * u - 1) * cmax) * _scale(1e4, 0.13, cmax, 0.3893793721)
    # units of 2^-53: 1 - c^2 1/2, 1 / p 1, 16 y - 12 up to 4 x those + 1/2, the product and sum 1,
    # the prefactor's five roundings
    assert np.max(np.abs(w / ref - 1)) < 16 * 2.0 ** -53


@pytest.mark.parametrize("threads,draws", [(1, 2), (2, 1), (3, 7), (1000, 1), (70001, 3), (5, 100003), (1, 300000)])
def test_splitmix_sums_over_shares(integ, threads, draws):
    """Runs of one draw, shares that cross many reference threads, shares inside one."""
    r = integ.partonic_splitmix(threads, draws, seed=99)
    with np.errstate(over="ignore"):
        i = np.repeat(np.arange(threads, dtype=np.uint64), draws)
        k = np.tile(np.arange(draws, dtype=np.uint64), threads)
        z = np.uint64(99) + i * np.uint64(0x100000001B3) + k + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    u = (z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
    w = _element((2 * u - 1) * 0.9) * _scale(1e4, 0.118, 0.9, 0.3893793721)
    n = threads * draws
    assert r["n_points"] == n
    assert abs(r["sum_w"] / w.sum() - 1) < 1e-13 and abs(r["sum_w2"] / (w * w).sum() - 1) < 1e-13
    assert abs(r["w_max"] / w.max() - 1) < 16 * 2.0 ** -53
