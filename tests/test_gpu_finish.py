"""The kernels that end a pass (threshold quantile, grid refinement, variance-gradient step) against
the oracle or plain numpy, over the bin counts and histograms where their splits over threads and
lanes have edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QBINS = 4096


def _quantile(hist, q):
    """The serial rule: down from the top while at most (1 - q) of the weights lie above."""
    allowed, above, b = (1.0 - q) * float(hist.sum()), 0, QBINS - 1
    while b > 0 and not float(above + int(hist[b])) > allowed:
        above += int(hist[b])
        b -= 1
    return float(np.array((b + 1 + ((127 - 64) << 5)) << 18, np.uint32).view(np.float32))


@pytest.mark.parametrize("kind", ["empty", "first", "last", "one_thread", "sparse", "full", "huge"])
@pytest.mark.parametrize("q", [1e-9, 0.5, 0.999, 1 - 1e-12])
def test_quantile_of_a_histogram(kind, q):
    import torch

    import cupythia_b200 as cp
    rng = np.random.default_rng(3)
    h = np.zeros(QBINS, np.int64)
    if kind == "first":
        h[0] = 5
    elif kind == "last":
        h[-1] = 1
    elif kind == "one_thread":
        h[2048:2052] = [7, 0, 1000, 1]
    elif kind == "sparse":
        h[rng.integers(0, QBINS, 9)] = rng.integers(1, 1 << 20, 9)
    elif kind == "full":
        h[:] = rng.integers(0, 1000, QBINS)
    elif kind == "huge":
        h[:] = rng.integers(0, 1 << 40, QBINS)
    with cp.Integrator() as it:
        assert it.quantile_from_histogram(torch.as_tensor(h, device=it.device), q) == _quantile(h, q)


@pytest.mark.parametrize("nb", [2, 3, 31, 33, 64, 128])
@pytest.mark.parametrize("alpha", [0.0, 0.5, 1.5])
def test_refinement_matches_the_oracle(orc, nb, alpha):
    import torch

    import cupythia_b200 as cp
    rng = np.random.default_rng(nb)
    with cp.Integrator(n_bins=nb) as it:
        for shape in ("random", "peak", "zero_dimension"):
            hist = rng.random((3, nb)) ** 4
            if shape == "peak":
                hist[:] = 0.0
                hist[:, nb // 2] = 1e3
            elif shape == "zero_dimension":
                hist[1] = 0.0
            edges = it.grid
            sums = np.concatenate([[2.0, 5.0, 1.5, 0.0], hist.reshape(-1)])
            r = it.refine(torch.as_tensor(sums, device=it.device), 1000.0, alpha)
            assert r["w_max"] == 1.5 and r["sigma"] == 2.0 / 1000.0
            if alpha > 0:
                orc.lib().cpo_vegas_refine(orc.dptr(edges), orc.dptr(np.ascontiguousarray(hist.reshape(-1))), 3, nb, alpha)
            assert np.max(np.abs(it.grid - edges)) < 1e-12, shape
            if shape == "random":
                it.grid = np.clip(it.grid, 0, 1)   # the next shape starts from a non-uniform grid


@pytest.mark.parametrize("nb", [2, 3, 33, 50, 128])
@pytest.mark.parametrize("p", [2.0, 4.0])
def test_gradient_step_of_given_sums(nb, p):
    import torch

    import cupythia_b200 as cp
    rng = np.random.default_rng(nb)
    n, lr = 4096, 0.3
    with cp.Integrator(n_bins=nb) as it:
        it.gradient_objective(p)
        head = np.array([1.1 * n, 3.7 * n, 0, 0, 0, 0, 0, 0, 9.0, 0])
        h = rng.standard_normal((3, 4, nb)) * n / nb
        g = it.gradient_apply(torch.as_tensor(np.concatenate([head, h.reshape(-1)]), device=it.device), n, lr)
        mean, mp = 1.1, 3.7
        var = mp - mean ** 2 if p == 2.0 else (mp / mean ** p - 1.0) * mean ** 2
        assert abs(g["sigma"] - mean) < 1e-13 and abs(g["var"] - var) < 1e-12
        cm = 2.0 * mean if p == 2.0 else p * mp / mean
        width = np.full(nb, 1.0 / nb)
        for d in range(3):
            a = np.concatenate([h[d, 0], [0.0]]) + np.concatenate([[0.0], h[d, 1]])
            aw = np.concatenate([h[d, 2], [0.0]]) + np.concatenate([[0.0], h[d, 3]])
            gv = p * aw / n - cm * a / n
            tail = np.array([gv[b + 1:nb].sum() for b in range(nb)])
            G = width * tail
            new = width * np.exp(-lr * G / np.abs(G).max())
            ref = np.concatenate([[0.0], np.cumsum(new / new.sum())])
            ref[-1] = 1.0
            assert np.max(np.abs(it.grid[d] - ref)) < 1e-12, d
