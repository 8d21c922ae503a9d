"""The tensor-core flow forward at the edges of its tiles and of a wave of them.

A point's output depends on its index and the stream alone, so a pass of any length has the same bytes as the
front of a longer one, whichever block, warpgroup and round took a point's tile.
"""
import pytest

pytestmark = pytest.mark.gpu

TILE, WAVE = 128, 5 * 128 * 148


@pytest.fixture(scope="module")
def sampled():
    import cupythia_b200 as cp

    it = cp.Integrator()
    it.flow_init(5)
    it.flow_train(6, batch=8192, lr=2e-3)
    return it, it.flow_sample(0, 2 * WAVE + 3 * TILE + 5, iteration=2, stream=0).cpu().numpy()


@pytest.mark.parametrize("n", [1, 31, TILE - 1, TILE, TILE + 1, 148 * TILE - 1, 148 * TILE + 1, WAVE - 1, WAVE, WAVE + 1,
                               2 * WAVE + TILE + 7])
def test_tiles_do_not_depend_on_the_length_of_the_pass(sampled, n):
    it, ref = sampled
    assert it.flow_sample(0, n, iteration=2, stream=0).cpu().numpy().tobytes() == ref[:n].tobytes()


@pytest.mark.parametrize("point0", [1, 129, WAVE + 64])
def test_tiles_do_not_depend_on_the_first_point(sampled, point0):
    it, ref = sampled
    n = 3 * TILE + 5
    assert it.flow_sample(point0, n, iteration=2, stream=0).cpu().numpy().tobytes() == ref[point0:point0 + n].tobytes()
