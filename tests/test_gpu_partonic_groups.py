"""SplitMix64 partonic sums over groups of 32 reference threads, and over more than one wave of blocks.

Reference thread i counts from seed + i 0x100000001B3, so a run over n threads is the sum of runs over consecutive
pieces of them.  The pieces below go through the other split of the draws, or fewer blocks.  Both sides add
positive FP64 terms, at most a few thousand in a row per thread, then trees: 1e-13."""
import pytest

pytestmark = pytest.mark.gpu

STEP = 0x100000001B3


@pytest.mark.parametrize("threads,draws,piece", [(1024, 1, 512), (1025, 7, 1000), (1056, 9, 33), (33_001, 3, 1000),
                                                 (70_000, 900, 8750), (1100, 60_000, 137)])
def test_sum_of_pieces(integ, threads, draws, piece):
    seed = 0xFFFFFFFFFFFF0000
    whole = integ.partonic_splitmix(threads, draws, seed=seed)
    s1 = s2 = wm = 0.0
    for first in range(0, threads, piece):
        r = integ.partonic_splitmix(min(piece, threads - first), draws, seed=(seed + first * STEP) % (1 << 64))
        s1, s2, wm = s1 + r["sum_w"], s2 + r["sum_w2"], max(wm, r["w_max"])
    assert whole["n_points"] == threads * draws
    assert abs(whole["sum_w"] / s1 - 1) < 1e-13 and abs(whole["sum_w2"] / s2 - 1) < 1e-13 and whole["w_max"] == wm
