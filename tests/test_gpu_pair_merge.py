"""A pair without gates: a side pass over few tiles merges its scores itself (handles without guided
buffers in both passes, handles with them in the second; the largest size here is above the line), and
one block writes the pairs of up to 8192 lefts.

Whole numbers throughout: the matches equal the oracle's."""
import numpy as np
import pytest

from v3dm import synth

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 33), (31, 1), (127, 129), (129, 256), (257, 255), (300, 1025), (2000, 31), (8192, 300),
          (8193, 257), (9000, 9100)]


@pytest.mark.parametrize("guided", [False, True])
@pytest.mark.parametrize("nL,nR", SHAPES)
def test_merged_pair_matches_the_oracle(v3dm_mod, oracle_mod, nL, nR, guided):
    L, R, _ = synth.pair(3 * nL + nR, max(nL, 300), max(nR, 300))
    L, R = L[:nL].copy(), R[:nR].copy()
    for k in range(0, min(nL, nR), 2):  # exact partners, some of them twice
        R[(7 * k + 3) % nR] = L[k]
    for k in range(0, min(nL, nR) - 1, 9):
        R[nR - 1 - k] = R[k]
        L[nL - 1 - k // 2] = L[k // 2]
    L[nL // 2] = 0  # a descriptor whose scores are all 0
    m = v3dm_mod.SIFTMatching(0, v3dm_mod.KERNEL_TCGEN05)
    m.allocate(nL, nR, guided)
    try:
        m.set_left_features(L)
        m.set_right_features(R)
        for ms, mr in ((0.7, 0.8), (0.5, 1.0), (0.7, -1.0), (-1.0, 1.5), (-1.0, -1.0)):
            for _ in range(2):
                np.testing.assert_array_equal(m.find_putative_matches(ms, mr), oracle_mod.match(L, R, ms, mr))
    finally:
        m.close()
