"""Edges of the float side pass: rows of two 128-descriptor blocks, tiles of 128 columns, and a
pair's few rows cut into segments of tiles whose top twos are merged.

Descriptors of the exact u/512 form go through the float path (hi exact, lo = 0), so its scores are
the integer ones and the expected matches are the oracle's, equal without a tolerance.  Copies of one
descriptor far apart make ties across tiles and segments: the first column wins, and the copy is the
second value that refuses it."""
import numpy as np
import pytest

from v3dm import synth

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 127), (127, 128), (128, 129), (129, 1), (255, 257), (256, 256), (257, 383), (1, 4096),
          (300, 5000), (5000, 300), (513, 3969), (4097, 130)]


def features(nL, nR):
    L, R, lp, rp, F, _ = synth.stereo(nL * 7 + nR, max(nL, 300), max(nR, 300))
    L, R, lp, rp = L[:nL].copy(), R[:nR].copy(), lp[:nL], rp[:nR]
    n = min(nL, nR)
    for k in range(0, n, 3):  # exact partners, in another order
        R[(k * 5 + 1) % nR] = L[k]
    for k in range(0, n - 1, 11):  # and a tie of one of them, far away
        R[nR - 1 - k] = R[k]
        L[nL - 1 - k // 2] = L[k // 2]
    return L, R, lp, rp, F


@pytest.mark.parametrize("nL,nR", SHAPES)
def test_edges_of_rows_tiles_and_segments(v3dm_mod, oracle_mod, nL, nR):
    L, R, lp, rp, F = features(nL, nR)
    m = v3dm_mod.SIFTMatching(0, v3dm_mod.KERNEL_TCGEN05)
    m.allocate(nL, nR, True)
    try:
        m.set_left_features_bf16x3(L.astype(np.float32) / 512)
        m.set_right_features_bf16x3(R.astype(np.float32) / 512)
        # minRatio 1: the copies' ties pass; 0.8: they do not
        for ms, mr in ((0.7, 0.8), (0.5, 1.0), (0.7, -1.0)):
            for _ in range(2):  # the merges leave their counters as they found them
                np.testing.assert_array_equal(m.find_putative_matches(ms, mr), oracle_mod.match(L, R, ms, mr))
        got = m.run_guided_matching(F, 2.0, lp, rp, 0.7, 0.8)
        np.testing.assert_array_equal(
            got, oracle_mod.match(L, R, 0.7, 0.8, gates=[("F", F, 2.0)], lpos=lp, rpos=rp))
        exact = (L.astype(np.int64) @ R.astype(np.int64).T).astype(np.float32) * np.float32(2.0 ** -18)
        np.testing.assert_array_equal(m.scores_f32(), exact)
    finally:
        m.close()


@pytest.mark.parametrize("nL,nR,ms", [(127, 129, 0.0), (300, 1000, 0.1), (1500, 1400, 0.3)])
def test_guided_with_most_scores_above_the_threshold(v3dm_mod, oracle_mod, nL, nR, ms):
    """Low thresholds: nearly every score is tested against the gate, many per descriptor and tile."""
    L, R, lp, rp, F = features(nL, nR)
    m = v3dm_mod.SIFTMatching(0, v3dm_mod.KERNEL_TCGEN05)
    m.allocate(nL, nR, True)
    try:
        m.set_left_features_bf16x3(L.astype(np.float32) / 512)
        m.set_right_features_bf16x3(R.astype(np.float32) / 512)
        for thr in (2.0, 400.0):  # 400: half of them pass
            oracle = oracle_mod.match(L, R, ms, 1.0, gates=[("F", F, thr)], lpos=lp, rpos=rp)
            np.testing.assert_array_equal(m.run_guided_matching(F, thr, lp, rp, ms, 1.0), oracle)
            m.find_putative_matches(ms, 1.0)  # drops the gate
    finally:
        m.close()
