"""Retrieval counts at the edges of the counting: numbers of words around the 64 rows after which a
carry ripples, many groups of threads per column (few images) and few (many), and bitmaps on either
side of 4 GB (byte and word offsets).  Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(v3dm_mod, oracle_mod, leaves, counts, words, n_best):
    off = np.zeros(len(counts) + 1, np.int32)
    off[1:] = np.cumsum(counts)
    exp = oracle_mod.retrieval(leaves, off, words, 0.1, n_best)
    with v3dm_mod.Retrieval() as r:
        docs, scores = r.binomial(leaves, off, words, 0.1, n_best)
    np.testing.assert_array_equal(docs, exp[0])
    np.testing.assert_array_equal(scores.view(np.uint32), exp[1].view(np.uint32))


@pytest.mark.parametrize("n_images", [3, 33, 200, 1100])
@pytest.mark.parametrize("n", [15, 16, 17, 1023, 1025, 4097])
def test_counts(v3dm_mod, oracle_mod, n_images, n):
    rng = np.random.default_rng(n_images * 10007 + n)
    counts = np.full(n_images, 20)
    counts[[0, n_images // 2, n_images - 1]] = n
    words = rng.integers(0, 64, int(counts.sum())).astype(np.int32)  # few words: large counts
    _check(v3dm_mod, oracle_mod, 6000, counts, words, min(5, n_images))


@pytest.mark.parametrize("leaves", [(1 << 32) // 400 - 2, (1 << 32) // 400 + 2])
def test_bitmap_around_four_gigabytes(v3dm_mod, oracle_mod, leaves):
    """3200 images: 100 words, 400 bytes per leaf."""
    rng = np.random.default_rng(7)
    counts = rng.integers(3, 40, 3200)
    words = (leaves - 1 - rng.integers(0, 300, int(counts.sum()))).astype(np.int32)
    _check(v3dm_mod, oracle_mod, leaves, counts, words, 7)


@pytest.mark.parametrize("n_images,n,leaves", [(1100, 400, 400_000), (1100, 400, 10_000), (33, 1023, 10_000), (33, 1023, 16_000),
                                               (3, 4097, 150_000), (3, 4097, 300_000), (3, 33_000, 200_000), (3, 66_000, 100_000),
                                               (3, 66_000, 120_000_000)])
def test_counts_where_groups_add_for_themselves_and_where_they_are_added_up(v3dm_mod, oracle_mod, n_images, n, leaves):
    """Both ways of emptying the counters, chosen by words, groups and leaves, with queries of more rows than the
    counters hold (32752) among them; n / leaves + 0.1 < 1, so that the scores are finite."""
    rng = np.random.default_rng(n_images * 10007 + n)
    counts = np.full(n_images, 20)
    counts[[0, n_images - 2, n_images - 1]] = n
    words = rng.integers(0, 64, int(counts.sum())).astype(np.int32)
    _check(v3dm_mod, oracle_mod, leaves, counts, words, min(5, n_images))
