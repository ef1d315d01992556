"""The error of split scores (BF16 hi + lo on the tensor cores, FP32 accumulation), against FP64.

The float vocabulary-tree descent decides a level from such scores when they differ by more than a bound, and the
bound assumes that the tensor core loses no more in one accumulation of 17 terms than 17 truncations to the 24 bits of
an FP32 sum would.  NVIDIA documents no figure for that, so it is measured here, on inputs made to lose as
much as they can: terms just below the last bit of a large sum, alternating signs, magnitudes over many
binades."""
import numpy as np
import pytest

from v3dm import synth

pytestmark = pytest.mark.gpu

# of sum |x_i y_i|: the lo . lo term and the rounding of both lo, 3 * 2^-18; 24 accumulations of 17 terms, each
# addition truncated to FP32, 408 * 2^-23
BOUND = 3 * 2.0 ** -18 + 408 * 2.0 ** -23


def _inputs(kind, rng, n):
    if kind == "unit":
        return synth.unit_sift(rng, n), synth.unit_sift(rng, n)
    if kind == "signs":
        return rng.normal(0, 1, (n, 128)).astype(np.float32), rng.normal(0, 1, (n, 128)).astype(np.float32)
    if kind == "binades":
        x = rng.choice([-1.0, 1.0], (2, n, 128)) * rng.uniform(1, 2, (2, n, 128)) * 2.0 ** rng.integers(-24, 1, (2, n, 128))
        return x[0].astype(np.float32), x[1].astype(np.float32)
    # one large product per 16 values (one K step) or in the first of them only, the others just below a fraction of its
    # last bit; all of one sign, so that truncations add up
    x = np.full((n, 128), 1.0)
    y = np.empty((n, 128))
    for r in range(n):
        y[r] = 2.0 ** -(16 + r % 12) * rng.uniform(0.9, 0.999)
        big = np.arange(0, 128, 16) if (r // 12) % 2 else np.array([0])
        y[r, big] = rng.uniform(1, 2, big.size)
        if kind == "late" and (r // 24) % 2:
            y[r] = y[r, ::-1]
    return x.astype(np.float32), y.astype(np.float32)


@pytest.mark.parametrize("kind", ["unit", "signs", "binades", "early", "late"])
def test_split_scores_stay_within_the_bound(v3dm_mod, kind):
    rng = synth.rng_for(51)
    n = 384
    x, y = _inputs(kind, rng, n)
    with v3dm_mod.SIFTMatching(0) as m:
        m.allocate(n, n)
        m.set_left_features_bf16x3(x)
        m.set_right_features_bf16x3(y)
        s = m.scores_f32().astype(np.float64)
    exact = x.astype(np.float64) @ y.astype(np.float64).T
    err = np.abs(s - exact) / (np.abs(x).astype(np.float64) @ np.abs(y).astype(np.float64).T)
    print(f"{kind}: largest error {err.max():.2e} of sum |x y|, bound {BOUND:.2e}")
    assert err.max() <= BOUND
