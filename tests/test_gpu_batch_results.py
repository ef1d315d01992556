"""What a batch handle keeps from call to call: the pair table's part of guided calls."""
import numpy as np
import pytest

from v3dm import synth

pytestmark = pytest.mark.gpu


def test_guided_calls_with_changing_pair_tables_and_gates(v3dm_mod, oracle_mod):
    """Guided calls on one handle with the pair table replaced between them (more pairs, fewer, another order,
    the same size), other gates for the same table, and another image layout: each call's pairs equal
    the oracle's for its own table and gates."""
    desc, counts, offs, pos, cams = synth.scene(41, 6, 200, 900)
    n = len(counts)
    full = synth.all_pairs(n)
    rng = synth.rng_for(42)
    with v3dm_mod.BatchMatching() as b:
        b.set_images(desc, counts)
        b.set_positions(pos)
        for pairs in (full[:4], full, full[::-1][:4], [full[7]], full[3:7]):
            pairs = np.asarray(pairs, np.int32)
            b.set_pairs(pairs)
            for thr0 in (2.0, 30.0):
                F = np.stack([synth.fundamental(cams, i, j) for i, j in pairs])
                thr = np.full(len(pairs), thr0, np.float32)
                if thr0 > 2.0:  # gates of other pairs
                    F = F[rng.permutation(len(pairs))]
                per = b.split_pairs(b.match_guided(F, thr, 0.7, 0.8))
                for k, (i, j) in enumerate(pairs):
                    exp = oracle_mod.match(desc[offs[i]:offs[i + 1]], desc[offs[j]:offs[j + 1]], 0.7, 0.8,
                                           gates=[("F", F[k], float(thr0))], lpos=pos[offs[i]:offs[i + 1]],
                                           rpos=pos[offs[j]:offs[j + 1]])
                    np.testing.assert_array_equal(per[k], exp, err_msg=f"pair {k} ({i}, {j})")
        # another layout: the pair table has to be set again
        b.set_images(desc[: offs[4]], counts[:4])
        with pytest.raises(v3dm_mod.V3DMError):
            b.match_guided(F, thr, 0.7, 0.8)
