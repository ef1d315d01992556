"""What a batch handle keeps from call to call: the pair table's part of guided calls, graphs and the pinned
memory that host calls take their triples from."""
import ctypes as C

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


@pytest.mark.parametrize("k", [1000, 32768, 32769, 40000])
def test_triples_around_the_pinned_memory_and_device_calls(v3dm_mod, k):
    """Host calls with 2 k triples, around the 65536 that a call leaves in pinned memory, between device calls on
    the same handle: two pairs of images, each the other's rows in reverse order."""
    import torch
    rng = synth.rng_for(43)
    L = synth.sift_like(rng, k)
    R = L[::-1].copy()
    desc, counts = np.concatenate([L, R, R]), np.array([k, k, k], np.int32)
    one = np.stack([np.arange(k), k - 1 - np.arange(k)], 1)
    exp = np.concatenate([np.c_[np.zeros(k, np.int64), one], np.c_[np.ones(k, np.int64), one]])
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    with v3dm_mod.BatchMatching() as b:
        b.set_images(desc, counts)
        b.set_pairs([(0, 1), (0, 2)])

        def device_call():
            count.zero_()
            torch.cuda.synchronize()
            for _ in range(2):  # a first call may have to grow the buffers
                b.match_device(0.7, 0.8, count.data_ptr())
                if b.wait() == v3dm_mod.OK:
                    break
            torch.cuda.synchronize()
            assert int(count[0]) == 2 * k

        device_call()
        for _ in range(2):
            np.testing.assert_array_equal(b.match(0.7, 0.8), exp)
            device_call()
        b.use_graph(False)
        np.testing.assert_array_equal(b.match(0.7, 0.8), exp)
        device_call()
        # the first rows, when the caller's buffer is smaller
        out = np.full((70000, 3), -1, np.int32)
        n = C.c_longlong(0)
        for cap in (5, min(2 * k, 65537) - 1):
            st = v3dm_mod.lib().v3dm_batch_match(b._h, 0.7, 0.8, out.ctypes.data, cap, C.byref(n))
            assert st == v3dm_mod.ERR_CAPACITY and n.value == 2 * k
            np.testing.assert_array_equal(out[:cap], exp[:cap])
            assert (out[cap:] == -1).all()


def test_proposal_calls_with_projections_made_in_turn(v3dm_mod):
    """Projections made and closed one after the other (each may get the address of the last, but not its device
    buffers): a batch handle's captured call is used only for the projection it was captured with."""
    desc, counts, offs, pos, cams = synth.scene(44, 5, 300, 900)
    rng = synth.rng_for(45)
    with v3dm_mod.BatchMatching() as kept:
        kept.set_images(desc, counts)
        kept.set_pairs(None)
        hold = []
        for k in range(6):
            net = v3dm_mod.Projection(0, seed=100 + k)
            hold.append(v3dm_mod.Projection(0, seed=1))  # takes the buffers that the last one gave back
            cells = rng.normal(0, 1, (16, 32)).astype(np.float32)
            net.set_cells(cells / np.linalg.norm(cells, axis=1, keepdims=True))
            got = kept.match_proposal(net, 2, 0.7, 0.8, probes_right=2)
            with v3dm_mod.BatchMatching() as fresh:
                fresh.set_images(desc, counts)
                fresh.set_pairs(None)
                np.testing.assert_array_equal(got, fresh.match_proposal(net, 2, 0.7, 0.8, probes_right=2))
            net.close()
        for h in hold:
            h.close()
