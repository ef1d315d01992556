"""Failure path of the tensor-core side pass, exercised without faulting the GPU.

Every device wait of the side kernel is bounded.  The matcher's test hook makes CTA 0's producer
leave one B tile unloaded and shortens the waits, so the MMA issuer's wait for that tile runs
out: the CTA aborts (every role stops, waits for its own copies and MMAs in flight, frees TMEM),
the other CTAs finish, and the call reports V3DM_ERR_TIMEOUT.  The handle must stay usable: with
the hook off, the next calls give the oracle's pairs.  The reference has no such path: it prints
and exits on any CUDA error (v3d_cudamatching.cu:12-27)."""
import numpy as np
import pytest

from v3dm import synth

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_reports_timeout_and_the_handle_recovers(v3dm_mod, oracle_mod):
    # 6000 x 5600 with 128 x 256 tiles: 47 x 22 tiles over 148 CTAs, so CTA 0 loads six B tiles
    L, R, lp, rp, F, _ = synth.stereo(23, 6000, 5600)
    exp = oracle_mod.match(L, R, 0.7, 0.8)
    exp_g = oracle_mod.match(L, R, 0.7, 0.8, gates=[("F", F, 2.0)], lpos=lp, rpos=rp)
    with v3dm_mod.SIFTMatching(0) as m:
        m.allocate(6000, 5600, True)
        m.set_config(0)
        m.set_left_features(L)
        m.set_right_features(R)
        np.testing.assert_array_equal(m.find_putative_matches(0.7, 0.8), exp)
        for skip in (1, 3):
            m.test_wait_fault(20_000_000, skip)  # ~10 ms at the B200's clocks
            m.profile(True)
            status = v3dm_mod.OK
            try:
                m.find_putative_matches(0.7, 0.8)
            except v3dm_mod.V3DMError as e:
                status = e.status
            pass_a_ms, _ = m.profile_read(0)
            m.profile(False)
            print(f"skip {skip}: status {status}, pass A {pass_a_ms:.3f} ms")
            assert status == v3dm_mod.ERR_TIMEOUT, (status, pass_a_ms)
            assert pass_a_ms >= 5.0  # the pass lasted as long as the shortened wait
            # a guided call after the failed pass recomputes it (the cached pass is incomplete)
            m.test_wait_fault(0, 0)
            np.testing.assert_array_equal(m.run_guided_matching(F, 2.0, lp, rp, 0.7, 0.8), exp_g)
            np.testing.assert_array_equal(m.find_putative_matches(0.7, 0.8), exp)


def test_short_wait_limit_alone_does_not_fail_a_call(v3dm_mod, oracle_mod):
    """A wait limit well above a tile's latency, with every load issued, changes nothing."""
    L, R, _ = synth.pair(24, 2000, 2100)
    with v3dm_mod.SIFTMatching(0) as m:
        m.allocate(2000, 2100)
        m.set_left_features(L)
        m.set_right_features(R)
        m.test_wait_fault(200_000_000, 0)
        np.testing.assert_array_equal(m.find_putative_matches(0.7, 0.8), oracle_mod.match(L, R, 0.7, 0.8))
        m.test_wait_fault(0, 0)


def test_hook_arguments(v3dm_mod):
    with v3dm_mod.SIFTMatching(0) as m:
        for args in ((-1, 0), (10, -1), (0, 2)):
            with pytest.raises(v3dm_mod.V3DMError) as e:
                m.test_wait_fault(*args)
            assert e.value.status == v3dm_mod.ERR_ARG


@pytest.mark.parametrize("bf,depth,floats", [(4, 6, False), (10, 4, False), (3, 4, False), (10, 4, True), (50, 3, True)])
def test_a_tree_wait_that_runs_out_reports_timeout_and_the_handle_recovers(v3dm_mod, oracle_mod, bf, depth, floats):
    """The first phase of a vocabulary-tree descent loses an item on a handle whose sorting buffers were
    never written: the phases behind it do nothing, the call reports V3DM_ERR_TIMEOUT (the device-resident
    call through wait()), and the next calls give the oracle's ids."""
    import torch
    n = 150_001
    rng = synth.rng_for(8200 + bf + floats)
    count = v3dm_mod.voctree_counts(bf, depth)[0]
    nodes, keys = synth.sift_like(rng, count), synth.sift_like(rng, n)
    if floats:
        nodes, keys = synth.unit_sift(rng, count), synth.unit_sift(rng, n)
    exp = oracle_mod.voctree(bf, depth, nodes, keys, False)
    with v3dm_mod.VocabularyTreeTraversal(bf, depth) as t:
        t.allocate(n)
        t.set_nodes(nodes)
        d_keys = torch.from_numpy(keys).cuda()
        d_ids = torch.empty(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        call = t.quantize_f32_device if floats else t.quantize_device
        t.test_wait_fault(20_000_000, 1)  # ~10 ms at the B200's clocks
        with pytest.raises(v3dm_mod.V3DMError) as e:
            t.traverse_tree(keys, v3dm_mod.LEAF_LOCAL)
        assert e.value.status == v3dm_mod.ERR_TIMEOUT and t.last_launches() > 1
        call(n, d_keys.data_ptr(), d_ids.data_ptr(), v3dm_mod.LEAF_LOCAL)
        with pytest.raises(v3dm_mod.V3DMError) as e:
            t.wait()
        assert e.value.status == v3dm_mod.ERR_TIMEOUT
        t.test_wait_fault(0, 0)
        np.testing.assert_array_equal(t.traverse_tree(keys, v3dm_mod.LEAF_LOCAL), exp)
        call(n, d_keys.data_ptr(), d_ids.data_ptr(), v3dm_mod.LEAF_LOCAL)
        t.wait()
        np.testing.assert_array_equal(d_ids.cpu().numpy(), exp)
        for args in ((-1, 0), (10, -1), (0, 2)):
            with pytest.raises(v3dm_mod.V3DMError) as e:
                t.test_wait_fault(*args)
            assert e.value.status == v3dm_mod.ERR_ARG


@pytest.mark.parametrize("nL,nR", [(300, 6000), (7000, 500), (9000, 9000)])
def test_a_float_wait_that_runs_out_reports_timeout_and_the_handle_recovers(v3dm_mod, oracle_mod, nL, nR):
    """Float descriptors: the rows of a CTA that gives up are not decided, and the kernels that read the
    decisions (never written on this handle, or left by a call with more rights) take none of them for
    an index past the rights.  300 lefts: a row in segments, whose merge never comes; 9000: two mutual kernels."""
    rng = synth.rng_for(8300 + nL)
    L, R = synth.unit_sift(rng, nL), synth.unit_sift(rng, nR)
    k = min(nL, nR) // 3
    R[:k] = L[rng.permutation(nL)[:k]]
    with v3dm_mod.SIFTMatching(0) as m:
        m.allocate(nL, nR)
        m.set_left_features(L)
        m.set_right_features(R)
        for _ in range(2):
            m.test_wait_fault(20_000_000, 1)
            with pytest.raises(v3dm_mod.V3DMError) as e:
                m.find_putative_matches(0.7, 0.8)
            assert e.value.status == v3dm_mod.ERR_TIMEOUT
            m.test_wait_fault(0, 0)
            got = m.find_putative_matches(0.7, 0.8)
            assert got.shape[0] >= 0.9 * k
            # fewer rights: the decisions of the call before name rights past them
            m.set_right_features(R[:40])
            m.test_wait_fault(20_000_000, 1)
            with pytest.raises(v3dm_mod.V3DMError) as e:
                m.find_putative_matches(0.7, 0.8)
            assert e.value.status == v3dm_mod.ERR_TIMEOUT
            m.test_wait_fault(0, 0)
            m.set_right_features(R)
            np.testing.assert_array_equal(m.find_putative_matches(0.7, 0.8), got)
