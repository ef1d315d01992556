"""Device memory that a vocabulary tree holds: what its kind of keys needs."""
import ctypes as C

import numpy as np
import pytest

from v3dm import synth

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("as_floats", [False, True])
def test_byte_trees_hold_nothing_for_float_keys_until_they_come(v3dm_mod, oracle_mod, as_floats):
    """A byte tree (given as bytes, or as floats of the form u/512) for a million keys: 128 bytes per key, 512 for the
    staging of float keys, and 16 of indices; 640 MB more only once float keys of other values come, which the
    tensor-core descent then takes with the oracle's ids."""
    bf, depth, n, m = 10, 3, 1_000_000, 30_000
    rng = synth.rng_for(8400)
    nodes = synth.sift_like(rng, v3dm_mod.voctree_counts(bf, depth)[0])
    keys, fkeys = synth.sift_like(rng, m), synth.unit_sift(rng, m)
    exp = oracle_mod.voctree(bf, depth, nodes, keys, False)
    exp_f = oracle_mod.voctree(bf, depth, nodes.astype(np.float32) / 512, fkeys, False)
    with v3dm_mod.VocabularyTreeTraversal(bf, depth) as t:
        t.allocate(1000)
        before = _free()
        t.allocate(n)
        t.set_nodes(nodes.astype(np.float32) / 512 if as_floats else nodes)
        np.testing.assert_array_equal(t.traverse_tree(keys, v3dm_mod.LEAF_LOCAL), exp)
        np.testing.assert_array_equal(t.traverse_tree(keys.astype(np.float32) / 512, v3dm_mod.LEAF_LOCAL), exp)
        held = before - _free()
        print(f"{held / 2**20:.0f} MB")
        assert held < 700 << 20
        np.testing.assert_array_equal(t.traverse_tree(fkeys, v3dm_mod.LEAF_LOCAL), exp_f)
        assert t.last_launches() > 1
        np.testing.assert_array_equal(t.traverse_tree(keys, v3dm_mod.LEAF_LOCAL), exp)


def test_first_float_call_of_a_byte_tree_inside_a_capture(v3dm_mod, oracle_mod):
    """Float keys of other values on a u/512 tree, the call captured before any other: nothing may be
    allocated then, so the one-kernel descent is captured, with the same ids."""
    import torch
    bf, depth, n = 10, 3, 20_000
    rng = synth.rng_for(8500)
    nodes = synth.sift_like(rng, v3dm_mod.voctree_counts(bf, depth)[0]).astype(np.float32) / 512
    keys = synth.unit_sift(rng, n)
    exp = oracle_mod.voctree(bf, depth, nodes, keys, False)
    d_keys = torch.from_numpy(keys).cuda()
    d_ids = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    rt = C.CDLL("libcudart.so.12")
    with v3dm_mod.VocabularyTreeTraversal(bf, depth) as t:
        t.allocate(n)
        t.set_nodes(nodes)
        torch.cuda.synchronize()
        stream, graph, exe = C.c_void_p(t.stream()), C.c_void_p(), C.c_void_p()
        assert rt.cudaStreamBeginCapture(stream, 1) == 0  # this thread's unsafe calls end the capture
        t.quantize_f32_device(n, d_keys.data_ptr(), d_ids.data_ptr(), v3dm_mod.LEAF_LOCAL)
        assert t.last_launches() == 1
        assert rt.cudaStreamEndCapture(stream, C.byref(graph)) == 0
        assert rt.cudaGraphInstantiate(C.byref(exe), graph, C.c_ulonglong(0)) == 0
        assert rt.cudaGraphLaunch(exe, stream) == 0
        t.wait()
        np.testing.assert_array_equal(d_ids.cpu().numpy(), exp)
        d_ids.fill_(-1)
        torch.cuda.synchronize()
        t.quantize_f32_device(n, d_keys.data_ptr(), d_ids.data_ptr(), v3dm_mod.LEAF_LOCAL)  # outside it, the phases
        t.wait()
        assert t.last_launches() > 1
        np.testing.assert_array_equal(d_ids.cpu().numpy(), exp)
        assert rt.cudaGraphExecDestroy(exe) == 0 and rt.cudaGraphDestroy(graph) == 0
