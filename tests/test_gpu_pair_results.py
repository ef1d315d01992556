"""Where a pair call's results go: calls captured into a graph, and more pairs than a host call's
pinned memory holds."""
import ctypes as C

import numpy as np
import pytest

from v3dm import synth

pytestmark = pytest.mark.gpu


class _Graph:
    """What a call enqueues on a handle's stream, captured and replayed (relaxed capture mode)."""

    def __init__(self, stream, enqueue):
        self.rt, self.stream = C.CDLL("libcudart.so.12"), C.c_void_p(stream)
        graph, self.exe = C.c_void_p(), C.c_void_p()
        assert self.rt.cudaStreamBeginCapture(self.stream, 2) == 0
        enqueue()
        assert self.rt.cudaStreamEndCapture(self.stream, C.byref(graph)) == 0
        assert self.rt.cudaGraphInstantiate(C.byref(self.exe), graph, C.c_ulonglong(0)) == 0
        assert self.rt.cudaGraphDestroy(graph) == 0

    def launch(self):
        assert self.rt.cudaGraphLaunch(self.exe, self.stream) == 0

    def close(self):
        assert self.rt.cudaGraphExecDestroy(self.exe) == 0


@pytest.mark.parametrize("n,floats", [(500, False), (9000, False), (700, True)])
def test_captured_call(v3dm_mod, oracle_mod, n, floats):
    """A call captured before any other has run: a wait that comes before the graph has nothing to report,
    whatever an earlier handle left in the memory; replays and host calls in turn give the same pairs."""
    import torch
    L, R, _ = synth.pair(31, n, n)
    with v3dm_mod.SIFTMatching(0) as m:  # a handle whose last call failed
        m.allocate(n, n)
        m.set_left_features(L)
        m.set_right_features(R)
        m.test_wait_fault(20_000_000, 1)
        with pytest.raises(v3dm_mod.V3DMError):
            m.find_putative_matches(0.7, 0.8)
    exp = oracle_mod.match(L, R, 0.7, 0.8)
    with v3dm_mod.SIFTMatching(0) as m:
        m.allocate(n, n)
        if floats:
            m.set_left_features_bf16x3(L.astype(np.float32) / 512)  # the float pass, same scores
            m.set_right_features_bf16x3(R.astype(np.float32) / 512)
        else:
            m.set_left_features(L)
            m.set_right_features(R)
        pairs = torch.full((n, 2), -1, dtype=torch.int32, device="cuda")
        count = torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        g = _Graph(m.stream(), lambda: m.putative_device(0.7, 0.8, pairs.data_ptr(), count.data_ptr()))
        m.wait()
        assert int(count[0]) == 0
        for k in range(3):
            pairs.fill_(-1)
            torch.cuda.synchronize()
            g.launch()
            m.wait()
            torch.cuda.synchronize()
            np.testing.assert_array_equal(pairs[: int(count[0])].cpu().numpy(), exp)
            if k != 1:
                np.testing.assert_array_equal(m.find_putative_matches(0.7, 0.8), exp)
        g.close()


@pytest.mark.parametrize("k", [16383, 16384, 16385, 20000])
def test_pairs_around_the_pinned_memory(v3dm_mod, k):
    """Host calls with k pairs, around the 16384 that a call leaves in pinned memory: every left's own row on the
    other side, in reverse order."""
    rng = synth.rng_for(32)
    L = synth.sift_like(rng, k)
    R = L[::-1].copy()
    with v3dm_mod.SIFTMatching(0) as m:
        m.allocate(k, k)
        m.set_left_features(L)
        m.set_right_features(R)
        got = m.find_putative_matches(0.7, 0.8)
        np.testing.assert_array_equal(got, np.stack([np.arange(k), k - 1 - np.arange(k)], 1))
