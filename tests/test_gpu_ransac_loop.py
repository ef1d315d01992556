"""The RANSAC loop on the GPU against the same loop on the host, one candidate after the other
(tests/ransac_loop_host.cpp, the library's solver, pose recovery and refinement in double without
fused multiply-adds), with the refinement and without.  The GPU's five-point solver is built with
fused multiply-adds, so its solutions agree to about 1e-12 and a near-tie of two costs may be
decided the other way: the same model on >= 90% of the pairs (as the refined loop is held to the
reference), and there the same inlier flags, the model to 1e-6 (1e-12 through a refinement that
stops at steps of 1e-8).  Sizes lie at the edges of the refinement's chunks of 224 inliers and of
256 threads, and of its lists (few and many correspondences, one pair and many); a call on many
pairs must equal the calls on each pair bit for bit."""
import ctypes as C
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT
from v3dm import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def loop(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    out = tmp_path_factory.mktemp("loop") / "libransac_loop.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", str(PKG / "csrc"),
                    str(ROOT / "tests" / "ransac_loop_host.cpp"), "-o", str(out)], check=True, capture_output=True,
                   text=True)
    fn = C.CDLL(str(out)).host_ransac

    def run(corrs, K, thr, n_samples, samples, refine):
        inv = np.linalg.inv(K)
        norm = np.empty((corrs.shape[0], 4))
        for v in range(2):
            h = np.c_[corrs[:, 2 * v:2 * v + 2].astype(np.float64), np.ones(corrs.shape[0])] @ inv[v].T
            norm[:, 2 * v:2 * v + 2] = h[:, :2] / h[:, 2:]
        model, flags, n_in = np.zeros(31), np.zeros(corrs.shape[0], np.uint8), C.c_int(0)
        c, inv, s = np.ascontiguousarray(corrs), np.ascontiguousarray(inv), np.ascontiguousarray(samples, np.int32)
        chosen = fn(corrs.shape[0], c.ctypes.data_as(C.c_void_p), norm.ctypes.data_as(C.c_void_p),
                    inv.ctypes.data_as(C.c_void_p), C.c_double(thr), n_samples, s.shape[0],
                    s.ctypes.data_as(C.c_void_p), int(refine), model.ctypes.data_as(C.c_void_p), C.byref(n_in),
                    flags.ctypes.data_as(C.c_void_p))
        return chosen, model, n_in.value, flags

    return run


def _samples(rng, n, k):
    return np.stack([rng.choice(n, 5, replace=False) for _ in range(k)]).astype(np.int32)


@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("sizes,n_draw,inliers", [
    ([6, 7, 12, 31, 33, 64], 60, 0.9),
    ([223, 224, 225, 226, 255, 256, 257, 300], 150, 0.7),
    ([447, 448, 449, 672, 673, 1500, 2200], 260, 0.5),
    ([400], 1001, 0.3),
])
def test_the_loop_equals_the_host_loop(v3dm_mod, loop, sizes, n_draw, inliers, refine):
    rng = np.random.default_rng(sum(sizes) + n_draw)
    parts, Ks, samples = [], [], []
    for i, n in enumerate(sizes):
        off, c, K, _, _, _ = synth.two_view_pairs(1000 + 17 * n + i, n_pairs=1, n_min=n, n_max=n,
                                                  inlier_min=inliers, inlier_max=inliers)
        parts.append(c)
        Ks.append(K[0])
        samples.append(_samples(rng, n, n_draw))
    off = np.r_[0, np.cumsum(sizes)].astype(np.int32)
    corrs, K, smp = np.concatenate(parts), np.stack(Ks), np.stack(samples)
    with v3dm_mod.Ransac() as r:
        r.set_refinement(refine)
        got = r.essential(off, corrs, K, 2.0, 1000, samples=smp)
        for p in range(len(sizes)):  # each pair by itself: the same bits
            one = r.essential(off[p:p + 2] - off[p], parts[p], K[p:p + 1], 2.0, 1000, samples=smp[p:p + 1])
            np.testing.assert_array_equal(one["models"][0], got["models"][p])
            np.testing.assert_array_equal(one["flags"], got["flags"][off[p]:off[p + 1]])
    agree = 0
    for p, n in enumerate(sizes):
        chosen, model, n_in, flags = loop(parts[p], K[p], 2.0, 1000, smp[p], refine)
        if chosen < 0 or got["n_inliers"][p] < 0:
            agree += chosen < 0 and got["n_inliers"][p] < 0
            continue
        e, h = got["E"][p].reshape(-1), model[:9]
        e, h = e / np.linalg.norm(e), h / np.linalg.norm(h)
        if min(np.abs(e - h).max(), np.abs(e + h).max()) > 1e-6:
            continue
        agree += 1
        assert got["n_inliers"][p] == n_in
        np.testing.assert_array_equal(got["flags"][off[p]:off[p + 1]], flags)
        np.testing.assert_allclose(got["error"][p], model[30], rtol=1e-6)
        assert np.abs(got["R"][p].reshape(-1) - model[18:27]).max() < 1e-6
    assert agree >= 0.9 * len(sizes) - 1e-9, (agree, len(sizes))
