"""Device memory that a RANSAC handle holds: in proportion to its calls."""
import numpy as np
import pytest

from v3dm import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_draw,refine,mb", [(300, 1001, False, 24), (300, 1001, True, 24), (100_000, 60, True, 64)])
def test_one_pair_holds_little(v3dm_mod, n, n_draw, refine, mb):
    """One pair: sample slots for its draws (1.6 KB each: 2 MB for 1001), inlier lists for the refinements it can
    have at once (sixteen, 4 bytes per correspondence: 6 MB for 100000), and about 80 bytes per correspondence.  Each of
    some twenty-five buffers is rounded up, by up to 2 MB where it is large."""
    import torch
    off, corrs, K, R, t, inl = synth.two_view_pairs(12, n_pairs=1, n_min=n, n_max=n, inlier_min=0.7, inlier_max=0.8)
    with v3dm_mod.Ransac(0) as r:  # the runtime's own allocations
        r.set_refinement(refine)
        r.essential(off, corrs, K, 2.0, n_draw, seed=1)
    with v3dm_mod.Ransac(0) as r:
        r.set_refinement(refine)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        res = r.essential(off, corrs, K, 2.0, n_draw, seed=1)
        held = before - torch.cuda.mem_get_info()[0]
    print(f"{held / 2**20:.1f} MB")
    assert held <= mb << 20
    assert int(res["n_inliers"][0]) > n // 2
    assert float(np.linalg.norm(res["R"][0] - R[0])) < 0.05
