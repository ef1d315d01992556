"""Performance cases of the SIFT matching library: what a structure-from-motion program has it do,
through the public Python entry points, from one thumbnail pair to a 200-image batch.

The kinds follow the stages such a program runs, one after the other:
  pair       one image pair, putative and (optionally) F-guided matching (``SIFTMatching``);
  batch      many image pairs in one call, putative or guided with one F per pair (``BatchMatching``);
  voctree    visual words of descriptors (``VocabularyTreeTraversal``);
  retrieval  the candidate pairs of an image sequence from its visual words (``Retrieval``);
  ransac     the relative orientation of many pairs (``Ransac``), plain or refined (the apps' mode);
  proposal   batched matching through the learned candidate proposal (``Projection``).

Descriptors are SIFT-like: Gamma(0.6) components, unit length, clamped at 0.2 and renormalised; as
bytes u = round(512 x), or as the unit-length floats the feature extractors store.  Sizes are those
of the benchmark workloads and of the tests.
"""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "eth-v3d-lgpl_b200"))
import v3dm  # noqa: E402

MIN_SCORE, MIN_RATIO = 0.7, 0.8
WIDTH, HEIGHT, FOCAL = 1600.0, 1200.0, 1200.0


def listed():
    return [
        # A thumbnail pair through the drop-in calls with host arrays, as the apps make them: latency.
        {"name": "pair_u8_512x480_host", "kind": "pair", "dtype": "u8", "n_left": 512, "n_right": 480,
         "guided": False, "host": True},
        # One ordinary pair, descriptors on the device (a loader's).
        {"name": "pair_u8_4096", "kind": "pair", "dtype": "u8", "n_left": 4096, "n_right": 4096,
         "guided": False, "host": False},
        # One large pair, putative then guided with its fundamental matrix.
        {"name": "pair_u8_16384_guided", "kind": "pair", "dtype": "u8", "n_left": 16384, "n_right": 16384,
         "guided": True, "host": False},
        # The extractors' floats through the drop-in calls with host arrays, ragged sizes, both calls.
        {"name": "pair_f32_7013x6450_host", "kind": "pair", "dtype": "f32", "n_left": 7013, "n_right": 6450,
         "guided": True, "host": True},
        # All pairs of a 200-image set with uneven feature counts: the largest matching call.
        {"name": "batch_u8_200", "kind": "batch", "dtype": "u8", "n_images": 200, "n_min": 1000, "n_max": 12000,
         "guided": False},
        # A small set with ragged, partly tiny images, guided after orientation.
        {"name": "batch_u8_24_guided", "kind": "batch", "dtype": "u8", "n_images": 24, "n_min": 5, "n_max": 2600,
         "guided": True},
        # All pairs of a set of float images (what the extractors write), ordinary feature counts.
        {"name": "batch_f32_40", "kind": "batch", "dtype": "f32", "n_images": 40, "n_min": 1000, "n_max": 8000,
         "guided": False},
        # Visual words of a whole collection on a deep byte tree.
        {"name": "voctree_u8_10x6_2M", "kind": "voctree", "dtype": "u8", "branch": 10, "depth": 6, "n": 2_000_000},
        # Visual words of an image set on the voctree app's tree shape, float centres and keys.
        {"name": "voctree_f32_50x3_300k", "kind": "voctree", "dtype": "f32", "branch": 50, "depth": 3, "n": 300_007},
        # The candidate pairs of a 4096-image sequence.
        {"name": "retrieval_4096", "kind": "retrieval", "n_images": 4096, "n_min": 2000, "n_max": 6000,
         "n_leaves": 125_000, "n_best": 20},
        # The relative orientation of 256 pairs with the refinement the apps switch on.
        {"name": "ransac_256_refined", "kind": "ransac", "n_pairs": 256, "n_min": 500, "n_max": 3000, "refine": True},
        # All pairs of a set through the learned proposal, at its measured operating point.
        {"name": "proposal_60x8000", "kind": "proposal", "n_images": 60, "n_features": 8000, "cells": 128,
         "probes": 4},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["pair", "pair", "batch", "batch", "voctree", "voctree", "retrieval", "ransac", "proposal"])
    if kind == "pair":
        return {"kind": kind, "dtype": rng.choice(["u8", "f32"]), "n_left": _log(rng, 33, 16384),
                "n_right": _log(rng, 33, 16384), "guided": rng.random() < 0.5, "host": rng.random() < 0.5}
    if kind == "batch":
        n_max = _log(rng, 200, 12000)
        return {"kind": kind, "dtype": rng.choice(["u8", "u8", "f32"]), "n_images": _log(rng, 3, 60),
                "n_min": rng.randint(1, n_max), "n_max": n_max, "guided": rng.random() < 0.5}
    if kind == "voctree":
        branch, depth = rng.choice([(10, 6), (10, 5), (10, 4), (50, 3), (5, 4)])
        dtype = rng.choice(["u8", "f32"])
        return {"kind": kind, "dtype": dtype, "branch": branch, "depth": depth,
                "n": _log(rng, 1000, 2_000_000 if dtype == "u8" else 1_000_000)}
    if kind == "retrieval":
        n_max = _log(rng, 500, 6000)
        return {"kind": kind, "n_images": _log(rng, 32, 4096), "n_min": rng.randint(n_max // 4, n_max),
                "n_max": n_max, "n_leaves": rng.choice([10_000, 100_000, 125_000]), "n_best": rng.randint(5, 100)}
    if kind == "ransac":
        n_max = _log(rng, 60, 3000)
        return {"kind": kind, "n_pairs": _log(rng, 1, 256), "n_min": rng.randint(max(20, n_max // 4), n_max),
                "n_max": n_max, "refine": rng.random() < 0.5}
    return {"kind": kind, "n_images": _log(rng, 6, 60), "n_features": _log(rng, 1000, 8000),
            "cells": rng.choice([64, 128, 256]), "probes": rng.randint(2, 5)}


# ---- inputs ------------------------------------------------------------------------------------


class _Gen:
    """Random numbers on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator("cuda").manual_seed(int(seed))
        self.host = np.random.Generator(np.random.PCG64(int(seed)))

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=torch.float32):
        return torch.rand(shape, generator=self.g, device="cuda", dtype=dtype) * (hi - lo) + lo

    def normal(self, *shape, dtype=torch.float32):
        return torch.randn(shape, generator=self.g, device="cuda", dtype=dtype)

    def ints(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device="cuda")

    def perm(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")

    def sift(self, n):
        """n unit-length float descriptors."""
        x = torch._standard_gamma(torch.full((n, 128), 0.6, device="cuda"), generator=self.g)
        x = torch.nn.functional.normalize(x).clamp_max_(0.2)
        return torch.nn.functional.normalize(x)

    def seen_again(self, x):
        """Another observation of the descriptors x: N(0, 8/512) noise per component."""
        return torch.nn.functional.normalize((x + self.normal(*x.shape) * (8.0 / 512)).clamp_(0.0, 0.5))

    def positions(self, n):
        return self.uniform(n, 2) * torch.tensor([WIDTH, HEIGHT], device="cuda")


def _as(x, dtype):
    return x.contiguous() if dtype == "f32" else (x * 512.0).round_().clamp_(0, 255).to(torch.uint8)


def _counts(g, c, n):
    """n counts spread evenly over the case's range, in random order: their sum is the same for every seed."""
    spread = np.rint(np.linspace(c["n_min"], c["n_max"], n) if n > 1 else np.array([c["n_max"]]))
    return g.host.permutation(spread.astype(np.int64))


def _yaw(a):
    c, s = np.cos(a), np.sin(a)
    return np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]])


def _fundamental(rot, t, f=FOCAL):
    ki = np.linalg.inv(np.array([[f, 0, WIDTH / 2], [0, f, HEIGHT / 2], [0, 0, 1.0]]))
    tx = np.array([[0, -t[2], t[1]], [t[2], 0, -t[0]], [-t[1], t[0], 0]])
    return ki.T @ tx @ rot @ ki


def _project(X, rot, t):
    """Pixels of points X (n, 3) in the camera (rot, t), with 1 px noise left to the caller."""
    Y = X @ torch.tensor(rot.T, device="cuda", dtype=X.dtype) + torch.tensor(t, device="cuda", dtype=X.dtype)
    return Y[:, :2] / Y[:, 2:] * FOCAL + torch.tensor([WIDTH / 2, HEIGHT / 2], device="cuda", dtype=X.dtype)


def _pair_inputs(c, seed):
    """Two views: 30% of the right features are left features seen again, where a stereo rig puts them."""
    g = _Gen(seed)
    nl, nr = c["n_left"], c["n_right"]
    L, lpos = g.sift(nl), g.positions(nl)
    k = min(int(round(0.3 * nr)), nl)
    src = g.perm(nl)[:k]
    R = torch.cat([g.seen_again(L[src]), g.sift(nr - k)])
    rot = _yaw(np.deg2rad(g.host.uniform(-10, 10)))
    t = -rot @ np.array([0.3, 0.0, 0.0])
    z = g.uniform(k, 1, lo=2.0, hi=20.0)
    X = torch.cat([(lpos[src] - torch.tensor([WIDTH / 2, HEIGHT / 2], device="cuda")) / FOCAL * z, z], 1)
    rpos = torch.cat([_project(X, rot, t) + g.normal(k, 2), g.positions(nr - k)])
    order = g.perm(nr)
    return _as(L, c["dtype"]), _as(R[order], c["dtype"]), lpos, rpos[order].contiguous(), _fundamental(rot, t)


def _images(c, seed, track_frac):
    """An image set with cameras along a line: track_frac of every image's features are observations
    of shared points, about five images per point."""
    g = _Gen(seed)
    n = c["n_images"]
    counts = _counts(g, c, n) if "n_min" in c else np.full(n, c["n_features"])
    slots = np.rint(track_frac * counts).astype(int)
    n_tracks = max(1, int(slots.sum()) // 5)
    base = g.sift(n_tracks)
    X = torch.stack([g.uniform(n_tracks, lo=-6.0, hi=6.0 + 0.3 * n), g.uniform(n_tracks, lo=-4.0, hi=4.0),
                     g.uniform(n_tracks, lo=4.0, hi=20.0)], 1)
    rots = [_yaw(np.deg2rad(a)) for a in g.host.uniform(-10, 10, n)]
    centres = [np.array([0.3 * i, 0.0, 0.0]) for i in range(n)]
    desc, pos = [], []
    for i in range(n):
        m = int(counts[i])
        tr = g.perm(n_tracks)[:slots[i]]
        k = int(tr.shape[0])
        order = g.perm(m)
        d = torch.cat([g.seen_again(base[tr]), g.sift(m - k)])[order]
        desc.append(_as(d, c.get("dtype", "u8")))
        pos.append(torch.cat([_project(X[tr], rots[i], -rots[i] @ centres[i]) + g.normal(k, 2),
                              g.positions(m - k)])[order])
    return torch.cat(desc), counts.astype(np.int32), torch.cat(pos), rots, centres


def _tree(g, bf, depth, floats, n_train):
    """A hierarchical k-means tree (breadth-first node order): per node bf of its members, one k-means
    step; sums in fixed point, so that the centres depend on the seed alone."""
    data = g.sift(n_train)
    if not floats:
        data = (data * 512.0).round_().clamp_(0, 255)
    scale = float(1 << 24) if floats else 1.0
    parent, levels, n_par = torch.zeros(n_train, dtype=torch.int64, device="cuda"), [], 1
    for _ in range(depth):
        order = torch.argsort(parent, stable=True)
        cnt = torch.bincount(parent, minlength=n_par)
        start = torch.cumsum(cnt, 0) - cnt
        pick = start[:, None] + (g.uniform(n_par, bf) * cnt[:, None].clamp(min=1)).long()
        cent = data[order[pick.clamp(max=n_train - 1)]]  # (n_par, bf, 128)
        noise = g.normal(*cent.shape) * (4.0 / 512 if floats else 4.0)
        cent = (cent + noise).abs_() if floats else (cent + noise).round_().clamp_(0, 255)

        def assign():
            child = torch.empty_like(parent)
            step = max(1, (1 << 26) // (bf * 128))
            for s in range(0, n_train, step):
                sc = torch.bmm(cent[parent[s:s + step]], data[s:s + step].unsqueeze(2)).squeeze(2)
                child[s:s + step] = sc.argmax(1)
            return parent * bf + child

        idx = assign()
        sums = torch.zeros(n_par * bf, 128, dtype=torch.int64, device="cuda")
        sums.index_add_(0, idx, (data * scale).round().long())
        num = torch.bincount(idx, minlength=n_par * bf)
        mean = (sums.double() / num.clamp(min=1)[:, None] / scale).float()
        mean = mean if floats else mean.round_().clamp_(0, 255)
        cent = torch.where((num > 0)[:, None], mean, cent.reshape(-1, 128)).reshape(n_par, bf, 128)
        parent = assign()
        levels.append(cent.reshape(-1, 128))
        n_par *= bf
    nodes = torch.cat(levels)
    return (nodes if floats else nodes.to(torch.uint8)).cpu().numpy()


def _words(c, seed):
    """Visual words of an image sequence: 42% of an image's words come from a window of scene points
    that slides along the sequence, the others from all leaves, popular ones more often (Zipf 0.5)."""
    g = _Gen(seed)
    n, leaves = c["n_images"], c["n_leaves"]
    counts = _counts(g, c, n)
    off = np.zeros(n + 1, np.int32)
    off[1:] = np.cumsum(counts)
    total = int(off[-1])
    cdf = torch.cumsum(torch.arange(1, leaves + 1, device="cuda", dtype=torch.float64) ** -0.5, 0)
    cdf /= cdf[-1].clone()
    popular = g.perm(leaves)

    def zipf(m):
        return popular[torch.searchsorted(cdf, g.uniform(m, dtype=torch.float64)).clamp_(max=leaves - 1)]

    window = max(8, int(counts.mean() * 0.42))
    step = max(1, window // 8)
    point = zipf(step * (n - 1) + window)
    image = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.tensor(counts, device="cuda"))
    seen = point[image * step + g.ints(window, total)]
    words = torch.where(g.uniform(total) < 0.42, seen, zipf(total))
    return off, words.to(torch.int32)


def _correspondences(c, seed):
    """Putative correspondences of image pairs: a random rig each, 30-80% inliers with 0.5 px noise."""
    g = _Gen(seed)
    n = c["n_pairs"]
    counts = _counts(g, c, n)
    off = np.zeros(n + 1, np.int32)
    off[1:] = np.cumsum(counts)
    K = np.zeros((n, 2, 3, 3))
    corrs = []
    for p in range(n):
        f, m = float(g.host.uniform(900, 1500)), int(counts[p])
        K[p, :] = np.array([[f, 0, WIDTH / 2], [0, f, HEIGHT / 2], [0, 0, 1.0]])
        rot = _yaw(np.deg2rad(g.host.uniform(-15, 15)))
        t = -rot @ np.array([g.host.uniform(0.2, 0.6), 0.0, 0.0])
        k = int(round(m * g.host.uniform(0.3, 0.8)))
        uv = g.host.uniform(0, 1, (m, 2)) * [WIDTH, HEIGHT]
        X = np.c_[(uv - [WIDTH / 2, HEIGHT / 2]) / f, np.ones(m)] * g.host.uniform(3, 12, (m, 1))
        Y = X @ rot.T + t
        q = Y[:, :2] / Y[:, 2:] * f + [WIDTH / 2, HEIGHT / 2]
        q[k:] = g.host.uniform(0, 1, (m - k, 2)) * [WIDTH, HEIGHT] - g.host.normal(0, 0.5, (m - k, 2))
        corrs.append((np.c_[uv, q] + g.host.normal(0, 0.5, (m, 4)))[g.host.permutation(m)])
    return off, np.concatenate(corrs).astype(np.float32), K


# ---- cases -------------------------------------------------------------------------------------


class _State:
    """A case's inputs, handle and output buffers."""


class _Kept:
    """A program's own array that a call's rows (pairs, triples) are put into: as many rows as a case
    can give, -1 past the last one, and their number."""

    def __init__(self, rows, width):
        self.rows, self.n = np.full((rows, width), -1, np.int32), 0

    def put(self, got):
        n = got.shape[0]
        m = min(n, self.rows.shape[0])
        self.rows[:m] = got[:m]
        self.rows[m:self.n] = -1
        self.n = m
        return [self.rows, n]


def _most_triples(c):
    """More triples than all pairs of a set have: twice the shared points two images see, and chance matches."""
    n = c["n_images"]
    m = (c["n_min"] + c["n_max"]) / 2 if "n_min" in c else c["n_features"]
    frac = 0.3 if c.get("guided") else 0.15
    return int(n * (n - 1) / 2 * (2 * frac * m * min(1.0, 5 / n) + 0.01 * m + 64))


def _prepare_pair(s, c, seed):
    L, R, lpos, rpos, s.F = _pair_inputs(c, seed)
    s.m = v3dm.SIFTMatching(0)
    s.m.allocate(c["n_left"], c["n_right"], c["guided"])
    n = min(c["n_left"], c["n_right"])
    if c["host"]:
        L, R, lpos, rpos = (x.cpu().numpy() for x in (L, R, lpos, rpos))
        s.kept = [_Kept(n, 2) for _ in range(2)]
    else:
        s.pairs = [torch.full((n, 2), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
        s.count = torch.zeros(2, dtype=torch.int32, device="cuda")
    s.L, s.R, s.lpos, s.rpos = L, R, lpos, rpos


def _run_pair(s, c):
    m = s.m
    if c["host"]:
        m.set_left_features(s.L)
        m.set_right_features(s.R)
        out = s.kept[0].put(m.find_putative_matches(MIN_SCORE, MIN_RATIO))
        if c["guided"]:
            out += s.kept[1].put(m.run_guided_matching(s.F, 2.0, s.lpos, s.rpos, MIN_SCORE, MIN_RATIO))
        return out
    if c["dtype"] == "f32":
        m.set_left_features_f32_device(s.L.data_ptr(), c["n_left"])
        m.set_right_features_f32_device(s.R.data_ptr(), c["n_right"])
    else:
        m.set_left_features_device(s.L.data_ptr(), c["n_left"])
        m.set_right_features_device(s.R.data_ptr(), c["n_right"])
    m.putative_device(MIN_SCORE, MIN_RATIO, s.pairs[0].data_ptr(), s.count.data_ptr())
    if not c["guided"]:
        m.wait()
        return [s.pairs[0], s.count[:1]]
    m.guided_F_device(s.F, 2.0, s.lpos.data_ptr(), s.rpos.data_ptr(), MIN_SCORE, MIN_RATIO, s.pairs[1].data_ptr(),
                      s.count.data_ptr() + 4)
    m.wait()
    return [s.pairs[0], s.pairs[1], s.count]


def _prepare_batch(s, c, seed):
    s.desc, s.counts, pos, rots, centres = _images(c, seed, 0.3 if c["guided"] else 0.15)
    s.b = v3dm.BatchMatching(0)
    s.dtype = np.float32 if c["dtype"] == "f32" else np.uint8
    s.b.set_images_device(s.desc.data_ptr(), s.counts, s.dtype)
    s.b.set_pairs()
    s.kept = _Kept(_most_triples(c), 3)
    if c["guided"]:
        s.pos = pos.cpu().numpy()
        n = c["n_images"]
        s.F = np.stack([_fundamental(rots[j] @ rots[i].T, rots[j] @ (centres[i] - centres[j]))
                        for i in range(n) for j in range(i + 1, n)])


def _run_batch(s, c):
    s.b.set_images_device(s.desc.data_ptr(), s.counts, s.dtype)
    if not c["guided"]:
        return s.kept.put(s.b.match(MIN_SCORE, MIN_RATIO))
    s.b.set_positions(s.pos)
    return s.kept.put(s.b.match_guided(s.F, 2.0, MIN_SCORE, MIN_RATIO))


def _prepare_voctree(s, c, seed):
    g = _Gen(seed)
    floats = c["dtype"] == "f32"
    s.t = v3dm.VocabularyTreeTraversal(c["branch"], c["depth"], 0)
    s.t.allocate(c["n"])
    s.t.set_nodes(_tree(g, c["branch"], c["depth"], floats, 500_000 if c["depth"] == 6 else 200_000))
    s.keys = _as(g.sift(c["n"]), c["dtype"])
    s.ids = torch.empty(c["n"], dtype=torch.int32, device="cuda")


def _run_voctree(s, c):
    call = s.t.quantize_f32_device if c["dtype"] == "f32" else s.t.quantize_device
    call(c["n"], s.keys.data_ptr(), s.ids.data_ptr(), v3dm.LEAF_LOCAL)
    return s.ids


def _prepare_retrieval(s, c, seed):
    s.off, s.words = _words(c, seed)
    s.r = v3dm.Retrieval(0)
    s.docs = torch.empty(c["n_images"], c["n_best"], dtype=torch.int32, device="cuda")
    s.scores = torch.empty(c["n_images"], c["n_best"], dtype=torch.float32, device="cuda")


def _run_retrieval(s, c):
    s.r.binomial_device(c["n_leaves"], s.off, s.words.data_ptr(), 0.1, c["n_best"], s.docs.data_ptr(),
                        s.scores.data_ptr())
    s.r.wait()
    return {"docs": s.docs, "scores": s.scores}


def _prepare_ransac(s, c, seed):
    s.off, corrs, s.K = _correspondences(c, seed)
    s.seed = int(seed)
    s.r = v3dm.Ransac(0)
    s.r.set_refinement(c["refine"])
    s.corrs = torch.from_numpy(corrs).cuda()
    s.models = torch.empty(c["n_pairs"], 31, dtype=torch.float64, device="cuda")
    s.n_in = torch.empty(c["n_pairs"], dtype=torch.int32, device="cuda")
    s.flags = torch.empty(corrs.shape[0], dtype=torch.uint8, device="cuda")


def _run_ransac(s, c):
    s.r.essential_device(s.off, s.corrs.data_ptr(), s.K, 2.0, 1000, 1001, None, s.seed, s.models.data_ptr(),
                         s.n_in.data_ptr(), s.flags.data_ptr())
    s.r.wait()
    return {"models": s.models, "n_inliers": s.n_in, "flags": s.flags}


def _prepare_proposal(s, c, seed):
    s.desc, s.counts = _images(c, seed, 0.15)[:2]
    s.b = v3dm.BatchMatching(0)
    s.b.set_config(0, 2)
    s.b.set_images_device(s.desc.data_ptr(), s.counts)
    s.b.set_pairs()
    s.kept = _Kept(_most_triples(c), 3)
    s.p = v3dm.Projection(0, seed=int(seed) & 0xffff)
    # the cells: spherical k-means of embedded descriptors
    z = torch.from_numpy(s.p.embed(s.desc[:: max(1, s.desc.shape[0] // 20000)].cpu().numpy())).cuda()
    cent = z[: c["cells"]].clone()
    for _ in range(8):
        member = torch.nn.functional.one_hot((z @ cent.T).argmax(1), c["cells"]).to(z.dtype)
        cent = torch.nn.functional.normalize(member.T @ z + 1e-3 * cent)
    s.p.set_cells(cent.cpu().numpy())


def _run_proposal(s, c):
    s.b.set_images_device(s.desc.data_ptr(), s.counts)
    return s.kept.put(s.b.match_proposal(s.p, c["probes"], MIN_SCORE, MIN_RATIO, probes_right=c["probes"]))


_PREPARE = {"pair": _prepare_pair, "batch": _prepare_batch, "voctree": _prepare_voctree,
            "retrieval": _prepare_retrieval, "ransac": _prepare_ransac, "proposal": _prepare_proposal}
_RUN = {"pair": _run_pair, "batch": _run_batch, "voctree": _run_voctree, "retrieval": _run_retrieval,
        "ransac": _run_ransac, "proposal": _run_proposal}


def prepare(case, seed):
    s = _State()
    s.case = dict(case)
    _PREPARE[case["kind"]](s, case, seed)
    torch.cuda.synchronize()
    return s


def run(state):
    return _RUN[state.case["kind"]](state, state.case)


def work(case):
    """Bytes and operations of one pass (2 per multiply-add), at the mean of random counts."""
    k = case["kind"]
    size = 4 if case.get("dtype") == "f32" else 1
    if k == "pair":
        nl, nr = case["n_left"], case["n_right"]
        return {"bytes": (nl + nr) * (128 * size + 8 * case["guided"]) + 8 * min(nl, nr) * (1 + case["guided"]),
                "flops": 256.0 * nl * nr}
    if k in ("batch", "proposal"):
        n = case["n_images"]
        m = (case["n_min"] + case["n_max"]) / 2 if k == "batch" else case["n_features"]
        pairs = n * (n - 1) / 2
        flops = 256.0 * m * m * pairs
        if k == "proposal":  # the share of scores that share a probed cell
            flops *= min(1.0, case["probes"] ** 2 / case["cells"])
        return {"bytes": n * m * 128 * size + pairs * 12 * 0.02 * m + 76 * pairs * case.get("guided", False),
                "flops": flops}
    if k == "voctree":
        bf, d, n = case["branch"], case["depth"], case["n"]
        nodes = sum(min(bf ** (i + 1), n * bf) for i in range(d))
        return {"bytes": n * (128 * size + 4) + nodes * 128 * size, "flops": 256.0 * bf * d * n}
    if k == "retrieval":
        n, m = case["n_images"], (case["n_min"] + case["n_max"]) / 2
        # every word's list of earlier images is a bit row
        return {"bytes": n * m * 4 + n * case["n_best"] * 8 + case["n_leaves"] * n / 8, "flops": n * n / 2 * 10}
    m = (case["n_min"] + case["n_max"]) / 2
    samples = 250  # the adaptive budget's mean over the inlier shares
    return {"bytes": case["n_pairs"] * (m * 17 + 400), "flops": case["n_pairs"] * samples * (4 * 35 * m + 20000)}


def exact(case, seed):
    """The retrieval scores in 64 bits.  Every other output is whole numbers, or (the orientation) the
    outcome of a search that has no value in closed form."""
    if case["kind"] != "retrieval":
        return None
    off, words = _words(case, seed)
    n, leaves, best = case["n_images"], case["n_leaves"], case["n_best"]
    counts = torch.tensor(np.diff(off), device="cuda")
    image = torch.repeat_interleave(torch.arange(n, device="cuda"), counts)
    common = torch.zeros(n, n, dtype=torch.float64, device="cuda")  # [query, document]
    step = max(1, (1 << 28) // n)
    for w0 in range(0, leaves, step):
        sel = (words >= w0) & (words < w0 + step)
        hist = torch.zeros(n, min(step, leaves - w0), device="cuda")
        hist.index_put_((image[sel], words[sel].long() - w0), torch.ones((), device="cuda"), accumulate=True)
        common += (hist @ (hist > 0).float().T).double()
    nf = counts.double()
    p0 = torch.maximum(nf[:, None], nf[None, :]) / leaves
    p1 = (p0 + 0.1).clamp(max=1.0)
    m = torch.minimum(nf[:, None], nf[None, :])
    score = (common * p0.log() + (m - common) * (1 - p0).log()) - (common * p1.log() + (m - common) * (1 - p1).log())
    earlier = torch.arange(n, device="cuda")[None, :] < torch.arange(n, device="cuda")[:, None]
    score = torch.where(earlier, score, torch.inf).sort(1).values[:, :best]
    if score.shape[1] < best:
        score = torch.nn.functional.pad(score, (0, best - score.shape[1]), value=torch.inf)
    return {"docs": None, "scores": torch.where(torch.isinf(score), 0.0, score)}
