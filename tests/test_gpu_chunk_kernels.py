"""The staged chunk kernels (camera sums, reduced right-hand side and border, Schur sums over the pair
lists) at the remainders of their 32-entry tiles: a single point seen by one or two cameras up to lists
that end one before, at and one after a tile and a chunk, every camera and global dimension, both
precisions, and the two ways through the pair lists.

Gradient blocks and the FP64 system against the C restatement; FP64 sums of at most a few hundred terms
in another order agree to 1e-16 * 1e3 (condition number of a point block at the damping used) * 1e2 = 1e-11
of the largest entry of the blocks they are formed from.  The mixed system rounds each stored block to FP32 (6e-8) and so agrees with the FP64
one to a few times 6e-8 of the undamped diagonal it is subtracted from: 1e-5 with the condition number."""
import numpy as np
import pytest

from oracle.bindings import Restatement
from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu

MODELS = {
    "std": lambda n, m, s: scenes.circle_scene(n_cams=n, n_points=m, obs_per_point=n, seed=s),
    "common7": lambda n, m, s: scenes.sequence_scene(n_cams=n, n_points=m, min_track=n, max_track=n, seed=s),
    "common1": lambda n, m, s: scenes.sequence_scene(n_cams=n, n_points=m, min_track=n, max_track=n, seed=s,
                                                     mode=scenes.FULL_BUNDLE_FOCAL_LENGTH),
    "common3": lambda n, m, s: scenes.sequence_scene(n_cams=n, n_points=m, min_track=n, max_track=n, seed=s,
                                                     mode=scenes.FULL_BUNDLE_FOCAL_LENGTH_PP),
    "common5": lambda n, m, s: scenes.sequence_scene(n_cams=n, n_points=m, min_track=n, max_track=n, seed=s,
                                                     mode=scenes.FULL_BUNDLE_RADIAL),
    "varying13": lambda n, m, s: scenes.varying_scene(n_cams=n, n_points=m, seed=s),
    "varying9": lambda n, m, s: scenes.varying_scene(n_cams=n, n_points=m, mode=scenes.FULL_BUNDLE_FOCAL_LENGTH_PP, seed=s),
}


def _many(sc, copies):
    """The scene next to itself `copies` times: other cameras, so the same blocks in more chunks."""
    n, m = sc.n_cams, sc.n_points
    rep = lambda a: np.concatenate([a] * copies)  # noqa: E731
    per = sc.K.ndim == 3
    return scenes.Scene(sc.model, sc.mode, sc.inlier_threshold, rep(sc.K) if per else sc.K, rep(sc.R), rep(sc.T), rep(sc.X),
                        rep(sc.meas), np.concatenate([sc.view + n * k for k in range(copies)]).astype(np.int32),
                        np.concatenate([sc.point + m * k for k in range(copies)]).astype(np.int32),
                        sc.dist if sc.dist is None or sc.dist.ndim == 1 else rep(sc.dist))


@pytest.mark.parametrize("points", [1, 31, 32, 33, 64, 65, 127, 129])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_system_at_tile_edges(name, points):
    sc = MODELS[name](3, points, 17 + points)
    h = capi.Handle.from_scene(sc)
    S0, _ = h.reduced_system(1e4)
    lam = 1e-3 * np.abs(np.diag(S0)).max()
    S, b = h.reduced_system(lam)
    orc = Restatement()
    blocks = orc.normal_blocks(sc)
    Sr, br, _, _ = orc.reduced_system(sc, blocks, lam)
    # the entries are differences from these
    big_S = max(np.abs(blocks[k]).max() for k in ("U", "X", "Z") if blocks[k].size)
    big_b = max(np.abs(blocks[k]).max() for k in ("ga", "gc") if blocks[k].size)
    assert np.abs(S - Sr).max() <= 1e-11 * big_S
    assert np.abs(b - br).max() <= 1e-11 * big_b
    Sm, bm = h.reduced_system(lam, capi.PRECISION_MIXED)
    assert np.abs(Sm - Sr).max() <= 1e-5 * big_S
    assert np.abs(bm - br).max() <= 1e-5 * big_b
    h.close()


@pytest.mark.parametrize("points", [5, 33, 130])
def test_staged_pair_lists_equal_direct(points):
    """A problem small enough for the direct loads, and copies of it that make enough chunks for the staged
    ones: every copy's blocks are the small problem's, bit for bit with FP32 blocks (the same sums in the
    same order), to rounding with FP64."""
    small = MODELS["std"](4, points, 3)
    copies = 1 + 1184 // 10 + 1     # 10 blocks of at least one chunk each
    big = _many(small, copies)
    hs, hb = capi.Handle.from_scene(small), capi.Handle.from_scene(big)
    for precision, tol in ((capi.PRECISION_MIXED, 0.0), (capi.PRECISION_FP64, 1e-11)):
        S, b = hs.reduced_system(1e3, precision)
        T, c = hb.reduced_system(1e3, precision)
        n = S.shape[0]
        for k in (0, copies // 2, copies - 1):
            at = slice(n * k, n * (k + 1))
            assert np.abs(T[at, at] - S).max() <= tol * np.abs(S).max()
            assert np.abs(c[at] - b).max() <= 1e-12 * np.abs(b).max()
    hs.close()
    hb.close()
