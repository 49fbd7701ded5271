"""The Schur complement by groups of points that the same cameras see (FP64 blocks) against the one
from the lists of observation pairs, on the same handle inputs: every model and camera dimension, tracks
in any order, cameras named twice in a track, fixed parameters, chunks of one point up to several
chunks per group.

The two ways sum the same terms in another order and factor (V + lambda I) instead of inverting it by
cofactors.  With lambda at 1e-3 of the largest diagonal entry the point blocks have condition numbers of
at most about 1e3, and a camera block sums about 1e3 terms no larger than the diagonal, so the entries
agree to 1e-16 * 1e3 * 1e2 = 1e-11 of the largest one."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu


def _shuffled(sc, seed):
    o = np.random.default_rng(seed).permutation(sc.n_obs)
    sc.view, sc.point, sc.meas = sc.view[o], sc.point[o], sc.meas[o]
    return sc


def _repeated(sc):
    again = np.flatnonzero(sc.point % 3 == 0)
    sc.view = np.concatenate([sc.view, sc.view[again]])
    sc.point = np.concatenate([sc.point, sc.point[again]])
    sc.meas = np.concatenate([sc.meas, sc.meas[again] + 0.3])
    return sc


SCENES = {
    "common7": lambda: scenes.sequence_scene(n_cams=20, n_points=2500, seed=1),
    "common0_norot": lambda: scenes.sequence_scene(n_cams=16, n_points=1500, seed=2,
                                                   mode=scenes.FULL_BUNDLE_NO_ROTATIONS),
    "shuffled": lambda: _shuffled(scenes.sequence_scene(n_cams=20, n_points=2500, seed=3), 3),
    "repeated": lambda: _repeated(scenes.sequence_scene(n_cams=12, n_points=900, seed=4, mode=scenes.FULL_BUNDLE_FOCAL_LENGTH)),
    "std_scattered": lambda: scenes.circle_scene(n_cams=9, n_points=700, seed=5),
    "long_tracks": lambda: scenes.sequence_scene(n_cams=48, n_points=400, min_track=20, max_track=24, seed=6),
    "stereo": lambda: scenes.stereo_rig_scene(n_poses=25, n_points=2000, seed=7),
    "varying7": lambda: scenes.varying_scene(n_cams=12, n_points=800, mode=scenes.FULL_BUNDLE_FOCAL_LENGTH, seed=8),
    "varying9": lambda: scenes.varying_scene(n_cams=12, n_points=800, mode=scenes.FULL_BUNDLE_FOCAL_LENGTH_PP, seed=9),
    "varying11": lambda: scenes.varying_scene(n_cams=12, n_points=800, mode=scenes.FULL_BUNDLE_RADIAL, seed=10),
    "varying13": lambda: scenes.varying_scene(n_cams=12, n_points=800, seed=11),
}


def _system(sc, fixed, how, monkeypatch):
    monkeypatch.setenv("V3DBA_SCHUR", how)
    h = capi.Handle.from_scene(sc)
    h.set_nonvarying(*fixed)
    S, _ = h.reduced_system(1e4)
    lam = 1e-3 * np.abs(np.diag(S)).max()
    out = h.reduced_system(lam)
    h.close()
    return out


@pytest.mark.parametrize("fixed", [(0, 0, 0), (2, 40, 0)], ids=["free", "fixed"])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_groups_equal_pairs(name, fixed, monkeypatch):
    sc = SCENES[name]()
    Sp, bp = _system(sc, fixed, "pairs", monkeypatch)
    Sg, bg = _system(sc, fixed, "groups", monkeypatch)
    assert not np.array_equal(Sp, Sg)   # another order of summation: the groups ran
    assert np.abs(Sg - Sp).max() <= 1e-11 * np.abs(Sp).max()
    assert np.abs(bg - bp).max() <= 1e-11 * np.abs(bp).max()


def test_minimize_by_groups_matches_pairs(monkeypatch):
    """A whole FP64 run, large enough for the groups without being forced."""
    sc = scenes.sequence_scene(n_cams=60, n_points=10000, seed=12)
    out = []
    for how in ("pairs", None):
        if how:
            monkeypatch.setenv("V3DBA_SCHUR", how)
        else:
            monkeypatch.delenv("V3DBA_SCHUR")
        h = capi.Handle.from_scene(sc)
        r = h.minimize(max_iterations=8, precision=capi.PRECISION_FP64)
        out.append((r, h.get_params()))
        h.close()
    (ra, pa), (rb, pb) = out
    assert (ra.status, ra.iterations, ra.n_rejected) == (rb.status, rb.iterations, rb.n_rejected)
    for a, b in zip(pa, pb):
        assert np.abs(a - b).max() <= 1e-9 * max(np.abs(a).max(), 1.0)
