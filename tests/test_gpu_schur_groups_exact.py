"""The grouped Schur complement on numbers that FP64 holds exactly, where the point blocks are singular to
rounding: both ways through the Schur sums have to use one and the same inverse of V + lambda I.

A point (a, 0, 1), a a whole number of 26 bits, is seen by two cameras without rotation, one unit apart, with
focal length 1 and residuals of zero.  Its block V has entries up to 2 a^2 + 2 a + 1 < 2^53 and determinant 2;
lambda is below the last bit of every entry, so the cofactors and the inverse are exact.  Two observations of
the two coordinates x and z say nothing about the cameras' x once the point is eliminated: in the rows of the
translations along x every product and sum is a whole number below 2^53, and nothing is left of U but lambda."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu

LAMBDA = 1e-20


def _scene(points, seed):
    a = np.random.default_rng(seed).choice(np.arange(1 << 25, (1 << 25) + (1 << 23)), size=points, replace=False)
    a = a.astype(np.float64)
    zero, one = np.zeros(points), np.ones(points)
    X = np.stack([a, zero, one], axis=1)
    meas = np.stack([np.stack([a, zero], axis=1), np.stack([a + 1, zero], axis=1)], axis=1)
    T = np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0]])
    eye = np.broadcast_to(np.eye(3), (2, 3, 3)).copy()
    return scenes.Scene(scenes.MODEL_STD, 0, 1.0, eye, eye.copy(), T, X, meas.reshape(-1, 2),
                        np.tile(np.arange(2), points).astype(np.int32), np.repeat(np.arange(points), 2).astype(np.int32), None)


@pytest.mark.parametrize("points", [1, 3, 4, 5, 31, 32, 33, 64, 200])
@pytest.mark.parametrize("how", ["pairs", "groups"])
def test_exact_elimination(how, points, monkeypatch):
    monkeypatch.setenv("V3DBA_SCHUR", how)
    h = capi.Handle.from_scene(_scene(points, points))
    S, _ = h.reduced_system(LAMBDA)
    h.close()
    tx = [0, 6]   # translations along x
    assert np.abs(S[np.ix_(tx, tx)]).max() <= LAMBDA
