"""Parameters in, out and reset for every model, with few cameras (their arrays go up as one copy) and with
many: what was set is what comes back, a reset brings back what the handle was made from, and a run from set
parameters is the run of a handle made from them, bit for bit."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "std": lambda: scenes.circle_scene(n_cams=6, n_points=151, seed=1),
    "std_many": lambda: scenes.circle_scene(n_cams=500, n_points=3000, seed=2),
    "common": lambda: scenes.sequence_scene(n_cams=12, n_points=501, seed=3),
    "common_many": lambda: scenes.sequence_scene(n_cams=700, n_points=9000, seed=4, mode=0),
    "varying": lambda: scenes.varying_scene(n_cams=9, n_points=303, seed=5),
    "stereo": lambda: scenes.stereo_rig_scene(n_poses=11, n_points=401, seed=6),
}


def _moved(params, seed):
    rng = np.random.default_rng(seed)
    K, R, T, dist, X = [None if p is None else np.array(p) for p in params]
    return K, R, T + 0.01 * rng.normal(size=T.shape), dist, X + 0.01 * rng.normal(size=X.shape)


def _equal(a, b):
    for x, y in zip(a, b):
        if x is not None and y is not None and np.size(x) and np.size(y):
            np.testing.assert_array_equal(np.reshape(x, -1), np.reshape(y, -1))


@pytest.mark.parametrize("name", sorted(SCENES))
def test_set_get_reset(name):
    sc = SCENES[name]()
    h = capi.Handle.from_scene(sc)
    first = h.get_params()
    for array, mine in zip((sc.R, sc.T, sc.X), (first[1], first[2], first[4])):
        np.testing.assert_array_equal(np.reshape(array, -1), np.reshape(mine, -1))
    moved = _moved(first, 1)
    h.set_params(*moved)
    _equal(h.get_params(), moved)
    options = dict(max_iterations=3, precision=capi.PRECISION_FP64, solver=capi.SOLVER_CHOLESKY)
    r = h.minimize(**options)
    after = h.get_params()
    h.reset_params()
    _equal(h.get_params(), first)
    h.close()
    other = sc.copy()
    other.T, other.X = moved[2].reshape(np.shape(sc.T)), moved[4].reshape(np.shape(sc.X))
    h = capi.Handle.from_scene(other)
    q = h.minimize(**options)
    assert (q.cost, q.iterations, q.n_rejected) == (r.cost, r.iterations, r.n_rejected)
    _equal(h.get_params(), after)
    h.close()
