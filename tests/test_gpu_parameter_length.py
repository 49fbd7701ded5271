"""The parameter length of the update test (|delta| < t (length + t)), summed on the device for large problems,
to one part in a million: the stop flips between t (1 - 1e-6) and t (1 + 1e-6), where t is computed from the
step that one iteration took.  Numbers of coordinates around the 256 threads and the 256 blocks of the sum."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu


def _rotation_vector(R):
    """Logarithm of the (small) rotations R."""
    v = 0.5 * np.stack([R[:, 2, 1] - R[:, 1, 2], R[:, 0, 2] - R[:, 2, 0], R[:, 1, 0] - R[:, 0, 1]], axis=1)
    s = np.linalg.norm(v, axis=1, keepdims=True)
    return v * (np.arcsin(s) / np.where(s > 0, s, 1.0))


@pytest.mark.parametrize("points", [8193, 9000, 21845, 21846, 30001])
def test_update_stop_at_the_parameter_length(points):
    sc = scenes.circle_scene(n_cams=12, n_points=points, obs_per_point=4, seed=points)
    assert sc.n_obs + sc.n_points >= 32768
    h = capi.Handle.from_scene(sc)
    options = dict(max_iterations=1, precision=capi.PRECISION_FP64)
    assert h.minimize(update_threshold=0.0, **options).n_rejected == 0
    _, R, T, _, X = h.get_params()
    w = _rotation_vector(R @ np.asarray(sc.R).transpose(0, 2, 1))
    step = np.sqrt(((T - sc.T) ** 2).sum() + (w ** 2).sum() + ((X - sc.X) ** 2).sum())
    length = np.sqrt((sc.T ** 2).sum() + 3 * sc.n_cams + (sc.X ** 2).sum())
    t = (np.sqrt(length * length + 4 * step) - length) / 2
    for factor, status in ((1 - 1e-6, capi.STATUS_TIMEOUT), (1 + 1e-6, capi.STATUS_SMALL_UPDATE)):
        h.reset_params()
        assert h.minimize(update_threshold=factor * t, **options).status == status
    h.close()
