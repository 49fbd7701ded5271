"""The packed camera records that the linearisation and the costs read follow the parameters wherever these
are written: at creation, by accepted steps, by set_params and by reset_params; every model, at camera counts
around the block size of the packing kernel.

Same parameters give the same records and so the same cost to the last bit.  Against the C restatement, a
residual of order one is the difference of two coordinates of order 1e3, so each squared term agrees to
1e3 * 1e-16 * 10 operations = 1e-12 and the sum of these non-negative terms to 1e-11 (relative)."""
import numpy as np
import pytest

from oracle.bindings import Restatement
from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu

MODELS = {
    "std": lambda n: scenes.circle_scene(n_cams=n, n_points=6 * n, obs_per_point=2, seed=n),
    "common": lambda n: scenes.sequence_scene(n_cams=n, n_points=6 * n, min_track=2, max_track=2, seed=n),
    "varying": lambda n: scenes.varying_scene(n_cams=n, n_points=6 * n, seed=n),
    "stereo": lambda n: scenes.stereo_rig_scene(n_poses=n, n_points=6 * n, seed=n),
}


@pytest.mark.parametrize("n", [2, 127, 128, 129])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_records_follow_the_parameters(name, n):
    sc = MODELS[name](n)
    h, other = capi.Handle.from_scene(sc), capi.Handle.from_scene(sc)
    c0 = h.cost()
    ref = Restatement().cost(sc)
    assert abs(c0 - ref) <= 1e-11 * ref
    r = h.minimize(max_iterations=3)
    assert r.cost < c0
    p = h.get_params()
    c1 = h.cost()
    other.set_params(*p)
    assert other.cost() == c1
    assert np.array_equal(h.reduced_system(1.0)[1], other.reduced_system(1.0)[1])
    h.reset_params()
    assert h.cost() == c0
    h.close()
    other.close()
