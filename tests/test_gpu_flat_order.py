"""Flat batches whose observations are not in point order go to the host's layout without an upload first, and
give the problems that the host's layout gives."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu


def _shuffled(flat, first):
    """The observations of the problems from `first` on in random order within each problem."""
    owner = np.repeat(np.arange(len(flat["n_obs"])), flat["n_obs"])
    key = np.where(owner >= first, np.random.default_rng(1).random(len(owner)), np.arange(len(owner)) / len(owner))
    o = np.lexsort((key, owner))
    return dict(flat, view=flat["view"][o], point=flat["point"][o], meas=np.ascontiguousarray(flat["meas"][o]))


def _create(flat):
    before = capi.launch_count()
    b = capi.Batch.from_flat(flat)
    launches = capi.launch_count() - before
    res, _ = b.minimize(max_iterations=3)
    out = [r.cost for r in res]
    b.close()
    return launches, out


@pytest.mark.parametrize("first", [0, 3])
def test_out_of_order_from_the_start(first):
    flat = capi.concat_problems(scenes.triplet_batch(n_triplets=60, min_points=100, max_points=500, seed=5))
    assert flat["n_obs"].sum() + flat["n_points"].sum() >= 32768
    launches, cost = _create(flat)
    assert launches > 0                  # checked and laid out on the device
    launches, shuffled = _create(_shuffled(flat, first))
    assert launches == 0
    np.testing.assert_allclose(shuffled, cost, rtol=1e-9)


def test_out_of_order_at_the_end():
    flat = capi.concat_problems(scenes.triplet_batch(n_triplets=60, min_points=100, max_points=500, seed=5))
    _, cost = _create(flat)
    _, shuffled = _create(_shuffled(flat, 59))
    np.testing.assert_allclose(shuffled, cost, rtol=1e-9)
