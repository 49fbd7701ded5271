"""A problem of a batch has the same result, bit for bit, whatever is beside it in the batch and however many
threads it runs on: alone, among others, in a part of a divided job, beside a problem of four cameras, and
with every schedule.  Points at the edges of the tiles of 32 and of the 256 of the largest block, and tracks
that name a camera twice."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, distributed, scenes

pytestmark = pytest.mark.gpu

POINTS = [6, 31, 32, 33, 64, 65, 127, 129, 255, 256, 257, 300, 511, 513, 800]


def _twice(sc):
    again = np.flatnonzero(sc.point % 5 == 0)
    o = np.argsort(np.concatenate([sc.point, sc.point[again]]), kind="stable")
    return scenes.Scene(sc.model, sc.mode, sc.inlier_threshold, sc.K, sc.R, sc.T, sc.X,
                        np.concatenate([sc.meas, sc.meas[again] + 0.3])[o], np.concatenate([sc.view, sc.view[again]])[o],
                        np.concatenate([sc.point, sc.point[again]])[o])


@pytest.fixture(scope="module")
def problems():
    out = [scenes.triplet_batch(n_triplets=1, min_points=n, max_points=n, seed=n)[0] for n in POINTS]
    return out + [_twice(out[3]), _twice(out[11])]


def _results(probs, schedule=None, keep=None):
    b = capi.Batch.from_flat(capi.concat_problems(probs))
    if schedule:
        b.set_schedule(*schedule)
    res, _ = b.minimize(max_iterations=5)
    out = [(r.status, r.iterations, r.n_rejected, r.cost, r.initial_cost, r.lambda_, b.get_params(i))
           for i, r in enumerate(res[:keep])]
    b.close()
    return out


def _same(a, b):
    assert len(a) == len(b)
    for i, (x, y) in enumerate(zip(a, b)):
        assert x[:-1] == y[:-1], i
        for p, q in zip(x[-1], y[-1]):
            np.testing.assert_array_equal(p, q, err_msg=str(i))


@pytest.fixture(scope="module")
def alone(problems):
    return [_results([p])[0] for p in problems]


@pytest.mark.parametrize("copies", [1, 20, 80])
def test_among_others(problems, alone, copies):
    """17, 340 and 1360 problems: the sizes that get 256, 128 and 64 threads by default."""
    _same(_results(problems * copies, keep=len(problems)), alone)


@pytest.mark.parametrize("schedule", [(64, 64, 0), (128, 128, 0), (256, 256, 0), (256, 64, 5), (128, 64, 9)])
def test_schedules(problems, alone, schedule):
    _same(_results(problems, schedule), alone)


@pytest.mark.parametrize("schedule", [None, (64, 64, 0), (128, 128, 0)])
def test_beside_four_cameras(problems, alone, schedule):
    four = scenes.circle_scene(n_cams=4, n_points=40, obs_per_point=4, seed=3)
    _same(_results(problems + [four], schedule, keep=len(problems)), alone)


def test_divided_job(problems, alone):
    for ranks in (2, 5):
        parts = []
        for r in range(ranks):
            first, last = distributed.shard_range(len(problems), r, ranks)
            parts += _results(problems[first:last])
        _same(parts, alone)


def test_stage():
    trips = scenes.triplet_stage_batch(n_triplets=700, min_tracks=30, max_tracks=300, seed=4)
    every = capi.triplet_stage_flat(capi.concat_triplets(trips))
    of = np.concatenate([[0], np.cumsum([t.n_tracks for t in trips])])
    for first, last in ((0, 1), (5, 9), (100, 420)):
        part = capi.triplet_stage_flat(capi.concat_triplets(trips[first:last]))
        for k in ("verdict", "n_points", "status", "iterations", "cost", "R", "T"):
            np.testing.assert_array_equal(part[k], every[k][first:last])
        np.testing.assert_array_equal(part["X"], every["X"][of[first]:of[last]])
