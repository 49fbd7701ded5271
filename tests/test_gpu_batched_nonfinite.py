"""Batched problems whose cameras hold values that are no numbers or overflow: the same status, iterations and
rejected steps as the C restatement's run of each problem, a cost that is no number, and the other problems
of the batch as they are without them.  Infinite translations end at once by the update test, whose length is
then infinite; the restatement, which sums that length another way, rejects the steps."""
import numpy as np
import pytest

from oracle.bindings import Restatement
from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu


def _twice(sc):
    o = np.argsort(np.concatenate([sc.point, sc.point]), kind="stable")
    return scenes.Scene(sc.model, sc.mode, sc.inlier_threshold, sc.K, sc.R, sc.T, sc.X, np.concatenate([sc.meas, sc.meas + 0.2])[o],
                        np.concatenate([sc.view, sc.view])[o], np.concatenate([sc.point, sc.point])[o])


def _run(probs, threads=None):
    b = capi.Batch(probs)
    if threads:
        b.set_schedule(threads, threads, 0)
    res, _ = b.minimize(max_iterations=3)
    out = [((r.status, r.iterations, r.n_rejected), r.cost, b.get_params(i)) for i, r in enumerate(res)]
    b.close()
    return out


@pytest.fixture(scope="module")
def problems():
    three = scenes.triplet_batch(n_triplets=3, min_points=40, max_points=70, seed=1)
    return three + [_twice(three[0])]


@pytest.mark.parametrize("threads", [None, 64, 128])
@pytest.mark.parametrize("camera", [0, 1, 2])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e160, 1e200])
def test_status(problems, value, camera, threads):
    sound = _run(problems, threads)
    for k in (0, 3):
        bad = list(problems)
        bad[k] = problems[k].copy()
        bad[k].T = np.array(problems[k].T)
        bad[k].T[camera, 1] = value
        got = _run(bad, threads)
        if np.isinf(value):
            want = (capi.STATUS_SMALL_UPDATE, 0, 0)
        else:
            _, info = Restatement().minimize(bad[k], max_iterations=3)
            want = (info["status"], info["iterations"], info["n_rejected"])
        assert got[k][0] == want
        assert np.isnan(got[k][1])
        for i in range(len(problems)):
            if i != k:
                assert got[i][:2] == sound[i][:2]
                for a, b in zip(got[i][2], sound[i][2]):
                    np.testing.assert_array_equal(a, b)
