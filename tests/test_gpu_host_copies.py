"""The copies between the caller's memory and the device: sizes on both sides of the staged path, slot
and page remainders, offsets inside a page, several threads at a time, and handles made and closed in
numbers beyond what the pools keep.  Values are copied, so they are compared exactly."""
import threading

import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu


def _tracks(n, seed):
    rng = np.random.default_rng(seed)
    length = rng.integers(0, 6, size=n)
    ptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
    K = int(ptr[-1])
    return dict(track_ptr=ptr, pos=rng.normal(size=(n, 3)), view=rng.integers(0, 50, size=K, dtype=np.int32),
                id=rng.integers(0, 999, size=K, dtype=np.int32), mpos=rng.uniform(0, 640, size=(K, 2)).astype(np.float32))


def _check(t, required):
    out = capi.bundle_point_structure(t, required)
    length = np.diff(t["track_ptr"])
    keep = (length >= required) & (required >= 0)
    per = np.repeat(keep, length)
    assert np.array_equal(out["points3d"], t["pos"][keep])
    assert np.array_equal(out["measurements"], t["mpos"][per].astype(np.float64))
    assert np.array_equal(out["measurement_ids"], t["id"][per])
    assert np.array_equal(out["corresponding_view"], t["view"][per])
    assert np.array_equal(out["corresponding_point"], np.repeat(np.arange(keep.sum()), length[keep]))
    assert np.array_equal(out["xs_indices"], np.flatnonzero(keep))


@pytest.mark.parametrize("n", [0, 1, 7000, 90001, 233333, 700001])
def test_structure_round_trip(n):
    """Up to 50 MB each way: below, at and beyond the sizes from which copies are staged."""
    _check(_tracks(n, n), 2)


def test_required_beyond_all_and_negative():
    for required in (-1, 0, 9):
        _check(_tracks(1000, 5), required)


def test_threads_share_the_rings():
    """Four threads, so that more ask for rings and helpers than are kept."""
    sets = [_tracks(400000 + 1111 * k, k) for k in range(4)]
    failed = []

    def work(t):
        try:
            for _ in range(2):
                _check(t, 3)
        except BaseException as e:   # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in sets]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_more_handles_than_are_kept():
    sc = scenes.circle_scene(n_cams=5, n_points=100, seed=3)
    hs = [capi.Handle.from_scene(sc) for _ in range(12)]
    want = None
    for _ in range(2):
        costs = []
        for h in hs:
            h.reset_params()
            costs.append(h.minimize(max_iterations=3, precision=capi.PRECISION_FP64).cost)
        want = want or costs[0]
        assert costs == [want] * len(hs)
        for h in hs:
            h.close()
        hs = [capi.Handle.from_scene(sc) for _ in range(12)]
    for h in hs:
        h.close()
