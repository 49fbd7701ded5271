"""Arrays that are checked on the device (large calls): the same refusals as the host's checks of small
calls, for a fault in the first, a middle and the last place, and the same results where the layout is
made on the device."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu


def _code(f):
    with pytest.raises(capi.V3dbaError) as e:
        f()
    return e.value.code


@pytest.fixture(scope="module")
def sequence():
    return scenes.sequence_scene(n_cams=40, n_points=9000, seed=2)


@pytest.mark.parametrize("where", [0, 31999, -1])
@pytest.mark.parametrize("what,value", [("view", -1), ("view", 40), ("point", -1), ("point", 9000), ("meas", np.nan),
                                        ("meas", np.inf), ("X", -np.inf)])
def test_create_refuses(sequence, what, value, where):
    sc = sequence.copy()
    a = getattr(sc, what).reshape(-1)
    a[min(where, a.size - 1)] = value
    assert _code(lambda: capi.Handle.from_scene(sc)) == capi.ERR_INVALID_INPUT
    h = capi.Handle.from_scene(sequence)   # and nothing is left behind
    assert h.minimize(max_iterations=1).iterations == 1
    h.close()


def test_create_refuses_subcamera():
    sc = scenes.stereo_rig_scene(n_poses=60, n_points=6000, seed=1)
    for k in (0, sc.n_obs - 1):
        for v in (-1, 2):
            bad = sc.copy()
            bad.sub = sc.sub.copy()
            bad.sub[k] = v
            assert _code(lambda: capi.Handle.from_scene(bad)) == capi.ERR_INVALID_INPUT


def test_update_stop_scale(sequence):
    """The parameter length of the update test, summed on the device: the same stop on both sides of the
    threshold that it sets."""
    length = np.sqrt((sequence.T ** 2).sum() + 3 * sequence.n_cams + (sequence.X ** 2).sum())
    h = capi.Handle.from_scene(sequence)
    h.minimize(max_iterations=1, precision=capi.PRECISION_FP64)
    before = sequence.params()
    step = np.sqrt(sum(((a - b) ** 2).sum() for a, b in zip(h.get_params()[2:], before[2:])))
    h.reset_params()
    big = h.minimize(max_iterations=1, precision=capi.PRECISION_FP64, update_threshold=1e3 * step / length)
    h.reset_params()
    small = h.minimize(max_iterations=1, precision=capi.PRECISION_FP64, update_threshold=1e-3 * step / length)
    assert (big.status, small.status) == (capi.STATUS_SMALL_UPDATE, capi.STATUS_TIMEOUT)
    h.close()


@pytest.mark.parametrize("where", [0, -1])
def test_rotations_refuse(where):
    g = scenes.rotation_graph(n_views=3000, n_pairs=40000, seed=1)
    for value in (-1, 3000):
        pairs = g.pairs.copy()
        pairs.reshape(-1)[where] = value
        assert _code(lambda: capi.refine_consistent_rotations(g.rel, pairs, g.R0)) == capi.ERR_INVALID_INPUT
    for name in ("rel", "R0"):
        arrays = dict(rel=g.rel.copy(), R0=g.R0.copy())
        arrays[name].reshape(-1)[where] = np.nan
        assert _code(lambda: capi.refine_consistent_rotations(arrays["rel"], g.pairs, arrays["R0"])) == capi.ERR_INVALID_INPUT


def test_stage_refuses():
    flat = capi.concat_triplets(scenes.triplet_stage_batch(n_triplets=100, seed=3))
    assert flat["tracks_of"][-1] >= 32768
    for where in (0, -1):
        for key, value in (("view", 3), ("view", -1), ("pos", np.nan), ("pos", np.inf)):
            bad = dict(flat, **{key: flat[key].copy()})
            bad[key].reshape(-1)[where] = value
            assert _code(lambda: capi.triplet_stage_flat(bad)) == capi.ERR_INVALID_INPUT
    ptr = flat["track_ptr"].copy()
    ptr[5] = ptr[6] + 1
    assert _code(lambda: capi.triplet_stage_flat(dict(flat, track_ptr=ptr))) == capi.ERR_INVALID_INPUT


def _solve(flat):
    b = capi.Batch.from_flat(flat)
    res, _ = b.minimize(max_iterations=3)
    out = b.get_all_params()
    b.reset()
    again = b.get_all_params()
    b.close()
    return [r.cost for r in res], out, again


def test_batch_layout():
    """The layout made on the device against the host's (problems passed one by one), with empty and
    partial tracks, points without observations at either end and problems of other camera counts."""
    probs = scenes.triplet_batch(n_triplets=40, min_points=100, max_points=500, seed=4)
    probs += [scenes.circle_scene(n_cams=n, n_points=150, obs_per_point=2, seed=n) for n in (2, 4)]
    for k, sc in enumerate(probs):
        keep = ~np.isin(sc.point, {0: [0], 1: [sc.n_points - 1, sc.n_points - 2], 2: [7, 8, 9]}.get(k % 5, []))
        keep &= (sc.point * 7 + sc.view * 3 + k) % 11 != 0
        sc.view, sc.point, sc.meas = sc.view[keep], sc.point[keep], sc.meas[keep]
    flat = capi.concat_problems(probs)
    costs, (R, T, X), start = _solve(flat)
    host = capi.Batch(probs)
    res, _ = host.minimize(max_iterations=3)
    assert costs == [r.cost for r in res]
    for a, b in zip((R, T, X), host.get_all_params()):
        assert np.array_equal(a, b)
    for a, key in zip(start, ("R", "T", "X")):
        assert np.array_equal(a, flat[key])
    host.close()


def test_batch_out_of_order_and_refused():
    probs = scenes.triplet_batch(n_triplets=60, min_points=100, max_points=500, seed=5)
    flat = capi.concat_problems(probs)
    costs, params, _ = _solve(flat)
    # out of point order in the last problem: the host's grouping, the same problem
    at = int(flat["n_obs"][:-1].sum())
    o = np.arange(len(flat["view"]))
    o[at:] = at + np.argsort(flat["view"][at:], kind="stable")
    costs2, params2, _ = _solve(dict(flat, view=flat["view"][o], point=flat["point"][o], meas=flat["meas"][o]))
    assert costs2 == costs
    for a, b in zip(params, params2):
        assert np.array_equal(a, b)
    for where in (0, -1):
        for key, value in (("view", 3), ("view", -1), ("point", -1), ("point", 900), ("meas", np.nan), ("X", np.inf),
                           ("R", np.nan), ("K", np.inf)):
            bad = dict(flat, **{key: flat[key].copy()})
            bad[key].reshape(-1)[where] = value
            assert _code(lambda: capi.Batch.from_flat(bad)) == capi.ERR_INVALID_INPUT
    n = int(flat["n_obs"][0])
    long = dict(flat, point=flat["point"].copy())
    long["point"][:18] = 0
    long["point"][18:n] = np.sort(long["point"][18:n])
    assert _code(lambda: capi.Batch.from_flat(long)) == capi.ERR_UNSUPPORTED
