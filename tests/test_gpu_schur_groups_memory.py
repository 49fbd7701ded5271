"""Where there is no device memory for the grouped Schur sums, a run takes the pair lists and ends as it does
with them, bit for bit; the next run makes the groups.  Failures are injected on the host in front of every
allocation of the grouping (v3dba_debug_fail_allocation)."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _injection_off():
    capi.debug_fail_allocation(-1)
    yield
    capi.debug_fail_allocation(-1)


def _run(h, fail_at=-1, **options):
    h.reset_params()
    capi.debug_fail_allocation(fail_at)
    r = h.minimize(**options)
    capi.debug_fail_allocation(-1)
    return (r.status, r.iterations, r.n_rejected, r.fp64_from_iteration, r.cost), h.get_params()


def _same(a, b):
    return a[0] == b[0] and all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))


def _handle(sc):
    h = capi.Handle.from_scene(sc)
    h.minimize(max_iterations=1)     # the plan of the direct solver, which a run cannot do without
    return h


FP64 = dict(max_iterations=4, precision=capi.PRECISION_FP64)
MIXED = dict(max_iterations=40)      # ends with FP64 blocks


@pytest.mark.parametrize("options", [FP64, MIXED], ids=["fp64", "mixed"])
def test_every_allocation_of_the_groups_may_fail(options, monkeypatch):
    sc = scenes.sequence_scene(n_cams=20, n_points=2500, seed=1)
    monkeypatch.setenv("V3DBA_SCHUR", "pairs")
    h = _handle(sc)
    pairs = _run(h, **options)
    assert options is FP64 or pairs[0][3] > 0
    h.close()
    monkeypatch.setenv("V3DBA_SCHUR", "groups")
    h = _handle(sc)
    groups = _run(h, **options)
    h.close()
    assert not _same(groups, pairs)      # another order of summation: the groups ran
    failed = 0
    for k in range(200):
        h = _handle(sc)
        got = _run(h, k, **options)
        if _same(got, groups):           # the injection was not reached
            h.close()
            break
        failed += 1
        assert _same(got, pairs)
        assert _same(_run(h, **options), groups)
        h.close()
    else:
        pytest.fail("the injected failure never ran out")
    assert failed > 10


@pytest.mark.parametrize("k", [0, 7, 13])
def test_reduced_system_without_room(k, monkeypatch):
    sc = scenes.sequence_scene(n_cams=20, n_points=2500, seed=1)
    out = {}
    for how, fail_at in (("pairs", -1), ("groups", k)):
        monkeypatch.setenv("V3DBA_SCHUR", how)
        h = _handle(sc)
        capi.debug_fail_allocation(fail_at)
        out[how] = h.reduced_system(1.0)
        capi.debug_fail_allocation(-1)
        h.close()
    np.testing.assert_array_equal(out["groups"][0], out["pairs"][0])
    np.testing.assert_array_equal(out["groups"][1], out["pairs"][1])
