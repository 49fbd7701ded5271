"""The staged pair-list kernels in every camera dimension: a problem small enough for the direct loads, next to
itself often enough for the staged ones, has the same blocks, bit for bit with FP32 blocks (the same sums in
the same order); and a problem of global unknowns with enough chunks for the merged staged launch agrees
with the C restatement.  Bounds as in test_gpu_chunk_kernels: FP64 sums 1e-16 * 1e3 (condition number of a
point block) * 1e2, FP32 blocks 1e-5 of the undamped blocks."""
import numpy as np
import pytest

from oracle.bindings import Restatement
from tests.test_gpu_chunk_kernels import _many
from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu

DIRECT_CHUNKS = 1184


def _chunks(sc):
    """Chunks of 128 pairs over the camera-pair blocks (tracks without repeated cameras)."""
    o = np.lexsort((sc.view, sc.point))
    v, p = sc.view[o].astype(np.int64), sc.point[o]
    pairs = {}
    n = np.bincount(p, minlength=sc.n_points)
    first = np.cumsum(n) - n
    for length in np.unique(n[n > 0]):
        at = first[n == length][:, None] + np.arange(length)
        for a in range(length):
            for b in range(a, length):
                keys, c = np.unique(v[at[:, a]] * sc.n_cams + v[at[:, b]], return_counts=True)
                for k, m in zip(keys, c):
                    pairs[k] = pairs.get(k, 0) + int(m)
    return sum(-(-m // 128) for m in pairs.values())


VARYING = {7: scenes.FULL_BUNDLE_FOCAL_LENGTH, 9: scenes.FULL_BUNDLE_FOCAL_LENGTH_PP, 11: scenes.FULL_BUNDLE_RADIAL,
           13: scenes.FULL_BUNDLE_RADIAL_TANGENTIAL}


@pytest.mark.parametrize("points", [5, 33, 150])
@pytest.mark.parametrize("unknowns", sorted(VARYING))
def test_staged_equal_direct(unknowns, points, monkeypatch):
    monkeypatch.setenv("V3DBA_SCHUR", "pairs")
    small = scenes.varying_scene(n_cams=4, n_points=points, mode=VARYING[unknowns], seed=points)
    copies = DIRECT_CHUNKS // _chunks(small) + 1
    big = _many(small, copies)
    assert _chunks(small) <= DIRECT_CHUNKS < _chunks(big)
    hs, hb = capi.Handle.from_scene(small), capi.Handle.from_scene(big)
    for precision, tol in ((capi.PRECISION_MIXED, 0.0), (capi.PRECISION_FP64, 1e-11)):
        S, b = hs.reduced_system(1e3, precision)
        T, c = hb.reduced_system(1e3, precision)
        n = S.shape[0]
        for k in (0, copies // 2, copies - 1):
            at = slice(n * k, n * (k + 1))
            assert np.abs(T[at, at] - S).max() <= tol * np.abs(S).max()
            assert np.abs(c[at] - b).max() <= 1e-12 * np.abs(b).max()
    hs.close()
    hb.close()


@pytest.mark.parametrize("mode", [scenes.FULL_BUNDLE_FOCAL_LENGTH, scenes.FULL_BUNDLE_FOCAL_LENGTH_PP,
                                  scenes.FULL_BUNDLE_RADIAL, scenes.FULL_BUNDLE_RADIAL_TANGENTIAL])
def test_merged_staged_launch_with_global_unknowns(mode, monkeypatch):
    monkeypatch.setenv("V3DBA_SCHUR", "pairs")
    sc = scenes.sequence_scene(n_cams=40, n_points=5001, mode=mode, seed=2)
    assert _chunks(sc) > DIRECT_CHUNKS
    h = capi.Handle.from_scene(sc)
    S0, _ = h.reduced_system(1e4)
    lam = 1e-3 * np.abs(np.diag(S0)).max()
    orc = Restatement()
    blocks = orc.normal_blocks(sc)
    Sr, br, _, _ = orc.reduced_system(sc, blocks, lam)
    big_S = max(np.abs(blocks[k]).max() for k in ("U", "X", "Z") if blocks[k].size)
    big_b = max(np.abs(blocks[k]).max() for k in ("ga", "gc") if blocks[k].size)
    for precision, tol in ((capi.PRECISION_FP64, 1e-11), (capi.PRECISION_MIXED, 1e-5)):
        S, b = h.reduced_system(lam, precision)
        assert np.abs(S - Sr).max() <= tol * big_S
        assert np.abs(b - br).max() <= tol * big_b
    h.close()
