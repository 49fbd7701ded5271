"""Per-observation blocks written through shared memory (FP64) and lane by lane (FP32): tracks of different
lengths in one warp, point counts around the sixteen points of a warp and the sixty-four of a block, fixed
cameras and points, every global dimension.

The system formed from the blocks against the C restatement: FP64 sums in another order agree to 1e-11 of the
largest entry that they are formed from (1e-16 * 1e3 condition number of a point block * 1e2 terms), FP32
blocks (rounded to 6e-8) to 1e-5."""
import numpy as np
import pytest

from oracle.bindings import Restatement
from v3dsfmtoolkit_b200 import capi, scenes

pytestmark = pytest.mark.gpu

MODES = {"metric": scenes.FULL_BUNDLE_METRIC, "focal": scenes.FULL_BUNDLE_FOCAL_LENGTH,
         "radial_tangential": scenes.FULL_BUNDLE_RADIAL_TANGENTIAL}


@pytest.mark.parametrize("fixed", [(0, 0, 0), (2, 3, 0)])
@pytest.mark.parametrize("points", [1, 15, 16, 17, 63, 65, 130])
@pytest.mark.parametrize("mode", sorted(MODES))
def test_blocks_of_unequal_tracks(mode, points, fixed):
    sc = scenes.sequence_scene(n_cams=9, n_points=points, min_track=2, max_track=9, seed=points, mode=MODES[mode])
    h = capi.Handle.from_scene(sc)
    h.set_nonvarying(*fixed)
    orc = Restatement()
    blocks = orc.normal_blocks(sc, nonvarying=fixed)
    big_S = max(np.abs(blocks[k]).max() for k in ("U", "X", "Z") if blocks[k].size)
    big_b = max(np.abs(blocks[k]).max() for k in ("ga", "gc") if blocks[k].size)
    lam = 1e-3 * np.abs(blocks["U"]).max()
    Sr, br, _, _ = orc.reduced_system(sc, blocks, lam, fixed)
    for precision, tol in ((capi.PRECISION_FP64, 1e-11), (capi.PRECISION_MIXED, 1e-5)):
        S, b = h.reduced_system(lam, precision)
        assert np.abs(S - Sr).max() <= tol * big_S
        assert np.abs(b - br).max() <= tol * big_b
    h.close()
