"""The room that the BundlePointStructure binding gives the library and the counts that it returns, with a
stand-in for the library: the library decides which tracks are kept."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi

TRACKS = dict(track_ptr=np.array([0, 3, 5, 5, 9], np.int32), pos=np.zeros((4, 3)), view=np.zeros(9, np.int32),
              id=np.zeros(9, np.int32), mpos=np.zeros((9, 2), np.float32))


class _Library:
    """Says what the call was given, and that it kept every track with `passed` or more measurements."""

    def v3dba_error_string(self, code):
        return b"error"

    def v3dba_bundle_point_structure(self, n, ptr, pos, view, ids, mpos, required, n_points, n_meas, pts, meas, mid, cv, cp, xs):
        passed = capi.C.c_int(required).value                  # as ctypes passes it
        length = np.diff(TRACKS["track_ptr"])
        keep = (length >= passed) & (passed >= 0)
        n_points._obj.value, n_meas._obj.value = int(keep.sum()), int(length[keep].sum())
        self.room = {k: capi.C.cast(p, capi.C.c_void_p).value for k, p in dict(pts=pts, meas=meas, xs=xs).items()}
        return capi.OK


@pytest.fixture
def library(monkeypatch):
    lib = _Library()
    monkeypatch.setattr(capi, "_lib", lambda: lib)
    return lib


@pytest.mark.parametrize("required,kept,meas", [(-1, 0, 0), (0, 4, 9), (2, 3, 9), (3, 2, 7), (5, 0, 0), (-0.5, 4, 9),
                                                (2**31 - 1, 0, 0), (-2**31, 0, 0)])
def test_results_have_the_counts_that_the_library_returns(library, required, kept, meas):
    out = capi.bundle_point_structure(TRACKS, required)
    assert [out[k].shape for k in ("points3d", "xs_indices")] == [(kept, 3), (kept,)]
    assert [out[k].shape for k in ("measurements", "measurement_ids", "corresponding_view", "corresponding_point")] == \
        [(meas, 2), (meas,), (meas,), (meas,)]


@pytest.mark.parametrize("required", [2**31, 2**32 + 2, -2**31 - 1, -2**32 + 2])
def test_values_outside_int_are_refused(library, required):
    with pytest.raises(capi.V3dbaError) as e:
        capi.bundle_point_structure(TRACKS, required)
    assert e.value.code == capi.ERR_INVALID_ARGUMENT


@pytest.mark.parametrize("required", [-1, 3, 5])
def test_room_for_every_track(library, monkeypatch, required):
    """The arrays hold every track and measurement, whichever of them the library keeps."""
    size = {}
    zeros = np.zeros

    def recorded(shape, dtype=float):
        a = zeros(shape, dtype)
        size[a.ctypes.data] = a.size
        return a

    monkeypatch.setattr(capi.np, "zeros", recorded)
    capi.bundle_point_structure(TRACKS, required)
    assert [size[library.room[k]] for k in ("pts", "meas", "xs")] == [12, 18, 4]
