"""Backward turns read the turn records below the particles' own steps: a tracker
with fewer of them is refused, by every entry point that goes backward."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import NAN, TUNES

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")


@pytest.mark.parametrize("turns", [10, 30])
def test_shorter_table_is_refused(gpu, turns):
    long = C.Tracker(200, *TUNES, "sps", NAN, 16.0, 0)
    short = C.Tracker(turns, *TUNES, "sps", NAN, 16.0, 0)
    p = C.Particles(*[np.full(40, 0.1)] * 4)
    long.track(p, 100, 0.0, 10.0)
    before = p.state()
    samples = np.array([1], np.uint64)
    out = np.empty((40, 1))
    message = "number of turns is too large"
    with pytest.raises(C.HMError, match=message):
        short.track(p, 5, 0.0, 10.0, NAN, True)
    with pytest.raises(C.HMError, match=message):
        C.tracker_orbit_tunes(short, p, 5, 0.0, 10.0, [], [], False, False, NAN, True)
    with pytest.raises(C.HMError, match=message):
        C.call("hm_tracker_megno", short.h, p.h, 5, 0.0, 10.0, NAN, 1,
               samples.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), 1, C.dptr(out))
    assert p.global_steps == 100
    for a, b in zip(p.state(), before):
        np.testing.assert_array_equal(a, b)
    # and the tracker that has them is not
    C.tracker_orbit_tunes(long, p, 5, 0.0, 10.0, [], [], False, False, NAN, True)
    C.call("hm_tracker_megno", long.h, p.h, 5, 0.0, 10.0, NAN, 1,
           samples.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), 1, C.dptr(out))
    assert p.global_steps == 90
