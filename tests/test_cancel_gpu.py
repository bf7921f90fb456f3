"""The cancel callback is asked between the chunks of turns of a tracking call,
from the first one on, and a call that it stops leaves the set at the end of
the chunk before."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import NAN, TUNES

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")
CALLBACK = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p)
N_TURNS = 40_000
# chunks of 512, 1024, ..., 16384 and what is left: where a call may stop
STOPS = [512, 1536, 3584, 7680, 15872, 32256]


def sets(n):
    rng = np.random.default_rng(n)
    c = [rng.uniform(0.0, 0.5, n) for _ in range(4)]
    return C.Particles(*c), C.Particles(*c)


@pytest.mark.parametrize("kick", [NAN, 1e-3])
@pytest.mark.parametrize("asked", [1, 2, 4, 6])
@pytest.mark.parametrize("n", [1, 3000])
def test_cancelled_between_chunks(gpu, n, asked, kick):
    count = [0]

    def stop(_):
        count[0] += 1
        return int(count[0] >= asked)

    fn = CALLBACK(stop)
    t = C.Tracker(N_TURNS, *TUNES, "sps", NAN, 16.0, 0)
    p, other = sets(n)
    if n == 1:
        kick = NAN  # a resting orbit: the kicks would lose the only particle
        p, other = (C.Particles([0.1], [0.0], [0.1], [0.0]) for _ in range(2))
    C.call("hm_set_cancel_callback", ctypes.cast(fn, ctypes.c_void_p), None)
    try:
        with pytest.raises(C.HMCancelled):
            t.track(p, N_TURNS, 0.0, 10.0, kick)
    finally:
        C.call("hm_set_cancel_callback", None, None)
    assert count[0] == asked
    assert p.global_steps == STOPS[asked - 1]
    t.track(other, STOPS[asked - 1], 0.0, 10.0, kick)
    for a, b in zip(p.state(), other.state()):
        np.testing.assert_array_equal(a, b)
    # and the call can be taken up where it stopped
    left = N_TURNS - STOPS[asked - 1]
    t.track(p, left, 0.0, 10.0, kick)
    t.track(other, left, 0.0, 10.0, kick)
    for a, b in zip(p.state(), other.state()):
        np.testing.assert_array_equal(a, b)


def test_not_asked_to_stop(gpu):
    asked = []
    fn = CALLBACK(lambda _: asked.append(1) or 0)
    t = C.Tracker(N_TURNS, *TUNES, "sps", NAN, 16.0, 0)
    p, other = sets(3000)
    C.call("hm_set_cancel_callback", ctypes.cast(fn, ctypes.c_void_p), None)
    try:
        t.track(p, N_TURNS, 0.0, 10.0)
    finally:
        C.call("hm_set_cancel_callback", None, None)
    assert len(asked) == len(STOPS)
    t.track(other, N_TURNS, 0.0, 10.0)
    for a, b in zip(p.state(), other.state()):
        np.testing.assert_array_equal(a, b)
