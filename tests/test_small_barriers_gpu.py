"""Barriers of the size of the orbits: the tracker's coarser looks at a block of
turns fail there without a loss, and it goes over to finer ones.  Results bit
for bit against the oracle, and the time within reach of a wide barrier's."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, assert_bitwise, grid
from oracle import oracle as O

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")


@pytest.mark.parametrize("per_thread", [1, 2, 4])
@pytest.mark.parametrize("mu", [0.0, 0.2, 3.0])
@pytest.mark.parametrize("barrier", [0.45, 0.8, 1.0, 1.5, 2.5])
def test_looks_of_a_stage(gpu, barrier, mu, per_thread):
    # two stages and a part of one, with a short last block
    n, n_turns = 3000, 512 + 512 + 77
    rng = np.random.default_rng(4)
    c = [rng.uniform(-0.5, 0.5, n) * rng.uniform(size=n) for _ in range(4)]
    tabs = O.tables(n_turns, *TUNES, "sps", epsilon=16.0)
    want = O.track(*c, np.zeros(n, np.uint32), tabs, n_turns, mu, barrier)
    assert (want[4] == n_turns).any() and (want[4] < n_turns).any()
    before = C.get_track_config()
    C.set_track_config(32, per_thread, before[2], before[3])
    try:
        t = C.Tracker(n_turns, *TUNES, "sps", NAN, 16.0, 0)
        p = C.Particles(*c)
        t.track(p, n_turns, mu, barrier)
        got = p.state()
        t.track(p, 600, mu, barrier, NAN, True)
        back = p.state()
    finally:
        C.set_track_config(*before)
    want_back = O.track(*want, tabs, 600, mu, barrier, inverse=True)
    for g, w in ((got, want), (back, want_back)):
        for a, b in zip(g[:4], w[:4]):
            assert_bitwise(a, b)
        np.testing.assert_array_equal(g[4], w[4])


def test_time_at_a_small_barrier(gpu):
    # The same orbits (all but a few) survive at both barriers: 1.6 times the
    # wide one's time at 1.5 (5.8 when each block was tested again).
    n_turns = 10_000
    t = C.Tracker(n_turns, *TUNES, "sps", NAN, 16.0, 0)
    ms, alive = {}, {}
    for barrier in (1.5, 100.0):
        times = []
        for _ in range(4):
            p = C.Particles(*grid(0.35, 60))
            C.set_profiling(True)
            t.track(p, n_turns, 0.0, barrier)
            times.append(C.get_profile()[0])
            C.set_profiling(False)
        ms[barrier] = min(times)
        alive[barrier] = p.get(C.FIELD_STEPS) == n_turns
    np.testing.assert_array_equal(alive[1.5], alive[100.0])
    assert alive[1.5].mean() > 0.99
    assert ms[1.5] < 2.5 * ms[100.0], ms
