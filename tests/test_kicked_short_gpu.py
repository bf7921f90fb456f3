"""Kicked calls of a few turns: a turn whose kicks each lane makes for itself,
groups shorter than a whole one, and calls cut otherwise give the same orbits,
and their time goes with their turns."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, assert_bitwise
from oracle import oracle as O

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")
SEED, KICK, MU = 77, 0.02, 0.2


@pytest.mark.parametrize("arith", ["exact", "fast"])
@pytest.mark.parametrize("parts", [[1] * 11, [2, 9], [3, 1, 7], [10, 1], [11]])
@pytest.mark.parametrize("n", [1, 70, 300])
def test_kicked_parts(gpu, n, parts, arith):
    rng = np.random.default_rng(n)
    c = [0.6 * rng.normal(size=n) * rng.uniform(size=n) for _ in range(4)]
    t = C.Tracker(11, *TUNES, "sps", NAN, 16.0, 0)
    t.arith = C.ARITH_FAST if arith == "fast" else C.ARITH_EXACT
    p, whole = C.Particles(*c), C.Particles(*c)
    p.kick_seed = whole.kick_seed = SEED
    for k in parts:
        t.track(p, k, MU, 10.0, KICK)
    t.track(whole, 11, MU, 10.0, KICK)
    for a, b in zip(p.state(), whole.state()):
        np.testing.assert_array_equal(a, b)
    if arith == "exact":
        tabs = O.tables(11, *TUNES, "sps", epsilon=16.0)
        want = O.track_kicked(*c, np.zeros(n, np.uint32), tabs, 11, MU, 10.0, KICK, SEED)
        got = p.state()
        for a, b in zip(got[:4], want[:4]):
            assert_bitwise(a, b)
        np.testing.assert_array_equal(got[4], want[4])
        for k in parts:
            want = O.track_kicked(*want, tabs, k, MU, 10.0, KICK, SEED, inverse=True)
            t.track(p, k, MU, 10.0, KICK, True)
        got = p.state()
        for a, b in zip(got[:4], want[:4]):
            assert_bitwise(a, b)
        np.testing.assert_array_equal(got[4], want[4])


def test_time_of_one_kicked_turn(gpu):
    # 2^20 particles: 28 us for one turn and 111 for eight (78 and 111 when the
    # kicks of eight were made for one).
    rng = np.random.default_rng(1)
    c = [rng.uniform(0.0, 0.3, 1 << 20) for _ in range(4)]
    t = C.Tracker(9 * 20, *TUNES, "sps", NAN, 16.0, 0)
    p = C.Particles(*c)
    ms = {1: [], 8: []}
    for _ in range(20):
        for k in ms:
            C.set_profiling(True)
            t.track(p, k, 0.2, 10.0, 1e-4)
            ms[k].append(C.get_profile()[0])
            C.set_profiling(False)
    assert np.median(ms[1]) < 0.5 * np.median(ms[8]), {k: np.median(v) for k, v in ms.items()}
