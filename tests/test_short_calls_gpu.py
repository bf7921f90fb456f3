"""Calls of a few turns around the sizes at which they go over from records
read directly to staged ones, and from one to two particles per thread, bit
for bit against the oracle (the sizes are those of 148 multiprocessors)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, assert_bitwise
from oracle import oracle as O

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")


@pytest.mark.parametrize("mu", [0.2, 0.0])
@pytest.mark.parametrize("n,turns", [
    (18_943, (15, 16)), (18_944, (31, 47, 48)), (56_832, (48, 111, 112)),
    (75_775, (16,)), (75_776, (31, 32)), (113_409, (8, 16)), (113_665, (1, 8, 33))])
def test_routes_of_short_calls(gpu, n, turns, mu):
    rng = np.random.default_rng(8)
    c = [0.6 * rng.normal(size=n) * rng.uniform(size=n) for _ in range(4)]
    c[1][n - 1] = np.nan
    total = sum(turns)
    tabs = O.tables(total, *TUNES, "sps", epsilon=16.0)
    t = C.Tracker(total, *TUNES, "sps", NAN, 16.0, 0)
    p = C.Particles(*c)
    want = (*c, np.zeros(n, np.uint32))
    for k, back in [(k, False) for k in turns] + [(k, True) for k in turns]:
        want = O.track(*want, tabs, k, mu, 10.0, inverse=back)
        t.track(p, k, mu, 10.0, NAN, back)
    got = p.state()
    for a, b in zip(got[:4], want[:4]):
        assert_bitwise(a, b)
    np.testing.assert_array_equal(got[4], want[4])
    assert np.isnan(want[0]).any() and not np.isnan(want[0]).all()
