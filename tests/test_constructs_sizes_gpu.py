"""The per-call construct kernels deal windows to the warps of a block by the
size of the set: every size against the fused loop, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, assert_bitwise

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")


@pytest.mark.parametrize("n", [1, 31, 33, 2000, 9473, 80_000])
@pytest.mark.parametrize("windows", [1, 4, 5, 13])
def test_per_call_equals_fused(gpu, n, windows):
    rng = np.random.default_rng(n)
    c = [rng.uniform(-0.45, 0.45, n) for _ in range(4)]
    wins = [1 + (7 * w) % 11 for w in range(windows)]
    turns = 12
    v0 = np.tile([1.0, 0.5, 0.0, 0.0], (n, 1))

    def build():
        t = C.Tracker(turns + 1, *TUNES, "sps", NAN, 32.0, 0)
        o = dict(matrix=C.Matrices(n), megno=C.Megno(n), megno_birkhoff=C.MegnoBirkhoff(n, wins),
                 vectors=C.Vectors(v0), lyapunov=C.Lyapunov(n, wins), tune=C.TuneBirkhoff(n, wins))
        p = C.Particles(*c)
        o["tune"].first_add(p)
        return t, p, o

    t, p, o = build()
    C.track_indicators(t, p, turns, 0.2, 10.0, **o)
    t2, q, k = build()
    old, jac = C.Matrices(n), C.Matrices(n)
    for _ in range(turns):
        old.explicit_copy(k["matrix"])
        t2.track(q, 1, 0.2, 10.0)
        k["matrix"].structured_multiply(t2, q, 0.2)
        k["megno"].add(k["matrix"], old)
        k["megno_birkhoff"].add(k["matrix"], old)
        jac.set_with_tracker(t2, q, 0.2)
        k["vectors"].multiply(jac)
        k["lyapunov"].add(k["vectors"])
        k["vectors"].normalize()
        k["tune"].add(q)
    for name in ("matrix", "megno", "megno_birkhoff", "vectors"):
        assert_bitwise(k[name].get(), o[name].get(), name)
    for b in (False, True):
        assert_bitwise(k["lyapunov"].get(b), o["lyapunov"].get(b), f"lyapunov {b}")
    for w in range(4):
        assert_bitwise(k["tune"].get(w), o["tune"].get(w), f"tune {w}")
