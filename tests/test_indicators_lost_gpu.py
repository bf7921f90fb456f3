"""The fused indicator loop with lost particles: the state it leaves does not
depend on how the turns are cut into calls and launches or on a particle's
neighbours, and a particle's tangent map, tangent vector, MEGNO layers and
angles are NaN from the first turn that is applied to a lost point."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, assert_bitwise

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")

WINDOWS = [3, 20, 3000, 5000]
N = 300


def run(parts, use, jacobian):
    rng = np.random.default_rng(2)
    c = [0.55 * rng.normal(size=N) * rng.uniform(size=N) for _ in range(4)]
    for f in c:
        f[64:160] = np.nan  # three whole warps lost before the first turn, ...
        f[170] = np.nan     # ... and one particle of another
    t = C.Tracker(sum(parts) + 1, *TUNES, "sps", NAN, 16.0, 0)
    p = C.Particles(*c)
    k = {}
    if "M" in use:
        k.update(matrix=C.Matrices(N), matrix_old=C.Matrices(N), megno=C.Megno(N),
                 megno_birkhoff=C.MegnoBirkhoff(N, WINDOWS))
    if "V" in use:
        k.update(vectors=C.Vectors(np.tile([1.0, 0.0, 0.0, 0.0], (N, 1))),
                 lyapunov=C.Lyapunov(N, WINDOWS))
    if "T" in use:
        k.update(tune=C.TuneBirkhoff(N, WINDOWS))
        k["tune"].first_add(p)
    for n in parts:
        C.track_indicators(t, p, n, 0.2, 10.0, jacobian_of_turn=jacobian, **k)
    out = {}
    for name in ("matrix", "matrix_old", "megno", "megno_birkhoff", "vectors"):
        if name in k:
            out[name] = k[name].get()
    if "V" in use:
        out["raw"], out["birkhoff"] = k["lyapunov"].get(False), k["lyapunov"].get(True)
    if "T" in use:
        for w in range(4):
            out[f"tune {w}"] = k["tune"].get(w)
    return p.state(), out


@pytest.mark.parametrize("jacobian", [False, True])
@pytest.mark.parametrize("use", ["MVT", "MV", "MT", "VT", "M", "V", "T"])
@pytest.mark.parametrize("parts", [[1, 1, 30], [31, 1], [4096, 2, 2]])
def test_lost_particles(gpu, parts, use, jacobian):
    n_turns = sum(parts)
    state, whole = run([n_turns], use, jacobian)
    state2, cut = run(parts, use, jacobian)
    for a, b in zip(state, state2):
        np.testing.assert_array_equal(a, b)
    for name in whole:
        assert_bitwise(whole[name], cut[name], name)
    steps = state[4].astype(np.int64)
    lost = np.isnan(state[0])
    assert (lost & (steps > 0)).any() and not lost.all()
    # With the Jacobian at the point before the turn, the turn of the loss
    # itself (turn `steps`) still has a finite one; a point that starts as NaN
    # has none.
    started = np.ones(N, bool)
    started[64:160] = started[170] = False
    after = steps + np.where(started & jacobian, 1, 0)  # first turn of NaN
    want = lost & (after < n_turns)
    for name in ("matrix", "megno", "vectors"):
        if name in whole:
            nan = np.isnan(whole[name].reshape(N, -1))
            np.testing.assert_array_equal(nan.all(axis=1), want, err_msg=name)
            np.testing.assert_array_equal(nan.any(axis=1), want, err_msg=name)
