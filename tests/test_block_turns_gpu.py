"""The tracker's blocks of turns without per-turn control flow: turn counts
around the block and stage lengths, losses between the turns that are looked
at, and tables that are not rotations, bit for bit against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, assert_bitwise
from oracle import oracle as O

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")

NAMES = ("x", "px", "y", "py")


def check(got, want, what):
    for a, b, name in zip(got[:4], want[:4], NAMES):
        assert_bitwise(a, b, f"{what}: {name}")
    np.testing.assert_array_equal(got[4], want[4], err_msg=what)


def points(n, scale, seed=5):
    rng = np.random.default_rng(seed)
    return [scale * rng.normal(size=n) * rng.uniform(size=n) ** 2 for _ in range(4)]


@pytest.mark.parametrize("n_turns", [1, 15, 16, 17, 31, 33, 511, 512, 513, 1537])
@pytest.mark.parametrize("n", [1, 33, 700])
def test_turn_counts_around_blocks_and_stages(gpu, n, n_turns):
    c = points(n, 0.3)
    tabs = O.tables(n_turns, *TUNES, "sps", epsilon=16.0)
    want = O.track(*c, np.zeros(n, np.uint32), tabs, n_turns, 0.2, 10.0)
    t = C.Tracker(n_turns, *TUNES, "sps", NAN, 16.0, 0)
    p = C.Particles(*c)
    t.track(p, n_turns, 0.2, 10.0)
    check(p.state(), want, "forward")
    back = n_turns // 2 + 1
    want = O.track(*want, tabs, back, 0.2, 10.0, inverse=True)
    t.track(p, back, 0.2, 10.0, NAN, True)
    check(p.state(), want, "backward")


@pytest.mark.parametrize("mu", [0.0, 0.2, -3.0])
@pytest.mark.parametrize("barrier", [0.02, 0.3, 1.0, 3.0, 10.0, 400.0])
def test_losses_between_the_turns_looked_at(gpu, barrier, mu):
    # Starts spread over several times the barrier: many particles are
    # outside after an odd turn and, without the loss, would be back inside
    # after the next one.
    n, n_turns = 4000, 96
    c = points(n, min(2.0, barrier), 7)
    tabs = O.tables(n_turns, *TUNES, "sps", epsilon=64.0)
    want = O.track(*c, np.zeros(n, np.uint32), tabs, n_turns, mu, barrier)
    odd = (want[4] % 2 == 0) & (want[4] > 0) & (want[4] < n_turns)
    assert odd.any()  # lost in an odd turn of the block (the first is turn 0)
    t = C.Tracker(n_turns, *TUNES, "sps", NAN, 64.0, 0)
    p = C.Particles(*c)
    t.track(p, n_turns, mu, barrier)
    check(p.state(), want, "tracker")
    sets = [dict(omega_x=TUNES[0], omega_y=TUNES[1], epsilon=64.0, mu=mu, n_particles=n,
                 n_turns=n_turns, barrier=barrier)]
    b = C.Batch(sets)
    b.load(*c)
    b.run()
    check([b.get(f) for f in (C.FIELD_X, C.FIELD_PX, C.FIELD_Y, C.FIELD_PY, C.FIELD_STEPS)],
          want, "batch")


@pytest.mark.parametrize("scale", [0.5, 0.97, 1.0, 1.02])
def test_device_tables_that_are_not_rotations(gpu, scale):
    # hm_track_device takes any records; damping or growth per turn breaks
    # the bound that looking at every second turn rests on.
    import torch

    n, n_turns = 2000, 700
    c = points(n, 0.5, 9)
    tabs = [scale * t for t in O.tables(n_turns, *TUNES, "sps", epsilon=1.0)]
    want = O.track(*c, np.zeros(n, np.uint32), tabs, n_turns, 0.0, 10.0)
    rec = torch.from_numpy(np.stack(tabs, axis=1).copy()).cuda()
    dev = [torch.from_numpy(a).cuda() for a in c]
    steps = torch.zeros(n, dtype=torch.int32, device="cuda")
    ws = torch.empty(C.load().hm_track_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    C.call("hm_track_device", *[d.data_ptr() for d in dev], steps.data_ptr(), n, rec.data_ptr(),
           n_turns, 0, n_turns, 0.0, 10.0, 0, 0, ws.data_ptr(), None)
    check([d.cpu().numpy() for d in dev] + [steps.cpu().numpy().view(np.uint32)], want,
          f"scale {scale}")


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("n_turns", [1, 7, 8, 9, 100])
@pytest.mark.parametrize("n", [1, 31, 33, 300])
def test_kicked_groups_of_turns(gpu, n, n_turns, inverse):
    # Kicks are made for groups of 8 turns, rejected points by whole warps:
    # part groups, part warps, losses inside a group, a set that starts
    # with NaN particles, both directions.
    c = points(n, 0.6, 11)
    if n > 2:
        c[2][n // 2] = np.nan
    seed, kick, mu = 0x9E3779B97F4A7C15, 0.02, 0.2
    tabs = O.tables(max(n_turns, 1), *TUNES, "sps", epsilon=16.0)
    t = C.Tracker(n_turns, *TUNES, "sps", NAN, 16.0, 0)
    p = C.Particles(*c)
    p.kick_seed = seed
    want = (*c, np.zeros(n, np.uint32))
    if inverse:
        want = O.track(*want, tabs, n_turns, mu, 10.0)
        t.track(p, n_turns, mu, 10.0)
    want = O.track_kicked(*want, tabs, n_turns, mu, 10.0, kick, seed, inverse=inverse)
    t.track(p, n_turns, mu, 10.0, kick, inverse)
    check(p.state(), want, "kicked")
