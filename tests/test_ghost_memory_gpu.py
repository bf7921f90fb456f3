"""Ghosts that do not fit on the device: a call that is refused leaves the set
usable, and one whose old and new arrays fit only one after the other is
served.  The device is filled up with one plain allocation; running out is an
error that the calls report."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, assert_bitwise

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")

N = 1 << 22  # a particle's thirteen arrays take 86 bytes: 361 MB, with a ghost each 721 MB
MIB = 1 << 20


def fill(torch, keep):
    """Takes all free device memory but about `keep` bytes."""
    torch.cuda.empty_cache()
    C.release_cached_memory()
    return torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")


def coords():
    rng = np.random.default_rng(3)
    return [rng.uniform(-0.2, 0.2, N) for _ in range(4)]


def warm_up(t):
    """Every kernel of the test is loaded while there is memory for it."""
    p = C.Particles(*[np.full(40, 0.1)] * 4)
    for d in (b"x", b"random"):
        C.call("hm_particles_add_ghost", p.h, 1e-3, d)
    t.track(p, 40, 0.0, 10.0)


@pytest.mark.parametrize("direction", ["x", "random"])
def test_refused_ghosts_leave_the_set_as_it_was(gpu, direction):
    torch = pytest.importorskip("torch")
    c = coords()
    t = C.Tracker(80, *TUNES, "sps", NAN, 16.0, 0)
    warm_up(t)
    p = C.Particles(*c)
    other = C.Particles(*c)
    t.track(p, 20, 0.0, 10.0)
    t.track(other, 20, 0.0, 10.0)
    want = other.state()
    # 16 + 361 (the old arrays) + 303 (the tracking workspace) < 721
    held = fill(torch, 16 * MIB)
    with pytest.raises(MemoryError):
        C.call("hm_particles_add_ghost", p.h, 1e-3, direction.encode())
    assert p.size() == (N, N, 0)
    for a, b in zip(p.state(), want):
        np.testing.assert_array_equal(a, b)
    del held
    torch.cuda.empty_cache()
    t.track(p, 20, 0.0, 10.0)
    t.track(other, 20, 0.0, 10.0)
    for a, b in zip(p.state(), other.state()):
        np.testing.assert_array_equal(a, b)
    # the refused call drew no direction
    for s in (p, other):
        C.call("hm_particles_add_ghost", s.h, 1e-3, direction.encode())
    assert p.size() == (2 * N, N, 1)
    for a, b in zip(p.state(), other.state()):
        np.testing.assert_array_equal(a, b)


def test_ghosts_that_fit_only_in_place_of_the_old_arrays(gpu):
    torch = pytest.importorskip("torch")
    c = coords()
    t = C.Tracker(80, *TUNES, "sps", NAN, 16.0, 0)
    warm_up(t)
    p = C.Particles(*c)
    held = fill(torch, 550 * MIB)  # < 721, and never tracked: no workspace
    C.call("hm_particles_add_ghost", p.h, 1e-3, b"x")
    del held
    torch.cuda.empty_cache()
    assert p.size() == (2 * N, N, 1)
    got = p.state()
    assert_bitwise(got[0], np.concatenate([c[0], c[0] + 1e-3]))
    assert_bitwise(got[3], np.concatenate([c[3], c[3]]))
    np.testing.assert_array_equal(p.get(C.FIELD_GHOST), np.repeat([0, 1], N))
