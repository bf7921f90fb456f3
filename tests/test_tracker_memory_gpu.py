"""New turn tables that do not fit on the device: a tracker that is refused them
keeps those it has, and one whose old and new tables fit only one after the
other gets the new ones."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, assert_bitwise

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")
MIB = 1 << 20


def fill(torch, keep):
    """Takes all free device memory but about `keep` bytes."""
    torch.cuda.empty_cache()
    C.release_cached_memory()
    return torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")


def test_refused_tables_leave_the_old_ones(gpu):
    torch = pytest.importorskip("torch")
    t = C.Tracker(1000, *TUNES, "sps", NAN, 16.0, 0)
    p, other = (C.Particles(*[np.full(40, 0.1)] * 4) for _ in range(2))
    t.track(other, 1000, 0.0, 10.0)
    want = t.tables()
    held = fill(torch, 16 * MIB)
    with pytest.raises(MemoryError):  # 4 million records are 128 MB
        t.compute_a_modulation(4_000_000, *TUNES, "sps", NAN, 1.0, 0)
    del held
    torch.cuda.empty_cache()
    assert t.allowed_steps == 1000
    for a, b in zip(t.tables(), want):
        assert_bitwise(a, b)
    t.track(p, 1000, 0.0, 10.0)
    for a, b in zip(p.state(), other.state()):
        np.testing.assert_array_equal(a, b)
    with pytest.raises(C.HMError):
        t.track(p, 1, 0.0, 10.0)


def test_tables_that_fit_only_in_place_of_the_old_ones(gpu):
    torch = pytest.importorskip("torch")
    t = C.Tracker(3_000_000, *TUNES, "sps", NAN, 16.0, 0)
    new = C.Tracker(4_000_000, *TUNES, "sps", NAN, 1.0, 0)
    want = new.tables()
    del new
    held = fill(torch, 64 * MIB)  # 64 + 96 (the old tables) hold the 128 MB
    t.compute_a_modulation(4_000_000, *TUNES, "sps", NAN, 1.0, 0)
    del held
    torch.cuda.empty_cache()
    assert t.allowed_steps == 4_000_000
    for a, b in zip(t.tables(), want):
        assert_bitwise(a, b)
