"""FFT tunes around the length at which their rows change kernels: short rows
(radices to 8) and long ones (radix 16), direct and Bluestein, against the
oracle; and the time of short windows."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import NAN, TUNES, grid
from oracle import oracle as O
from oracle import tunes as T

pytestmark = pytest.mark.gpu

C = pytest.importorskip("henon_map_cpp_b200._capi")


@pytest.mark.parametrize("remove_mean", [False, True])
def test_short_and_long_rows(gpu, remove_mean):
    x, px, y, py = grid(0.25, 3, px0=0.001)
    # direct up to 7040: 6912 and 7000 below it, 7200 above; Bluestein lengths
    # M = 64 .. 6912, 7200 and 7500; powers of two in radices 8, 4 and 2
    lengths = [3, 4, 6, 15, 16, 30, 61, 64, 100, 127, 199, 200, 499, 512, 999, 1000, 1024, 2047,
               2048, 2999, 3000, 3071, 3456, 3457, 3501, 3600, 3601, 4096, 6561, 6750, 6912, 7200]
    n_turns = 7300
    frm = [(13 * j) % 90 for j in range(len(lengths))]
    to = [f + n - 1 for f, n in zip(frm, lengths)]
    tr = C.Tracker(n_turns, *TUNES, "sps", NAN, 8.0, 0)
    p = C.Particles(x, px, y, py)
    _, f = C.tracker_orbit_tunes(tr, p, n_turns, 0.0, 10.0, frm, to, remove_mean, True)
    orb = T.orbit(x, px, y, py, O.tables(n_turns, *TUNES, "sps", epsilon=8.0), n_turns, 0.0)
    if remove_mean:
        orb = T.remove_mean(orb)
    want = np.array([T.tune_vec(*(orb[c, :, i] for c in range(4)), frm, to, "fft")
                     for i in range(x.size)])
    assert np.isfinite(want).all()
    np.testing.assert_allclose(f, want, rtol=1e-10, atol=0)


def test_time_of_short_windows(gpu):
    # Device time of the transforms of 16,000 rows of 301 samples against that
    # of the Birkhoff sums of the same call: 6.9 (10.9 when an SM held few short
    # rows).
    torch = pytest.importorskip("torch")
    n, n_turns = 8000, 300
    rng = np.random.default_rng(2)
    c = [rng.uniform(0.0, 0.3, n) for _ in range(4)]
    tr = C.Tracker(n_turns, *TUNES, "sps", NAN, 16.0, 0)

    def call():
        C.tracker_orbit_tunes(tr, C.Particles(*c), n_turns, 0.0, 10.0, [0] * 3, [n_turns] * 3,
                              False, True)

    call()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for _ in range(5):
            call()
        torch.cuda.synchronize()
    us = {k: sum(e.device_time_total for e in prof.key_averages() if k in e.key)
          for k in ("fft_tune_kernel", "birkhoff_seg_kernel")}
    assert us["birkhoff_seg_kernel"] > 0
    ratio = us["fft_tune_kernel"] / us["birkhoff_seg_kernel"]
    assert ratio < 8.5, us
