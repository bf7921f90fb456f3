"""Points that are lost before the first turn: no turn survived, no loss, no
gradient, whichever sweep runs."""
from __future__ import annotations

import math

import numpy as np
import pytest

from conftest import TUNES

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from henon_map_cpp_b200 import autograd as AG  # noqa: E402


@pytest.mark.parametrize("kind", [dict(reverse="inverse"), dict(reverse="replay"),
                                  dict(mode="tangent"), dict(mode="loss")])
@pytest.mark.parametrize("n_turns", [2, 64, 150])
@pytest.mark.parametrize("mu", [0.0, 0.1])
def test_points_that_start_lost(gpu, mu, n_turns, kind):
    rng = np.random.default_rng(31)
    n = 200
    pts = [torch.tensor(a, dtype=torch.float64, device="cuda")
           for a in (rng.uniform(0, 0.6, n), rng.normal(0, 0.01, n),
                     rng.uniform(0, 0.6, n), rng.normal(0, 0.01, n))]
    bad = [0, 33, 64, 65, 199]
    for k, i in enumerate(bad):
        pts[k % 4][i] = math.nan
    th = torch.tensor([2 * math.pi * TUNES[0], 2 * math.pi * TUNES[1], 16.0, mu],
                      dtype=torch.float64)
    a = AG.per_particle(*pts, th, n_turns, **kind)
    assert (a["steps"].cpu().numpy()[bad] == 0).all()
    assert not a["survived"].cpu().numpy()[bad].any()
    assert (a["loss"].cpu().numpy()[bad] == 0.0).all()
    for k in ("grad_ic", "grad_theta"):
        if a.get(k) is not None:
            assert (a[k].cpu().numpy()[:, bad] == 0.0).all(), k
    steps = a["steps"].cpu().numpy()
    lost = ~a["survived"].cpu().numpy().astype(bool)
    assert (steps[~lost] == n_turns).all() and (steps[lost] < n_turns).all()
