"""The inverse-sweep adjoint at the edges of its stretches of turns: horizons
around the 64-turn stage and checkpoint spacings around it, with points lost
inside a stretch.  Loss, loss turn and survival equal the replay sweep's bit
for bit (same operations per turn); the gradients agree to the bounds of
test_adjoint_gpu.py::test_reverse_sweeps_agree_and_mu_gradient_at_zero."""
from __future__ import annotations

import math

import numpy as np
import pytest

from conftest import TUNES

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from henon_map_cpp_b200 import autograd as AG  # noqa: E402


@pytest.mark.parametrize("n_turns", [1, 63, 64, 65, 129])
@pytest.mark.parametrize("every", [1, 5, 63, 64, 65, 200])
@pytest.mark.parametrize("mu", [0.0, 0.1])
def test_stretch_edges(gpu, n_turns, every, mu):
    rng = np.random.default_rng(17)
    n = 300
    pts = [torch.tensor(a, dtype=torch.float64, device="cuda")
           for a in (rng.uniform(0, 0.6, n), rng.normal(0, 0.01, n),
                     rng.uniform(0, 0.6, n), rng.normal(0, 0.01, n))]
    pts[0][7] = math.nan
    th = torch.tensor([2 * math.pi * TUNES[0], 2 * math.pi * TUNES[1], 16.0, mu],
                      dtype=torch.float64)
    a = AG.per_particle(*pts, th, n_turns, checkpoint_every=every, reverse="inverse")
    b = AG.per_particle(*pts, th, n_turns, checkpoint_every=every, reverse="replay")
    for k in ("loss", "survived"):
        np.testing.assert_array_equal(a[k].cpu().numpy(), b[k].cpu().numpy(), err_msg=k)
    # The sweeps count a point that is lost before the first turn differently.
    played = np.arange(n) != 7
    np.testing.assert_array_equal(a["steps"].cpu().numpy()[played],
                                  b["steps"].cpu().numpy()[played])
    assert not a["survived"][7] and a["loss"][7] == 0.0
    s = a["survived"]
    assert s.any()
    if n_turns >= 63:
        assert not s.all()
    for k, tol in (("grad_ic", 1e-12), ("grad_theta", 1e-10)):
        x, y = a[k][:, s].cpu().numpy(), b[k][:, s].cpu().numpy()
        np.testing.assert_array_equal(np.isnan(x), np.isnan(y), err_msg=k)
        if n_turns == 1:  # one Birkhoff weight, 0/0: NaN in both sweeps
            assert np.isnan(a["loss"].cpu().numpy()[s.cpu().numpy()]).all()
            continue
        rel = np.abs(x - y) / np.maximum(np.abs(y), 1e-300)
        assert np.median(rel) < tol, (k, np.median(rel))


@pytest.mark.parametrize("n", [1, 300, 20_000])
@pytest.mark.parametrize("n_turns", [1, 64, 129])
@pytest.mark.parametrize("mu", [0.0, 0.1])
def test_loss_alone(gpu, n, n_turns, mu):
    """mode "loss" equals the tangent kernel's loss, loss turns and survival
    bit for bit (one turn at a time there)."""
    rng = np.random.default_rng(23)
    pts = [torch.tensor(a, dtype=torch.float64, device="cuda")
           for a in (rng.uniform(0, 0.6, n), rng.normal(0, 0.01, n),
                     rng.uniform(0, 0.6, n), rng.normal(0, 0.01, n))]
    if n > 1:
        pts[2][n // 2] = math.nan
    th = torch.tensor([2 * math.pi * TUNES[0], 2 * math.pi * TUNES[1], 16.0, mu],
                      dtype=torch.float64)
    a = AG.per_particle(*pts, th, n_turns, mode="loss")
    b = AG.per_particle(*pts, th, n_turns, mode="tangent")
    for k in ("loss", "steps", "survived"):
        np.testing.assert_array_equal(a[k].cpu().numpy(), b[k].cpu().numpy(), err_msg=k)
