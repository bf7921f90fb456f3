"""Particle sets and tangent vectors from arrays, strided arrays and lists: the
same sets, and the same inputs refused."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E = pytest.importorskip("henon_map_cpp_b200.henon_map_engine")

V = np.linspace(-0.4, 0.9, 13)


@pytest.mark.parametrize("make", [
    lambda v: v, lambda v: list(v), lambda v: tuple(v), lambda v: np.repeat(v, 3)[::3],
    lambda v: v[::-1].copy()[::-1], lambda v: v.astype(">f8"),
    lambda v: np.ma.masked_array(v, mask=False),
    lambda v: np.frombuffer(b"x" + v.tobytes(), dtype=np.uint8)[1:].view("f8")])
def test_same_particles(gpu, make):
    p = E.particles_4d_gpu(make(V), make(V + 1), make(V + 2), make(V + 3))
    for k, get in enumerate((p.get_x, p.get_px, p.get_y, p.get_py)):
        np.testing.assert_array_equal(np.asarray(get()), V + k)


def test_other_numbers_and_refusals(gpu):
    f32 = V.astype(np.float32)
    p = E.particles_4d_gpu(f32, [0] * 13, np.arange(13), V)
    np.testing.assert_array_equal(np.asarray(p.get_x()), f32.astype(np.float64))
    np.testing.assert_array_equal(np.asarray(p.get_y()), np.arange(13.0))
    assert np.asarray(E.particles_4d_gpu(V[:0], V[:0], V[:0], V[:0]).get_x()).size == 0
    with pytest.raises(ValueError):
        E.particles_4d_gpu(V, V, V[:5], V)
    with pytest.warns(np.exceptions.ComplexWarning):  # the imaginary part is dropped, as ever
        p = E.particles_4d_gpu(V.astype(complex), V, V, V)
    np.testing.assert_array_equal(np.asarray(p.get_x()), V)
    for bad in (np.zeros((13, 2)), np.float64(1.0), V.astype(str), None):
        with pytest.raises(TypeError):
            E.particles_4d_gpu(bad, V, V, V)


def test_same_vectors(gpu):
    rv = np.arange(20.0).reshape(5, 4)
    for make in (lambda a: a, lambda a: a.tolist(), np.asfortranarray,
                 lambda a: a.astype(np.float32)):
        np.testing.assert_array_equal(np.asarray(E.vector_4d_gpu(make(rv)).get_vectors()), rv)
    for bad in (rv[:, :3], rv.ravel()):
        with pytest.raises((TypeError, ValueError)):
            E.vector_4d_gpu(bad)


@pytest.mark.parametrize("n", [1, 255, 257])
@pytest.mark.parametrize("dirs", [("x",), ("px", "y"), ("y", "random", "py"), ("random", "x")])
def test_ghosts_on_the_device_and_through_the_host(gpu, n, dirs):
    # Ghosts along a coordinate are appended on the device, random ones (and
    # all after them) through the host mirrors: coordinates, bookkeeping and
    # the state after a reset.
    from henon_map_cpp_b200 import _capi as C

    rng = np.random.default_rng(n)
    c = [rng.uniform(-0.3, 0.3, n) for _ in range(4)]
    t = C.Tracker(50, 0.168, 0.201, "sps", float("nan"), 16.0, 0)
    p = C.Particles(*c)
    t.track(p, 20, 0.0, 10.0)  # add_ghost restarts from the initial conditions
    for d in dirs:
        C.call("hm_particles_add_ghost", p.h, 1e-3, d.encode())
    k = 1 + len(dirs)
    assert p.size() == (n * k, n, len(dirs))
    got = p.state()
    np.testing.assert_array_equal(got[4], np.zeros(n * k, np.uint32))
    for f in range(4):
        np.testing.assert_array_equal(got[f][:n], c[f])
        for g, d in enumerate(dirs):
            ghost = got[f][n * (1 + g):n * (2 + g)]
            if d != "random":
                np.testing.assert_array_equal(
                    ghost, c[f] + 1e-3 if d == ("x", "px", "y", "py")[f] else c[f])
    for g, d in enumerate(dirs):
        if d == "random":
            off = np.stack([got[f][n * (1 + g):n * (2 + g)] - c[f] for f in range(4)])
            np.testing.assert_allclose(np.sqrt((off ** 2).sum(0)), 1e-3, rtol=1e-9)
    np.testing.assert_array_equal(p.get(C.FIELD_VALID), np.ones(n * k, np.uint8))
    np.testing.assert_array_equal(p.get(C.FIELD_GHOST), np.repeat([0] + [1] * len(dirs), n))
    np.testing.assert_array_equal(p.get(C.FIELD_IDX_BASE), np.tile(np.arange(n), k))
    np.testing.assert_array_equal(p.get(C.FIELD_IDX),
                                  np.concatenate([np.arange(n)] + [np.full(n, g) for g in
                                                                   range(len(dirs))]))
    t.track(p, 20, 0.0, 10.0)
    p.reset()
    for a, b in zip(p.state(), got):
        np.testing.assert_array_equal(a, b)
