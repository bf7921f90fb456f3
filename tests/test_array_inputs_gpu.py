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
