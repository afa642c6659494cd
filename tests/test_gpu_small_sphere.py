"""The float64 push's float test against the sphere, which only lets a
particle skip the float64 one when it lies surely outside: in a world so small
that squared distances leave the float range's normal numbers, every particle
inside the sphere is still removed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-24, 1e-22, 1e-20, 1e-18, 1.0, 1e18])
def test_particles_inside_are_removed(espic, scale):
    radius, half = 1.0 * scale, 4.0 * scale
    rng = np.random.default_rng(22)
    x = rng.standard_normal((3, 20_000))
    x *= radius * rng.uniform(0.85, 1.15, 20_000) / np.sqrt((x ** 2).sum(0))
    P = np.zeros((7, x.shape[1]))
    P[:3], P[6] = x, 1.0
    inside = ((x[0] * x[0] + x[1] * x[1]) + x[2] * x[2]) <= radius * radius
    assert 5000 < inside.sum() < 15000
    with espic.World(9, 9, 9, [-half] * 3, [half] * 3) as w:
        w.setTime(1e-7, 10)
        w.addSphere([0.0, 0.0, 0.0], radius, -1.0)
        s = espic.Species(w, "O", 2.66e-26, 1.602176565e-19, mpw0=1.0, capacity=x.shape[1], form=espic.FORM_FP64,
                          walls=espic.WALLS_ABSORB)
        s.set_particles(P)
        s.advance(deposit=False)
        left = s.particles()
    assert left.shape[1] == np.sum(~inside)
