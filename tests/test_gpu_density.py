"""Density from the fixed-point charge on grids large enough for two nodes a
thread (4096 nodes per SM), an odd number of nodes: bit for bit the oracle's
conversion and quotient, with counts below and above 2^53 (which round), of
either sign, and the last node's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NODES, X0, XM = (87, 89, 91), [-0.1, -0.1, 0.0], [0.1, 0.1, 0.2]


def state(rng, n):
    P = np.zeros((7, n))
    P[:3] = np.array(X0)[:, None] + rng.random((3, n)) * (np.array(XM) - X0)[:, None]
    P[:3, 0] = np.nextafter(np.array(XM), -1)  # the last cell's last corner
    P[6] = 1e3 * rng.uniform(0.3, 1, n) * rng.choice([-1.0, 1.0], n)
    P[6, 0] = 1e3
    return P


@pytest.mark.parametrize("n", [1, 3, 50, 20_000])
def test_float64_density(espic, po, n):
    g = po.grid(NODES, X0, XM)
    P = state(np.random.default_rng(n), n)
    with espic.World(*NODES, X0, XM) as w:
        s = espic.Species(w, "O", 2.66e-26, 0.0, mpw0=1e3, capacity=n, form=espic.FORM_FP64, weight_bound=1e3)
        s.set_particles(P)
        s.computeNumberDensity()
        den = s.den
    fx = 2.0 ** po.fixed_scale_exponent(1e3, n)
    acc = po.deposit_fixed(g, P, fx)
    assert (np.max(np.abs(acc)) > 2 ** 53) == (n <= 50)
    want = po.density_from_fixed(acc, fx, po.node_volumes(g))
    assert np.array_equal(den, want)
    assert den[-1] != 0


def test_mixed_density(espic, po):
    g = po.grid(NODES, X0, XM)
    n = 300_000
    P = state(np.random.default_rng(9), n)
    P[6] = 1024.0
    with espic.World(*NODES, X0, XM) as w:
        s = espic.Species(w, "O", 2.66e-26, 0.0, mpw0=1024.0, capacity=n, form=espic.FORM_MIXED)
        s.set_particles(P)
        s.computeNumberDensity()
        den = s.den
        cell, off, _ = s.get_mixed()
    acc = po.deposit_mixed(g, cell, off)
    assert np.array_equal(den, po.density_from_fixed(acc, 2.0 ** 13, po.node_volumes(g)))
