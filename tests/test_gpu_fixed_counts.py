"""Fixed-point counts made with integer operations: the float64 charge deposit
and the gas moments, at the edges of a warp and over the whole range of a
count.

* espic_deposit_noalloc on a grid whose spacings are powers of two, against
  the same sums in Python integers: every corner weight
  value (1-di)(1-dj)(1-dk) in the reference's operand order, rounded once
  (ties to even) to a count, added exactly.  Bit for bit; one particle makes
  the largest counts (2^61 and above take the conversion), many make small
  ones.  Positions lie on nodes, on cell faces, on both ends of the domain
  and outside it.
* sampleMoments against the oracle: a count is rounded by at most half of
  2^-S <= b 2^-50 for the largest value b of a sum, a corner's product on
  either side by at most 4 b 2^-53 together, and a float64 sum of n such terms
  by n^2 b 2^-53, so that n b (2^-50 + n 2^-53) bounds a node's difference.
"""
import ctypes as C
import math
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID, X0, XM = (9, 5, 5), (-0.5, 0.0, 0.25), (0.5, 1.0, 1.25)
DH = np.array([0.125, 0.25, 0.25])


def positions(rng, n, outside):
    x = rng.random((3, n)) * (np.array(XM) - X0)[:, None] + np.array(X0)[:, None]
    edge = rng.random((3, n))
    cell = np.array(X0)[:, None] + DH[:, None] * rng.integers(0, np.array(GRID)[:, None], (3, n))
    x = np.where(edge < 0.2, cell, x)
    if outside:
        x[0, rng.random(n) < 0.1] = XM[0] + 0.01
        x[1, rng.random(n) < 0.1] = X0[1] - 0.3
    return x


@pytest.mark.parametrize("n,spread", [(1, 0), (2, 0), (31, 3), (33, 40), (257, 12), (1000, 70)])
def test_deposit_counts(espic, n, spread):
    import torch
    rng = np.random.default_rng(n)
    P = np.zeros((7, n))
    P[:3] = positions(rng, n, outside=n > 2)
    P[6] = rng.choice([-1.0, 1.0], n) * rng.uniform(0.5, 1, n) * 2.0 ** -rng.integers(0, spread + 1, n)
    P[6, 0] = 1.0
    P[6] *= 2.0 ** 40
    wb = 2.0 ** 40
    S = min(52, math.frexp(2.0 ** 62 / (n * wb))[1] - 1)
    f = espic.lib().espic_deposit_noalloc
    f.argtypes = [C.c_void_p, C.c_int64, C.c_int64, C.c_int, C.c_int, C.c_int, C.POINTER(C.c_double),
                  C.POINTER(C.c_double), C.c_double, C.c_void_p, C.c_void_p, C.c_void_p]
    nn = GRID[0] * GRID[1] * GRID[2]
    den = torch.zeros(nn, dtype=torch.float64, device="cuda")
    dP = torch.from_numpy(P).to("cuda")
    rc = f(dP.data_ptr(), n, n, *GRID, (C.c_double * 3)(*X0), (C.c_double * 3)(*XM), wb, den.data_ptr(), None,
           torch.cuda.current_stream().cuda_stream)
    assert rc == 0, espic.last_error()
    torch.cuda.synchronize()
    want = [0] * nn
    for p in range(n):
        c, d = [], []
        for a in range(3):
            lc = (P[a, p] - X0[a]) / DH[a]
            c.append(min(max(int(lc), 0), GRID[a] - 2))
            d.append(lc - c[-1])
        v = float(P[6, p]) * 2.0 ** S
        for k in (0, 1):
            for j in (0, 1):
                for i in (0, 1):
                    w = v * (d[0] if i else 1 - d[0])
                    w *= d[1] if j else 1 - d[1]
                    w *= d[2] if k else 1 - d[2]
                    want[((c[2] + k) * GRID[1] + c[1] + j) * GRID[0] + c[0] + i] += round(w)
    got = den.cpu().numpy()
    V = DH.prod()
    for u in range(nn):
        ijk = (u % GRID[0], u // GRID[0] % GRID[1], u // (GRID[0] * GRID[1]))
        faces = sum(t in (0, m - 1) for t, m in zip(ijk, GRID))
        assert got[u] == float(want[u]) * 2.0 ** (faces - S) / V, (u, got[u], want[u])


@pytest.mark.parametrize("n,uniform", [(1, False), (33, False), (33, True), (257, False)])
def test_moment_counts(espic, po, n, uniform):
    rng = np.random.default_rng(n)
    P = np.zeros((7, n))
    P[:3] = positions(rng, n, outside=False)
    P[:3] = np.minimum(P[:3], np.nextafter(np.array(XM), -1)[:, None])
    P[3:6] = 700 * rng.standard_normal((3, n)) * 2.0 ** -rng.integers(0, 40, n)
    P[4, rng.random(n) < 0.2] = 0.0
    P[6] = 1e12 if uniform else 1e12 * 2.0 ** -rng.integers(0, 60, n)
    g = po.grid(GRID, X0, XM)
    nn = int(np.prod(GRID))
    ref = po.sample_moments(g, P).reshape(7, nn)
    with espic.World(*GRID, X0, XM) as w:
        w.setTime(1e-7, 10)
        kw = {} if uniform else {"weight_bound": 1e12}
        s = espic.Species(w, "O", 2.66e-26, 0.0, mpw0=1e12, capacity=n + 3, form=espic.FORM_FP64, **kw)
        s.set_particles(P)
        s.sampleMoments()
        mom = s.moments
    values = [P[6]] + [P[6] * P[3 + d] for d in range(3)] + [P[6] * P[3 + d] ** 2 for d in range(3)]
    for q in range(7):
        assert np.max(np.abs(mom[q] - ref[q])) <= n * np.max(np.abs(values[q])) * (2.0 ** -50 + n * 2.0 ** -53), q


@pytest.mark.parametrize("n,spread", [(4096, 0), (4099, 30)])
def test_deposit_counts_below_the_conversions(espic, monkeypatch, n, spread):
    """Every count below 2^51 (2^40 2^S with S <= 10), cells up to 1023: the
    products and offsets that are integer operations throughout."""
    here = sys.modules[__name__]
    monkeypatch.setattr(here, "GRID", (1025, 3, 5))
    monkeypatch.setattr(here, "DH", np.array([2.0 ** -10, 0.5, 0.25]))
    test_deposit_counts(espic, n, spread)
