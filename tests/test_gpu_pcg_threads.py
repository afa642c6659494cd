"""Newton-PCG solves of several worlds at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tunnel(espic, nodes):
    w = espic.World(*nodes, [-0.1, -0.1, 0.0], [0.1, 0.1, 0.4])
    w.addSphere([0.0, 0.0, 0.15], 0.05, -100.0)
    w.addInlet()
    w.write(espic.FIELD_RHO, 1.6e-9 * (1 + 0.3 * np.random.default_rng(5).random(int(np.prod(nodes)))))
    sol = espic.PotentialSolver(w, espic.SOLVER_PCG, 10000, 1e-4)
    sol.setReferenceValues(0.0, 1.5, 1e10)
    return w, sol


def test_two_worlds_from_two_threads(espic):
    """A world whose coarse levels run in one block's shared memory (119 KB)
    beside one that needs none, each solved by its own host thread: a launch
    must not depend on what the other thread set up."""
    errors = []

    def solves(sol):
        try:
            for _ in range(2000):
                sol.solve(wait=False)
            sol.solve()
        except Exception as e:
            errors.append(e)

    (wa, a), (wb, b) = tunnel(espic, (34, 34, 66)), tunnel(espic, (34, 34, 66))
    with wa, wb:
        a.setNewton(30, 1e-9, 1000, 1e-12)
        a.setDense(0)
        a.setCoarse(2048)
        b.setNewton(30, 1e-9, 1000, 1e-12)
        threads = [threading.Thread(target=solves, args=(s,)) for s in (a, b)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not errors, errors
