"""The multigrid preconditioner's routes: half sweeps merged into one phase per
level or run one by one (a bound on the blocks leaves a level more items than
threads), the coarsest level's dense inverse with its rows in shared memory or
in place, and the block-local levels.

The nonlinear solve of a sphere in a box.  Float64 inner solves against the
solve with the Jacobi preconditioner, which shares none of the routes: a
relative residual of 1e-12 leaves an error below cond 1e-12 |phi| <= 1e4 1e-12
100 V on either side, 2e-6 V together.  Float inner solves (whose own error
against that is larger, a few 1e-2 V) against the run with two blocks, where
no large level is merged: the stop at an RMS update of 1e-4 V allows 1e-2 V at
the worst node.  A preconditioner that is
wrong in places still converges, only later: the routes may differ by one
inner iteration a Newton step (the dot products' order), no more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(espic, nodes, fp32, levels=12, blocks=0, dense=1024, coarse=None):
    with espic.World(*nodes, [-0.1, -0.1, 0.0], [0.1, 0.1, 0.4]) as w:
        w.addSphere([0.0, 0.0, 0.15], 0.05, -100.0)
        w.addInlet()
        w.write(espic.FIELD_RHO, 1.6e-9 * (1 + 0.3 * np.random.default_rng(sum(nodes)).random(int(np.prod(nodes)))))
        sol = espic.PotentialSolver(w, espic.SOLVER_PCG, 10000, 1e-4)
        sol.setReferenceValues(0.0, 1.5, 1e10)
        sol.setNewton(30, 1e-4 if fp32 else 1e-9, 10000, 1e-6 if fp32 else 1e-12, fp32_inner=fp32)
        sol.setMultigrid(levels)
        sol.setLaunch(blocks)
        sol.setDense(dense)
        if coarse is not None:
            sol.setCoarse(coarse)
        ok, newton, inner, _ = sol.solve()
        assert ok
        return w.phi, newton, inner


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("nodes,dense", [
    ((5, 5, 6), 1024), ((9, 6, 17), 1024), ((18, 34, 50), 1024), ((33, 29, 65), 1024), ((33, 29, 65), 2048),
    ((40, 40, 80), 4096), ((64, 64, 128), 1024)])
def test_multigrid_routes(espic, nodes, dense, fp32):
    phi, newton, inner = solve(espic, nodes, fp32, dense=dense)
    few, newton2, inner2 = solve(espic, nodes, fp32, dense=dense, blocks=2)
    want = few if fp32 else solve(espic, nodes, fp32, levels=0)[0]
    tol = 1e-2 if fp32 else 2e-6
    assert np.max(np.abs(phi - want)) <= tol
    assert np.max(np.abs(few - want)) <= tol
    assert newton == newton2
    assert abs(inner - inner2) <= newton


def test_block_local_levels(espic):
    want, _, _ = solve(espic, (18, 34, 50), False, levels=0)
    phi, _, _ = solve(espic, (18, 34, 50), False, dense=0, coarse=512)
    assert np.max(np.abs(phi - want)) <= 2e-6
