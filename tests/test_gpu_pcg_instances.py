"""The Newton-PCG kernel's instances on either side of the sizes at which the
solver changes from one to the next: float64 with 512 threads and inlined
passes or 1024 and called ones (2^20 nodes), float inlined or called (2^21),
where a thread takes a whole coarse node of the first restriction.

The potentials against the solve with the Jacobi preconditioner in float64,
which shares none of the passes: float64 to 2e-6 V (1e-12 of the residual on
either side, a condition number of at most 1e4, 100 V); float to the last
update, whose RMS is below nr_tol, so no node's is above nr_tol sqrt(nn).  A
preconditioner that is wrong in places still converges, only later: the
neighbouring grids are one problem but for two planes of nodes, so their
counts of inner iterations differ by no more than one a Newton step and a
quarter (odd numbers of planes coarsen a little worse)."""
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


def solve(espic, nodes, fp32, nr_tol, pcg_tol, levels=12):
    w, sol = tunnel(espic, nodes)
    with w:
        sol.setNewton(30, nr_tol, 20000, pcg_tol, fp32_inner=fp32)
        sol.setMultigrid(levels)
        ok, newton, inner, _ = sol.solve()
        assert ok
        return w.phi, newton, inner


@pytest.mark.parametrize("fp32,below,above", [
    (False, (102, 102, 100), (102, 102, 102)), (True, (128, 128, 127), (128, 128, 129))])
def test_instances_on_either_side_of_their_sizes(espic, fp32, below, above):
    nr_tol, pcg_tol = (1e-6, 1e-6) if fp32 else (1e-9, 1e-12)
    edge = 1 << (21 if fp32 else 20)
    runs = []
    for nodes in (below, above):
        nn = int(np.prod(nodes))
        assert (nn <= edge) == (nodes is below)
        phi, newton, inner = solve(espic, nodes, fp32, nr_tol, pcg_tol)
        want, _, _ = solve(espic, nodes, False, 1e-9, 1e-12, levels=0)
        assert np.max(np.abs(phi - want)) <= (nr_tol * np.sqrt(nn) if fp32 else 2e-6)
        runs.append((newton, inner))
    (n0, i0), (n1, i1) = runs
    assert n0 == n1
    assert abs(i0 - i1) <= n0 + 0.25 * i0, runs


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("nodes", [(5, 5, 6), (29, 29, 30), (30, 30, 29), (33, 34, 34), (34, 34, 34), (37, 37, 37),
                                   (37, 37, 38), (42, 42, 44)])
def test_small_grids_on_their_share_of_the_sms(espic, nodes, fp32):
    """Grids at the edges of the shares of the SMs that small solves take (on
    152 SMs: a node per thread on a third with 512 threads, on half, on a
    third with 1024, on all)."""
    nr_tol, pcg_tol = (1e-6, 1e-6) if fp32 else (1e-9, 1e-12)
    phi, _, _ = solve(espic, nodes, fp32, nr_tol, pcg_tol)
    want, _, _ = solve(espic, nodes, False, 1e-9, 1e-12, levels=0)
    assert np.max(np.abs(phi - want)) <= (nr_tol * np.sqrt(phi.size) if fp32 else 2e-6)
