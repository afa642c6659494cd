"""The linear box solver's three routes (one cluster of blocks, the whole grid
with its nodes held in registers, the whole grid without) against the oracle's
red-black SOR, bit for bit, at the edges of each: the smallest grids, thin
ones, the last box that the cluster takes and the first that it does not, a
bounded block count, and a grid past the held nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes,blocks", [
    ((3, 3, 3), 0), ((4, 3, 5), 0), ((3, 40, 9), 0), ((40, 4, 9), 0), ((5, 5, 200), 0), ((21, 21, 21), 0),
    ((21, 21, 21), 4), ((26, 25, 23), 0), ((27, 26, 24), 0), ((30, 31, 33), 0), ((62, 50, 70), 3)])
def test_sor_routes_match_the_oracle(espic, po, nodes, blocks):
    x0, xm = [-0.1, -0.1, 0.0], [0.1, 0.1, 0.2]
    g = po.grid(nodes, x0, xm)
    rng = np.random.default_rng(sum(nodes))
    rho = 1.6e-8 * rng.standard_normal(g.nn)
    its = 26
    with espic.World(*nodes, x0, xm) as w:
        w.write(espic.FIELD_RHO, rho)
        sol = espic.PotentialSolver(w, espic.SOLVER_SOR, its, 0.0)
        if blocks:
            sol.setLaunch(blocks)
        sol.solve()
        want, _, _, _ = po.sor_box(g, np.zeros(g.nn), rho, its, 0.0, "rb")
        assert np.array_equal(w.phi, want)


def test_thin_box_of_many_rows(espic, po):
    """11.6M interior rows of three entries a colour: the route with 64-bit
    division (its 46,899 entries that a float estimate would misplace lie at
    the far end)."""
    nodes, x0, xm = (7, 3402, 3402), [-0.1, -0.1, 0.0], [0.1, 0.1, 0.2]
    g = po.grid(nodes, x0, xm)
    rho = 1.6e-8 * np.random.default_rng(7).standard_normal(g.nn)
    with espic.World(*nodes, x0, xm) as w:
        w.write(espic.FIELD_RHO, rho)
        espic.PotentialSolver(w, espic.SOLVER_SOR, 2, 0.0).solve()
        want, _, _, _ = po.sor_box(g, np.zeros(g.nn), rho, 2, 0.0, "rb")
        assert np.array_equal(w.phi, want)
