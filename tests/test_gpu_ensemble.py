"""The batched ensemble of grounded boxes (espic_ensemble_*).

* A box of the ensemble evolves bit for bit like the same box run as a World
  in the mixed form: charge density after the initial deposit, then, from
  the same potential, the push, the deposit and the charge density of a step.
* The solve (float32 red-black sweeps under a float64 residual) meets the
  reference's own convergence test, evaluated by the oracle's restatement of
  ch2/PotentialSolver.cpp:44-61 on the returned phi and rho, and agrees with a
  tight float64 SOR solution.
* Graph replay, direct launches and every autotuned launch shape (work-item
  size, block sizes, CTAs per box cluster) give the same bits.
* The ch2 box of the reference's golden run (3000 O+, 600 e-) stepped inside an
  ensemble keeps the reference's energy history (KE + PE) within 1e-4.
"""
import numpy as np
import pytest

from conftest import golden

pytestmark = pytest.mark.gpu

QE, AMU, ME = 1.602176565e-19, 1.660538921e-27, 9.10938215e-31
MASS = [16 * AMU, ME]
CHARGE = [QE, -QE]
X0, XM = [-0.1, -0.1, 0.0], [0.1, 0.1, 0.2]
NODES = [[21, 21, 21], [16, 16, 16], [23, 17, 29], [33, 20, 25]]
EXT = [(X0, XM), ([0.0, 0.0, 0.0], [0.05, 0.05, 0.05]), ([-0.2, -0.1, 0.0], [0.2, 0.1, 0.3]), (X0, XM)]


def box_state(x0, xm, n, seed, octant=False, vth=0.0):
    rng = np.random.default_rng(seed)
    x0, xm = np.array(x0), np.array(xm)
    hi = (x0 + xm) / 2 if octant else xm
    P = np.zeros((7, n))
    P[0:3] = (x0[:, None] + rng.random((3, n)) * (hi - x0)[:, None])
    P[3:6] = rng.standard_normal((3, n)) * vth
    return P


def build(espic, n_i=20000, n_e=4000, seed=1):
    nb = len(NODES)
    x0 = np.array([e[0] for e in EXT])
    xm = np.array([e[1] for e in EXT])
    vol = np.prod(xm - x0, axis=1)
    mpw = np.stack([1e11 * vol / n_i, 1e11 * vol / 8 / n_e], axis=1)
    E = espic.Ensemble(NODES, x0, xm, MASS, CHARGE, mpw, [[n_i + 100, n_e + 100]] * nb, 2e-10)
    states = []
    for b in range(nb):
        Pi = box_state(x0[b], xm[b], n_i, seed + 10 * b, vth=2e3)
        Pe = box_state(x0[b], xm[b], n_e, seed + 10 * b + 1, octant=True, vth=3e5)
        Pi[6], Pe[6] = mpw[b, 0], mpw[b, 1]
        E.set_particles(b, 0, Pi)
        E.set_particles(b, 1, Pe)
        states.append((Pi, Pe))
    return E, states, x0, xm, mpw


def world_for(espic, b, x0, xm, mpw, states, ens):
    w = espic.World(*NODES[b], x0[b], xm[b])
    w.setTime(2e-10, 100)
    cap = max(states[b][0].shape[1], states[b][1].shape[1]) + 100
    si = espic.Species(w, "O+", MASS[0], QE, mpw0=mpw[b, 0], capacity=cap, form=espic.FORM_MIXED)
    se = espic.Species(w, "e-", MASS[1], -QE, mpw0=mpw[b, 1], capacity=cap, form=espic.FORM_MIXED)
    si.set_particles(ens.particles(b, 0))
    se.set_particles(ens.particles(b, 1))
    return w, si, se


def test_ensemble_box_matches_world(espic):
    E, states, x0, xm, mpw = build(espic)
    with E:
        E.set_solver(10000, 1e-4, 0.0)
        E.prepare()
        for b in range(len(NODES)):
            w, si, se = world_for(espic, b, x0, xm, mpw, states, E)
            with w:
                si.computeNumberDensity()
                se.computeNumberDensity()
                w.computeChargeDensity()
                assert np.array_equal(w.rho, E.read(b, espic.FIELD_RHO)), b
                # the same potential, then one step on both
                w.write(espic.FIELD_PHI, E.read(b, espic.FIELD_PHI))
                espic.PotentialSolver(w).computeEF()
                assert np.array_equal(w.ef, E.read(b, espic.FIELD_EF)), b
        E.step(1)
        E.sync()
        # compare each box after the ensemble step with a World stepped from
        # the pre-step state: rebuild the pre-step ensemble state first
        E2, _, _, _, _ = build(espic)
        with E2:
            E2.set_solver(10000, 1e-4, 0.0)
            E2.prepare()
            for b in range(len(NODES)):
                w, si, se = world_for(espic, b, x0, xm, mpw, states, E2)
                with w:
                    w.write(espic.FIELD_PHI, E2.read(b, espic.FIELD_PHI))
                    espic.PotentialSolver(w).computeEF()
                    si.advance(deposit=True)
                    se.advance(deposit=True)
                    w.computeChargeDensity()
                    assert np.array_equal(si.particles(), E.particles(b, 0)), b
                    assert np.array_equal(se.particles(), E.particles(b, 1)), b
                    assert np.array_equal(w.rho, E.read(b, espic.FIELD_RHO)), b
                    assert np.array_equal(si.den, E.read(b, espic.FIELD_DEN, 0)), b
                    assert np.array_equal(se.den, E.read(b, espic.FIELD_DEN, 1)), b


@pytest.mark.parametrize("omega", [1.4, 0.0])
def test_ensemble_solve_meets_reference_test(espic, po, omega):
    E, states, x0, xm, mpw = build(espic)
    with E:
        E.set_solver(20000, 1e-4, omega)
        E.prepare()
        sweeps, conv, res = E.status()
        assert conv.all(), (sweeps, res)
        for b in range(len(NODES)):
            g = po.grid(NODES[b], x0[b], xm[b])
            phi, rho = E.read(b, espic.FIELD_PHI), E.read(b, espic.FIELD_RHO)
            r_oracle = po.residual_box(g, phi, rho)
            assert r_oracle < 1e-4, (b, r_oracle)
            assert abs(r_oracle - res[b]) <= 1e-6 * r_oracle + 1e-12
            tight, ok, _, _ = po.sor_box(g, np.zeros(g.nn), rho, 200000, 1e-10, "rb")
            assert ok
            assert np.max(np.abs(phi - tight)) <= 1e-5 * np.max(np.abs(tight)), b


def test_ensemble_graph_direct_and_autotune_agree(espic):
    results = []
    for mode in ("graph", "direct", "tuned"):
        E, *_ = build(espic, seed=3)
        with E:
            E.set_solver(10000, 1e-4, 0.0)
            E.prepare()
            if mode == "tuned":
                E.autotune()  # 27 real steps
                E.step(3)
            elif mode == "graph":
                E.step(30)
            else:
                E.set_launch(1024, 128, 512, 2)
                E.step(30, graph=False)
            E.sync()
            results.append([(E.particles(b, 0), E.particles(b, 1), E.read(b, espic.FIELD_PHI))
                            for b in range(len(NODES))])
    for other in results[1:]:
        for a, b in zip(results[0], other):
            for x, y in zip(a, b):
                assert np.array_equal(x, y)


def test_ensemble_reference_box_energy_history(espic):
    """The ch2 box (21^3 nodes, 3000 O+ and 600 e- from the reference's golden
    load) as box 0 of an ensemble, 40 steps: KE_i + KE_e + PE against the
    reference's FP64 history."""
    f = golden("box_steps")
    Pi0, Pe0 = f["Pi0"], f["Pe0"]
    nodes = [[21, 21, 21], [16, 16, 16]]
    x0 = np.array([X0, X0])
    xm = np.array([XM, XM])
    mpw = np.array([[Pi0[6, 0], Pe0[6, 0]], [Pi0[6, 0], Pe0[6, 0]]])
    E = espic.Ensemble(nodes, x0, xm, MASS, CHARGE, mpw, [[4000, 1000]] * 2, float(f["dt"]))
    with E:
        for b in range(2):
            E.set_particles(b, 0, Pi0)
            E.set_particles(b, 1, Pe0)
        E.set_solver(10000, 1e-4, 1.4)
        E.prepare()
        hist = f["hist"]
        worst = 0.0
        for st in range(hist.shape[0]):
            E.step(1)
            d = E.diag()
            e_ens = d[0, 0] + d[0, 1] + d[0, 2]
            ref = hist[st]
            e_ref = ref[6] + ref[12] + ref[13]
            worst = max(worst, abs(e_ens - e_ref) / abs(e_ref))
        assert worst <= 1e-4, worst


def test_sharded_ensemble_matches_whole(espic):
    """The ensemble split by work into two parts (the per-rank shards of a
    2-GPU run, stepped here one after the other on one GPU: no part waits on
    the other) evolves every box bit for bit like the whole ensemble: boxes
    load from streams keyed by their ids in the whole ensemble, and nothing
    is exchanged between parts."""
    nb = 10
    rng = np.random.default_rng(4)
    nodes = rng.integers(9, 20, size=(nb, 3))
    n_i = rng.integers(2000, 20000, size=nb)
    n_e = n_i // 4
    x0, xm = np.array(X0), np.array(XM)
    mpw = np.stack([1e11 * 0.008 / n_i, 1e11 * 0.001 / n_e], axis=1)

    def make(ids):
        E = espic.Ensemble(nodes[ids], x0, xm, MASS, CHARGE, mpw[ids], np.stack([n_i[ids], n_e[ids]], axis=1), 2e-10)
        if len(ids) < nb:
            E.set_box_ids(ids)
        E.set_seed(99)
        for loc, b in enumerate(ids):
            E.load_box(loc, 0, x0, xm, int(n_i[b]))
            E.load_box(loc, 1, x0, (x0 + xm) / 2, int(n_e[b]))
        E.set_solver(10000, 1e-4, 0.0)
        E.prepare()
        E.step(3)
        E.sync()
        return {b: (E.particles(loc, 0), E.particles(loc, 1), E.read(loc, espic.FIELD_PHI)) for loc, b in
                enumerate(ids)}, E

    owner, load = espic.partition_boxes(espic.ensemble_work(nodes, n_i + n_e), 2)
    assert set(owner) == {0, 1} and max(load) <= 1.5 * min(load)
    whole, Ew = make(np.arange(nb))
    with Ew:
        parts = {}
        for r in (0, 1):
            res, Er = make(np.nonzero(owner == r)[0])
            with Er:
                parts.update(res)
    assert sorted(parts) == list(range(nb))
    for b in range(nb):
        for a, c in zip(whole[b], parts[b]):
            assert np.array_equal(a, c), b


@pytest.mark.parametrize("cluster", [1, 8])
@pytest.mark.parametrize("nodes", [(3, 3, 3), (4, 5, 3), (16, 64, 9), (64, 17, 10), (17, 16, 64), (61, 64, 64),
                                   (120, 118, 20)])
def test_solve_routes_by_box_shape(espic, po, nodes, cluster):
    """Boxes at the edges of the shared-memory sweeps: fewer planes than CTAs,
    rows that fill no whole float4, the correction alone in shared memory,
    and one too large for it.  The solve meets the reference's test and does
    not depend on the cluster's size."""
    x0, xm = [-0.1, -0.1, 0.0], [0.1, 0.1, 0.2]
    n = 5000
    mpw = [[1e11 * 0.008 / n, 1e11 * 0.001 / n]]

    def solved(cl):
        E = espic.Ensemble([list(nodes)], x0, xm, MASS, CHARGE, mpw, [[n, n]], 2e-10)
        with E:
            E.set_launch(4096, 256, 1024, cl)
            for sp in range(2):
                P = box_state(x0, xm, n, 5 + sp, octant=sp == 1)
                P[6] = mpw[0][sp]
                E.set_particles(0, sp, P)
            E.set_solver(20000, 1e-4, 0.0)
            E.prepare()
            E.step(1)
            E.sync()
            _, conv, _ = E.status()
            return E.read(0, espic.FIELD_PHI), E.read(0, espic.FIELD_RHO), E.read(0, espic.FIELD_EF), conv

    phi, rho, ef, conv = solved(cluster)
    assert conv.all()
    g = po.grid(nodes, x0, xm)
    assert np.array_equal(ef, po.efield(g, phi))
    tight, ok, _, _ = po.sor_box(g, phi, rho, 20000, 1e-9, "rb")
    assert ok and np.max(np.abs(phi - tight)) <= 1e-5 * np.max(np.abs(tight))
    other = solved(2)
    for a, b in zip((phi, rho, ef), other):
        assert np.array_equal(a, b)


def test_two_ensembles_from_two_threads(espic):
    """An ensemble whose boxes need no slab in shared memory beside one whose
    boxes need most of it, each stepped by its own host thread: a launch must
    not depend on what the other thread set up."""
    import threading

    def make(nodes):
        n = 100
        E = espic.Ensemble([nodes], X0, XM, MASS, CHARGE, [[1e5, 1e5]], [[n, n]], 2e-10)
        E.set_launch(4096, 256, 1024, 1)
        for sp in range(2):
            P = box_state(X0, XM, n, sp)
            P[6] = 1e5
            E.set_particles(0, sp, P)
        E.set_solver(25, 1e-4, 0.0)
        E.prepare()
        return E

    errors = []

    def steps(E):
        try:
            for _ in range(800):
                E.step(1, graph=False)
            E.sync()
        except Exception as e:
            errors.append(e)

    with make([120, 118, 20]) as a, make([30, 30, 20]) as b:
        threads = [threading.Thread(target=steps, args=(E,)) for E in (a, b)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not errors, errors


@pytest.mark.parametrize("nodes", [(61, 64, 64), (4, 5, 3), (9, 10, 200)])
def test_residual_does_not_depend_on_the_cluster(espic, nodes):
    """The residuals' bits and the sweep counts of sixteen boxes' solves, for
    cluster sizes and block sizes that sweep a box in shared memory and that
    do not."""
    n, nb = 5000, 16
    mpw = [1e11 * 0.008 / n, 1e11 * 0.001 / n]
    got = []
    for cluster, threads in ((1, 1024), (2, 256), (4, 1024), (8, 512)):
        with espic.Ensemble([list(nodes)] * nb, X0, XM, MASS, CHARGE, mpw, [[n, n]] * nb, 2e-10) as E:
            E.set_launch(4096, 256, threads, cluster)
            for b in range(nb):
                for sp in range(2):
                    P = box_state(X0, XM, n, 2 * b + sp, octant=sp == 1)
                    P[6] = mpw[sp]
                    E.set_particles(b, sp, P)
            E.set_solver(75, 1e-300, 0.0)
            E.prepare()
            sweeps, _, res = E.status()
            got.append([(int(k), float(r).hex()) for k, r in zip(sweeps, res)])
    for other in got[1:]:
        assert other == got[0]
