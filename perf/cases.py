"""The work that programs give this framework, as cases to time.

A case is one pass through the public entry points: whole time steps of the
grounded ch2 box, of the flow past a sphere (mixed and float64 form), of the
ch4 neutral gas and of an ensemble of boxes; the ion transport and the
potential solve by themselves; a density deposit of the caller's own device
arrays; forward and backward of the differentiable sphere run.

A program that steps a World leaves its fields and particles on the GPU and
reads them when it writes output, so run() returns them as they lie there:
the values of `Held` come through the public read calls when they are looked
up.  What such a program reads every step (the diagnostics row) is read in
the pass.
"""
import ctypes
import gc
import importlib
import math

import numpy as np
import torch

E = importlib.import_module("plasma-simulations-by-example_gb300")

M_O = 16 * E.AMU
V_DRIFT, N0, TI, TE, DT_ION = 7000.0, 1e10, 0.1 * E.QE / E.K, 3.0, 1e-7
BOX_X0, BOX_XM, DT_BOX = (-0.1, -0.1, 0.0), (0.1, 0.1, 0.2), 2e-10
TUN_X0, TUN_XM, CENTER = (-0.1, -0.1, 0.0), (0.1, 0.1, 0.4), (0.0, 0.0, 0.15)
GAS_X0, GAS_XM, GAS_N, GAS_T, GAS_MPW = (-0.2, -0.1, 0.0), (0.2, 0.1, 0.4), 2e20, 1000.0, 1e12
DIFF_XM, WAKE = (0.1, 0.1, 0.3), (0.2, 0.3)


def listed():
    return [
        # a host code's own particles deposited on its own grid (no World): the
        # smallest call, three launches
        dict(name="deposit21", kind="deposit", ni=21, nj=21, nk=21, n=20_000),
        # the same entry near its grid limit, ragged sizes, unsorted particles
        dict(name="deposit97", kind="deposit", ni=97, nj=89, nk=117, n=6_000_001),
        # the ch2 program: 80,000 O+ and 10,000 electrons in the 21^3 box, one
        # iteration of its main loop with the diagnostics row
        dict(name="box21", kind="box", ni=21, nj=21, nk=21, n=90_000),
        # a small sphere run on an uneven grid: a sort period of steps, each with its row
        dict(name="sphere33", kind="sphere", form="mixed", ni=33, nj=29, nk=65, n=200_001, steps=20),
        # the reference's sphere, 64x64x128 nodes and 4M ions
        dict(name="sphere64", kind="sphere", form="mixed", ni=64, nj=64, nk=128, n=4_000_000, steps=20),
        # the same plasma in the plain float64 form (the accuracy baseline)
        dict(name="sphere64_fp64", kind="sphere", form="fp64", ni=64, nj=64, nk=128, n=4_000_000, steps=4),
        # the largest grid, 256x256x512 nodes: ten steps (one sort period)
        dict(name="sphere256", kind="sphere", form="mixed", ni=256, nj=256, nk=512, n=240_000_000, steps=10),
        # ions followed through a held field: injection, sort, push, deposit
        dict(name="transport128", kind="transport", ni=128, nj=128, nk=256, n=60_000_000, steps=10),
        # a static potential from a given charge density, float64 throughout
        dict(name="poisson64", kind="poisson", ni=64, nj=64, nk=128, fp32=False),
        # the ch4 neutral gas: its main loop's body over 6.4M atoms
        dict(name="gas41", kind="gas", ni=41, nj=21, nk=41, n=6_400_000),
        # a parameter study: 64 boxes of drawn sizes stepped together
        dict(name="ensemble64", kind="ensemble", boxes=64, lo=10_000, hi=2_000_000, steps=5),
        # gradients of a sphere run, forward and backward over 40 steps
        dict(name="diff32", kind="diff", ni=32, nj=32, nk=64, n=500_000, steps=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["deposit", "deposit", "box", "sphere", "sphere", "sphere", "sphere", "transport", "poisson",
                       "gas", "ensemble", "diff"])
    if kind == "deposit":
        ni, nj, nk = (_log(rng, 16, 100) for _ in range(3))
        return dict(kind=kind, ni=ni, nj=nj, nk=nk, n=_log(rng, 10_000, 6_000_000))
    if kind == "box":
        ni, nj, nk = (_log(rng, 13, 49) for _ in range(3))
        return dict(kind=kind, ni=ni, nj=nj, nk=nk, n=_log(rng, 20_000, 1_000_000))
    if kind in ("sphere", "transport"):
        big = rng.random() < 0.3
        ni = _log(rng, 17, 192 if big else 80)
        nj = max(17, round(ni * rng.uniform(0.8, 1.25)))
        nk = max(33, round(ni * rng.uniform(1.6, 2.4)))
        n = int(ni * nj * nk * math.exp(rng.uniform(math.log(3), math.log(15))))
        form = "fp64" if kind == "sphere" and n < 4_000_000 and rng.random() < 0.3 else "mixed"
        c = dict(kind=kind, ni=ni, nj=nj, nk=nk, n=n, steps=rng.choice([4, 5]) if form == "fp64" else rng.choice([10, 20]))
        return dict(c, form=form) if kind == "sphere" else c
    if kind == "poisson":
        ni = _log(rng, 17, 96)
        nj = max(17, round(ni * rng.uniform(0.8, 1.25)))
        return dict(kind=kind, ni=ni, nj=nj, nk=max(33, round(ni * rng.uniform(1.6, 2.4))), fp32=rng.random() < 0.5)
    if kind == "gas":
        ni, nj, nk = (_log(rng, 17, 49) for _ in range(3))
        return dict(kind=kind, ni=ni, nj=nj, nk=nk, n=_log(rng, 100_000, 6_400_000))
    if kind == "ensemble":
        hi = _log(rng, 50_000, 2_000_000)
        return dict(kind=kind, boxes=_log(rng, 8, 64), lo=10_000, hi=hi, steps=rng.choice([3, 5]))
    ni = _log(rng, 17, 32)
    return dict(kind=kind, ni=ni, nj=ni + rng.choice([-1, 0, 1]), nk=2 * ni + rng.choice([-1, 0, 1]),
                n=_log(rng, 20_000, 500_000), steps=rng.choice([20, 40]))


class Held(dict):
    """Outputs on the GPU, by name: a value is read when it is looked up."""

    def __getitem__(self, key):
        return dict.__getitem__(self, key)()


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _nodes(case):
    return case["ni"] * case["nj"] * case["nk"]


def _uniform(case, n, x0, xm, seed):
    """[7][n] float64 on the GPU: positions uniform in the box, velocities 0, weights 1."""
    P = torch.zeros((7, n), dtype=torch.float64, device="cuda")
    r = torch.rand((3, n), dtype=torch.float64, device="cuda", generator=_generator(seed))
    lo = torch.tensor(x0, dtype=torch.float64, device="cuda")[:, None]
    hi = torch.tensor(xm, dtype=torch.float64, device="cuda")[:, None]
    P[:3] = lo + r * (hi - lo)
    P[6] = 1.0
    return P


def _d3(v):
    return (ctypes.c_double * 3)(*v)


def _padded(a, length):
    """The last axis filled up with zeros: the number of particles that have
    left differs from run to run, the outputs' shapes do not."""
    return torch.nn.functional.pad(a, (0, length - a.shape[-1]))


def _components(s, form):
    """A species' particles.  The float64 form keeps their order; the mixed
    form's sort leaves the order within a cell open, so its particles, a
    set, come as each component's values in ascending order."""
    if form == "fp64":
        return {"p": _padded(torch.from_numpy(s.particles()), s.capacity)}
    cell, off, vel = (torch.from_numpy(a).cuda() for a in s.get_mixed())
    out = {"np": cell.numel()}
    for d, (shift, mask) in enumerate(((0, 1023), (10, 1023), (20, 2047))):
        x = ((cell >> shift) & mask).double() + off[d].double()
        out["x%d" % d] = _padded(torch.sort(x)[0], s.capacity)
        out["v%d" % d] = _padded(torch.sort(vel[d])[0], s.capacity)
    return out


def _tunnel(case, seed, fp32, nr_tol, pcg_tol):
    w = E.World(case["ni"], case["nj"], case["nk"], TUN_X0, TUN_XM)
    w.set_seed(seed)
    w.setTime(DT_ION, 1 << 30)
    w.addSphere(CENTER, 0.05, -100.0)
    w.addInlet()
    sol = E.PotentialSolver(w, E.SOLVER_PCG, 1000, 1e-4)
    sol.setReferenceValues(0.0, TE, N0)
    sol.setNewton(nr_max=30, nr_tol=nr_tol, pcg_max=20000, pcg_tol=pcg_tol, fp32_inner=fp32)
    return w, sol


def prepare(case, seed):
    gc.collect()  # worlds of earlier states
    kind = case["kind"]
    if kind == "deposit":
        P = _uniform(case, case["n"], BOX_X0, BOX_XM, seed)
        den = torch.empty(_nodes(case), dtype=torch.float64, device="cuda")
        flags = torch.zeros(1, dtype=torch.int32, device="cuda")
        f = E.lib().espic_deposit_noalloc
        f.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int64] + 3 * [ctypes.c_int] + 2 * [E.PD] + [
            ctypes.c_double] + 3 * [ctypes.c_void_p]
        return dict(case=case, P=P, den=den, flags=flags, f=f, x0=_d3(BOX_X0), xm=_d3(BOX_XM))
    if kind == "box":
        w = E.World(case["ni"], case["nj"], case["nk"], BOX_X0, BOX_XM)
        w.set_seed(seed)
        w.setTime(DT_BOX, 1 << 30)
        ni, ne = case["n"] - case["n"] // 9, case["n"] // 9
        si = E.Species(w, "O+", M_O, E.QE, capacity=ni)
        se = E.Species(w, "e-", E.ME, -E.QE, capacity=ne)
        si.loadParticlesBox(BOX_X0, BOX_XM, 1e11, ni)
        se.loadParticlesBox(BOX_X0, (0.0, 0.0, 0.1), 1e11, ne)
        sol = E.PotentialSolver(w, E.SOLVER_SOR, 10000, 1e-4)
        sol.solve()
        sol.computeEF()
        return dict(case=case, w=w, species=[si, se], sol=sol)
    if kind in ("sphere", "transport"):
        form = case.get("form", "mixed")
        w, sol = _tunnel(case, seed, form == "mixed", 1e-8, 1e-5)
        mpw = N0 * 0.2 * 0.2 * 0.4 / case["n"]
        s = E.Species(w, "O+", M_O, E.QE, mpw0=mpw, capacity=int(1.05 * case["n"]) + 65536,
                      form=E.FORM_MIXED if form == "mixed" else E.FORM_FP64, walls=E.WALLS_ABSORB)
        src = E.BeamSource(s, V_DRIFT, N0, TI)
        s.loadParticlesBoxThermal(TUN_X0, TUN_XM, 0.0, case["n"], (0.0, 0.0, V_DRIFT), TI)
        s.sort()
        s.computeNumberDensity()
        w.computeChargeDensity()
        sol.solve()
        sol.computeEF()
        return dict(case=case, w=w, s=s, src=src, sol=sol, form=form, row=np.zeros(7))
    if kind == "poisson":
        w, sol = _tunnel(case, seed, case["fp32"], 1e-10, 1e-7)
        rho, phi0 = _poisson_input(case, seed)
        return dict(case=case, w=w, sol=sol, rho=rho, phi0=phi0)
    if kind == "gas":
        w = E.World(case["ni"], case["nj"], case["nk"], GAS_X0, GAS_XM)
        w.set_seed(seed)
        w.setTime(DT_ION, 1 << 30)
        w.addSphere(CENTER, 0.05, -100.0)
        mpw = GAS_MPW * 6.4e6 / case["n"]
        s = E.Species(w, "O", M_O, 0.0, mpw0=mpw, capacity=int(1.25 * case["n"]) + 65536)
        src = E.BeamSource(s, V_DRIFT, GAS_N, GAS_T)
        s.set_particles(_gas_state(case, mpw, seed))
        s.enable_dsmc()
        return dict(case=case, w=w, s=s, src=src)
    if kind == "ensemble":
        return _ensemble(case, seed)
    return _diff(case, seed)


def _gas_state(case, mpw, seed):
    """Drifting thermal atoms outside the sphere."""
    g = _generator(seed)
    n = case["n"]
    P = _uniform(case, int(1.1 * n) + 1000, GAS_X0, GAS_XM, seed)
    c = torch.tensor(CENTER, dtype=torch.float64, device="cuda")[:, None]
    P = P[:, ((P[:3] - c) ** 2).sum(0) > 0.0501 ** 2][:, :n].contiguous()
    P[3:6] = torch.randn((3, n), dtype=torch.float64, device="cuda", generator=g) * math.sqrt(E.K * GAS_T / M_O)
    P[5] += V_DRIFT
    P[6] = mpw
    return P.cpu().numpy()


def _poisson_input(case, seed):
    """An ion density around n0 with particle noise, and the potential that addSphere sets."""
    rng = np.random.default_rng(seed)
    rho = E.QE * N0 * (0.6 + 0.8 * rng.random(_nodes(case)))
    phi0 = np.zeros(_nodes(case))
    phi0[_sphere(case).reshape(-1)] = -100.0
    return rho, phi0


def _sphere(case):
    """[nk][nj][ni] truth: the node lies in the sphere."""
    n = (case["ni"], case["nj"], case["nk"])
    r2 = 0.0
    for d in range(3):
        dh = (TUN_XM[d] - TUN_X0[d]) / (n[d] - 1)
        x = TUN_X0[d] + dh * np.arange(n[d]) - CENTER[d]
        r2 = r2 + (x * x).reshape([-1 if q == 2 - d else 1 for q in range(3)])
    return r2 <= 0.05 * 0.05


def _ensemble(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["boxes"] + case["hi"])  # the study's boxes do not depend on the inputs
    nb = case["boxes"]
    nodes = sizes.integers(16, 65, size=(nb, 3))
    npart = np.exp(sizes.uniform(np.log(case["lo"]), np.log(case["hi"]), size=nb)).astype(np.int64)
    dens = np.exp(rng.uniform(np.log(1e10), np.log(1e12), size=nb))
    n_i = npart // 2
    n_e = npart - n_i
    x0, xm = np.array(BOX_X0), np.array(BOX_XM)
    vol = np.prod(xm - x0)
    mpw = np.stack([dens * vol / n_i, dens * vol / 8 / n_e], axis=1)
    ens = E.Ensemble(nodes, x0, xm, [M_O, E.ME], [E.QE, -E.QE], mpw, np.stack([n_i, n_e], axis=1), DT_BOX)
    ens.set_seed(seed)
    mid = (x0 + xm) / 2
    for b in range(nb):
        octant = rng.integers(0, 8) >> np.arange(3) & 1
        ens.load_box(b, 0, x0, xm, n_i[b])
        ens.load_box(b, 1, np.where(octant, mid, x0), np.where(octant, xm, mid), n_e[b])
    ens.set_solver(10000, 1e-4, 0.0)
    ens.prepare()
    return dict(case=case, ens=ens)


def _diff(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    x0, xm, c = np.array(TUN_X0), np.array(DIFF_XM), np.array(CENTER)
    pos = x0 + rng.random((2 * n + 1000, 3)) * (xm - x0)
    pos = pos[np.sum((pos - c) ** 2, axis=1) > 0.055 ** 2][:n]
    x = np.ascontiguousarray(pos.T)
    v = rng.normal(0, math.sqrt(0.1 * E.QE / M_O), (3, n))
    v[2] += V_DRIFT
    w = E.World(case["ni"], case["nj"], case["nk"], TUN_X0, DIFF_XM)
    w.setTime(DT_ION, 1 << 30)
    w.addSphere(CENTER, 0.05, -100.0)
    w.addInlet()
    sol = E.PotentialSolver(w, E.SOLVER_PCG, 100, 1e-4)
    sol.setReferenceValues(0.0, TE, N0)
    sol.setNewton(nr_max=60, nr_tol=1e-12, pcg_max=5000, pcg_tol=1e-10, fp32_inner=False)
    dh = min((xm - x0) / (np.array([case["ni"], case["nj"], case["nk"]]) - 1))
    run_ = E.DiffRun(w, n=n, mass=M_O, charge=E.QE, mpw0=N0 * 0.0115 / n, delta=0.5 * dh, wake_z=WAKE, alpha=1e8,
                     beta=1e-7, checkpoint_every=20)
    return dict(case=case, w=w, run=run_, x=x, v=v)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "deposit":
        rc = st["f"](st["P"].data_ptr(), case["n"], case["n"], case["ni"], case["nj"], case["nk"], st["x0"], st["xm"],
                     1.0, st["den"].data_ptr(), st["flags"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        E.check(rc)
        return {"den": st["den"], "flags": st["flags"]}
    if kind == "box":
        w, (si, se), sol = st["w"], st["species"], st["sol"]
        w.advanceTime()
        si.advance(deposit=True)
        se.advance(deposit=True)
        w.computeChargeDensity()
        sol.solve(wait=False)
        sol.computeEF()
        row = w.diag_row()
        return Held(row=lambda: row, phi=lambda: w.phi, rho=lambda: w.rho, ef=lambda: w.ef, ions=si.particles,
                    electrons=se.particles)
    if kind == "sphere":
        w, s, form = st["w"], st["s"], st["form"]
        for _ in range(case["steps"]):
            w.advanceTime()
            row = w.step(case["steps"], st["row"])
        row = row.copy()
        return Held(row=lambda: row, phi=lambda: w.phi, rho=lambda: w.rho, den=lambda: s.den,
                    ions=lambda: _components(s, form))
    if kind == "transport":
        w, s, src = st["w"], st["s"], st["src"]
        s.sort()
        for _ in range(case["steps"]):
            src.sample()
            s.advance(deposit=True)
        return Held(den=lambda: s.den, ions=lambda: _components(s, "mixed"))
    if kind == "poisson":
        w, sol = st["w"], st["sol"]
        w.write(E.FIELD_RHO, st["rho"])
        w.write(E.FIELD_PHI, st["phi0"])
        sol.solve(wait=False)
        sol.computeEF()
        return Held(phi=lambda: w.phi, ef=lambda: w.ef)
    if kind == "gas":
        w, s = st["w"], st["s"]
        w.advanceTime()
        st["src"].sample()
        s.computeNumberDensity()
        s.sampleMoments()
        s.computeGasProperties()
        s.dsmc(DT_ION)
        s.advance_ch4()
        s.computeMPC()
        return Held(den=lambda: s.den, vel=lambda: s.vel, T=lambda: s.T, mpc=lambda: s.mpc, moments=lambda: s.moments,
                    p=lambda: _components(s, "fp64"))
    if kind == "ensemble":
        ens = st["ens"]
        ens.step(case["steps"])
        nb = case["boxes"]

        def cat(f, count):
            return np.concatenate([np.ravel(f(b)) for b in range(count)])

        return Held(phi=lambda: cat(lambda b: ens.read(b, E.FIELD_PHI), nb),
                    rho=lambda: cat(lambda b: ens.read(b, E.FIELD_RHO), nb),
                    ions=lambda: cat(lambda b: ens.particles(b, 0)[:6], nb),
                    electrons=lambda: cat(lambda b: ens.particles(b, 1)[:6], nb))
    st["run"].set_state(st["x"], st["v"])
    loss = st["run"].forward(-100.0, case["steps"])
    dphi_s, dx, dv = st["run"].backward()
    return {"loss": loss, "dphi_s": dphi_s, "dx": dx, "dv": dv}


def work(case):
    """One pass: particle state read and written once a step, node fields
    read and written once a step, the arithmetic of the particle step (about
    130 operations for gather, move and deposit) and of a field step (about
    60 a node: one residual and one E)."""
    kind = case["kind"]
    n = case.get("n", 0)
    if kind == "deposit":
        return {"bytes": 32.0 * n + 8.0 * _nodes(case), "flops": 45.0 * n}
    if kind == "box":
        return {"bytes": 96.0 * n + 64.0 * _nodes(case), "flops": 130.0 * n + 60.0 * _nodes(case)}
    if kind in ("sphere", "transport"):
        per = 96.0 if case.get("form") == "fp64" else 56.0
        field = (64.0, 60.0) if kind == "sphere" else (24.0, 0.0)
        return {"bytes": case["steps"] * (per * n + field[0] * _nodes(case)),
                "flops": case["steps"] * (130.0 * n + field[1] * _nodes(case))}
    if kind == "poisson":
        return {"bytes": 64.0 * _nodes(case), "flops": 60.0 * _nodes(case)}
    if kind == "gas":
        return {"bytes": 104.0 * n + 160.0 * _nodes(case), "flops": 400.0 * n}
    if kind == "ensemble":
        sizes = np.random.default_rng(case["boxes"] + case["hi"])
        nodes = float(np.prod(sizes.integers(16, 65, size=(case["boxes"], 3)), axis=1).sum())
        npart = float(np.exp(sizes.uniform(np.log(case["lo"]), np.log(case["hi"]), size=case["boxes"])).sum())
        return {"bytes": case["steps"] * (56.0 * npart + 64.0 * nodes),
                "flops": case["steps"] * (130.0 * npart + 60.0 * nodes)}
    # forward, its replay and the adjoint: three passes over the state a step
    return {"bytes": case["steps"] * 3 * (104.0 * n + 64.0 * _nodes(case)),
            "flops": case["steps"] * 3 * (130.0 * n + 60.0 * _nodes(case))}


def exact(case, seed):
    if case["kind"] == "deposit":
        return _exact_deposit(case, seed)
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    return None  # a chaotic trajectory over several steps has no such value


def _exact_deposit(case, seed):
    x = _uniform(case, case["n"], BOX_X0, BOX_XM, seed)[:3]
    n = (case["ni"], case["nj"], case["nk"])
    cell, frac, vol = [], [], torch.ones((n[2], n[1], n[0]), dtype=torch.float64, device=x.device)
    for d in range(3):
        dh = (BOX_XM[d] - BOX_X0[d]) / (n[d] - 1)
        l = (x[d] - BOX_X0[d]) / dh
        c = l.floor().long().clamp(0, n[d] - 2)
        cell.append(c)
        frac.append(l - c)
        h = torch.full((n[d],), dh, dtype=torch.float64, device=x.device)
        h[0] *= 0.5
        h[-1] *= 0.5
        vol *= h.reshape([-1 if q == 2 - d else 1 for q in range(3)])
    den = torch.zeros(_nodes(case), dtype=torch.float64, device=x.device)
    for m in range(8):
        w, u = 1.0, 0
        for d in (2, 1, 0):
            b = m >> d & 1
            w = w * (frac[d] if b else 1 - frac[d])
            u = u * n[d] + cell[d] + b
        den.index_add_(0, u, w)
    return {"den": den / vol.reshape(-1), "flags": None}


def _exact_poisson(case, seed):
    """Newton with Jacobi-preconditioned CG in float64 on the 7-point Poisson
    equation with Boltzmann electrons: sphere and inlet nodes hold their
    potential, the other boundary nodes copy their inner neighbour."""
    rho, phi = (torch.from_numpy(a).cuda().reshape(case["nk"], case["nj"], case["ni"])
                for a in _poisson_input(case, seed))
    n = (case["ni"], case["nj"], case["nk"])
    dh = [(TUN_XM[d] - TUN_X0[d]) / (n[d] - 1) for d in range(3)]
    fixed = torch.from_numpy(_sphere(case)).cuda()
    fixed[0] = True
    phi = phi.clone()
    phi[0] = 0.0
    inner = torch.zeros_like(fixed)
    inner[1:-1, 1:-1, 1:-1] = True
    free = inner & ~fixed
    wall = ~inner & ~fixed
    links = []  # per axis, between i and i + 1: 1 / dh^2 where an unknown sees a node that is not its own copy
    for d in range(3):
        free0, free1, wall0, wall1 = (t.narrow(2 - d, s, n[d] - 1) for t in (free, wall) for s in (0, 1))
        links.append(((free0 & ~wall1) | (free1 & ~wall0)).double() / dh[d] ** 2)
    eps0, te = E.EPS_0, TE

    def minus_laplacian(p):
        out = torch.zeros_like(p)
        for d in range(3):
            ax = 2 - d
            flux = links[d] * (p.narrow(ax, 1, n[d] - 1) - p.narrow(ax, 0, n[d] - 1))
            out.narrow(ax, 0, n[d] - 1).sub_(flux)
            out.narrow(ax, 1, n[d] - 1).add_(flux)
        return out * free

    diag = torch.zeros_like(phi)
    for d in range(3):
        diag.narrow(2 - d, 0, n[d] - 1).add_(links[d])
        diag.narrow(2 - d, 1, n[d] - 1).add_(links[d])
    for _ in range(40):
        ne = E.QE * N0 * torch.exp(phi / te) / eps0 * free
        res = (rho / eps0 * free - ne) - minus_laplacian(phi)
        jd = ne / te
        pre = torch.where(free, 1.0 / (diag + jd), torch.zeros_like(diag))
        y, r = torch.zeros_like(res), res.clone()
        z = pre * r
        p, rz, stop = z.clone(), (r * z).sum(), 1e-11 * res.norm()
        for it in range(4000):
            q = minus_laplacian(p) + jd * p
            alpha = rz / (p * q).sum()
            y += alpha * p
            r -= alpha * q
            if it % 20 == 19 and bool(r.norm() <= stop):
                break
            z = pre * r
            new = (r * z).sum()
            p = z + new / rz * p
            rz = new
        phi = phi + y
        if float(y.square().mean().sqrt()) < 1e-11:
            break
    for ax, size in ((0, n[2]), (1, n[1]), (2, n[0])):  # x faces last: they come first in a chain of copies
        for at, of in ((0, 1), (size - 1, size - 2)):
            face, src, w = phi.select(ax, at), phi.select(ax, of), wall.select(ax, at)
            face.copy_(torch.where(w, src, face))
    ef = torch.empty((case["nk"], case["nj"], case["ni"], 3), dtype=torch.float64, device=phi.device)
    for d in range(3):
        ax, m = 2 - d, n[d]
        e, p = ef[..., d], lambda i, ax=ax: phi.select(ax, i)  # noqa: E731
        e.narrow(ax, 1, m - 2).copy_(-(phi.narrow(ax, 2, m - 2) - phi.narrow(ax, 0, m - 2)) / (2 * dh[d]))
        e.select(ax, 0).copy_(-(-3 * p(0) + 4 * p(1) - p(2)) / (2 * dh[d]))
        e.select(ax, m - 1).copy_(-(p(m - 3) - 4 * p(m - 2) + 3 * p(m - 1)) / (2 * dh[d]))
    return {"phi": phi.reshape(-1), "ef": ef.reshape(-1, 3)}
