"""The work that is timed: partitioning jobs and density evaluations through the package's public entry points.

Kinds of case (``kind``):

``call``      one whole ``do_partitioning`` of a partitioning class on host arrays, as a script runs it: job creation,
              every iteration, charges, parameters, promolecule and at_weights back on the host
``run``       one resident job from its initial parameters to convergence (``Job.reset``, ``run``, ``results``), as a
              program does that partitions the same grid again
``steps``     the first outer iterations of one job or of a batch of jobs that share launches (``Context.step``); MBIS
              and aLISA on larger molecules take hundreds of them, all alike
``evaluate``  the evaluation service that the host-iterated gLISA solvers call (objective, gradient, Hessian)
``density``   the electron density of a contracted-Gaussian wavefunction on grid points (``DensityPlan``)

All inputs are synthetic and made from the seed: bonded chains of the case's formula, Slater-shell densities with
jittered exponents and smooth bumps, Becke grids (see ``horton_part_gb300.synthetic``).
"""

from __future__ import annotations

import logging
import math
import re

import numpy as np
import torch

from horton_part_gb300 import _lib, synthetic
from horton_part_gb300.density import DensityPlan
from horton_part_gb300.mbis import get_initial_mbis_propars, get_nshell
from horton_part_gb300.molgrid import AtomGrid, MolecularGrid, radial_becke_gauss_chebyshev
from horton_part_gb300.utils import wpart_schemes

SYMBOLS = {"H": 1, "C": 6, "N": 7, "O": 8}
# shells per element of the Gaussian bases (exponents geometric in [0.05, 300])
BASIS_SHELLS = {1: 6, 6: 9, 7: 9, 8: 9}
CUTOFF = 1e-15  # the classes' density_cutoff

LOG = logging.getLogger("perf.cases")
LOG.setLevel(logging.WARNING)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest partitioning: one water molecule through the class with its default options (FP64,
        # threshold 1e-6) on the molecular grid; short kernels, so launches and host waits count
        dict(name="mbis-water-call", kind="call", scheme="mbis", precision="fp64", grid_type=3, formula="H2O",
             nrad=75, nang=110, threshold=1e-6),
        # the classes' default grid_type: atom grids, inner solves on spherical averages
        dict(name="mbis-atomgrid-call", kind="call", scheme="mbis", precision="fp64", grid_type=1, formula="C2H6O",
             nrad=75, nang=110, threshold=1e-6),
        # an ordinary molecule in the default precision
        dict(name="mbis-chain", kind="steps", scheme="mbis", precision="fp64", formula="C8H11NO2", nrad=75, nang=194,
             steps=2, threshold=1e-8, molecules=1),
        # the largest molecule of the batched mix, float-float
        dict(name="mbis-ff-chain60", kind="steps", scheme="mbis", precision="ff", formula="C20H34N3O3", nrad=75,
             nang=194, steps=2, threshold=1e-8, molecules=1),
        # a batch of molecules of uneven size that share launches, mixed precision
        dict(name="mbis-batch-mixed", kind="steps", scheme="mbis", precision="mixed", formula="C10H17NO2", nrad=75,
             nang=194, steps=2, threshold=1e-8, molecules=8),
        # GISA on the 20-atom benchmark molecule, to convergence
        dict(name="gisa-run", kind="run", scheme="gisa", precision="fp64", formula="C6H10N2O2", nrad=100, nang=302,
             threshold=1e-6, maxiter=500),
        # aLISA's self-consistent solver, one outer iteration with at most 50 inner ones
        dict(name="alisa-chain", kind="steps", scheme="lisa", precision="fp64", formula="C10H16N2O2", nrad=75,
             nang=194, steps=1, threshold=1e-6, molecules=1),
        # the benchmark job: gLISA with non-negative populations, tensor-core Hessian
        dict(name="glisa-mixed-run", kind="run", scheme="glisa", precision="mixed", formula="C6H10N2O2", nrad=100,
             nang=302, threshold=1e-8, maxiter=100),
        # gLISA through the class with its default solver and precision
        dict(name="glisa-call", kind="call", scheme="glisa", precision="fp64", grid_type=3, formula="C3H6O",
             nrad=60, nang=110, threshold=1e-6),
        # one evaluation with and one without the Hessian, as the host-iterated solvers ask for them
        dict(name="glisa-evaluate", kind="evaluate", scheme="glisa", precision="fp64", formula="C6H10N2O2", nrad=100,
             nang=302, threshold=1e-6),
        # the density generator on a whole molecular grid, points and density on the device
        dict(name="density-chain", kind="density", formula="C6H10N2O2", nrad=100, nang=302, spin=False, host=False),
        # the smallest call: density and spin density of water on host points
        dict(name="density-water-host", kind="density", formula="H2O", nrad=30, nang=50, spin=True, host=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_formula(rng, lo, hi, even=False):
    """A formula of lo..hi atoms, H : C : N : O about 10 : 6 : 1 : 1 (`even`: an even number of heavy atoms)."""
    n = _log_int(rng, lo, hi)
    c = max(1, round(n * rng.uniform(0.25, 0.4)))
    o = max(0, round(n * rng.uniform(0.0, 0.12)))
    ni = max(0, round(n * rng.uniform(0.0, 0.12)))
    if even:
        c += (c + o + ni) % 2
    return "C%dH%dN%dO%d" % (c, max(1, n - c - o - ni), ni, o)


def draw(rng):
    kind = rng.choice(["call", "call", "steps", "steps", "run", "evaluate", "density"])
    nang = rng.choice([50, 110, 194, 302])
    if kind == "call":
        scheme = rng.choice(["mbis", "mbis", "glisa", "gisa"])
        return dict(kind=kind, scheme=scheme, precision="fp64", grid_type=rng.choice([1, 3]),
                    formula=_draw_formula(rng, 3, 8), nrad=_log_int(rng, 20, 75), nang=rng.choice([50, 110]),
                    threshold=1e-6)
    if kind == "steps":
        scheme, precision = rng.choice([("mbis", "fp64"), ("mbis", "ff"), ("mbis", "mixed"), ("lisa", "fp64")])
        big = 20 if precision == "fp64" else 50
        return dict(kind=kind, scheme=scheme, precision=precision, formula=_draw_formula(rng, 4, big),
                    nrad=_log_int(rng, 25, 75), nang=min(nang, 194), steps=1, threshold=1e-8,
                    molecules=rng.choice([1, 1, 2, 4]) if precision != "fp64" else 1)
    if kind == "run":
        scheme, precision = rng.choice([("gisa", "fp64"), ("glisa", "mixed"), ("glisa", "mixed")])
        # mixed gLISA: molecules with an even number of shells (those with an odd one are not measured)
        return dict(kind=kind, scheme=scheme, precision=precision,
                    formula=_draw_formula(rng, 3, 18, even=scheme == "glisa"),
                    nrad=_log_int(rng, 25, 90), nang=nang, threshold=1e-8 if scheme == "glisa" else 1e-6,
                    maxiter=100 if scheme == "glisa" else 500)
    if kind == "evaluate":
        return dict(kind=kind, scheme="glisa", precision="fp64", formula=_draw_formula(rng, 3, 18),
                    nrad=_log_int(rng, 25, 90), nang=nang, threshold=1e-6)
    return dict(kind=kind, formula=_draw_formula(rng, 3, 18), nrad=_log_int(rng, 20, 90), nang=nang,
                spin=rng.choice([False, True]), host=rng.choice([False, True]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _counts(formula):
    return {SYMBOLS[s]: int(n or 1) for s, n in re.findall(r"([A-Z])(\d*)", formula) if int(n or 1) > 0}


def _natom(case):
    return sum(_counts(case["formula"]).values())


def _molecule(case, seed, counts=None):
    counts = counts or _counts(case["formula"])
    nrad, nang = case["nrad"], case["nang"]
    if counts == {1: 2, 8: 1}:
        mol = synthetic.water(nrad, nang, seed=seed)
    else:
        mol = synthetic.peptide_molecule(counts, nrad, nang, seed=seed)
    if case.get("grid_type") == 1:
        r, wr = radial_becke_gauss_chebyshev(nrad)
        g = mol.grid
        grid = MolecularGrid(g.points, g.weights, indices=g.indices,
                             atgrids=[AtomGrid(r, wr, nang) for _ in range(mol.natom)])
        mol = synthetic.Molecule(mol.coordinates, mol.numbers, grid, mol.density, name=mol.name)
    return mol


def _molecules(case, seed):
    """The molecules of a batch: the formula scaled to 1, 5/6, 4/6, ... of its atoms, at least a tenth."""
    base, mols = _counts(case["formula"]), []
    for m in range(case.get("molecules", 1)):
        f = max(0.1, 1.0 - m / 6.0)
        mols.append(_molecule(case, seed + 1000 * m, {z: max(1, round(n * f)) for z, n in base.items()}))
    return mols


def _basis():
    return synthetic.geometric_gaussian_basis(BASIS_SHELLS, 0.05, 300.0)


def _shells(scheme, mol):
    """(offsets, initial parameters, orders, exponents) of a job, as the classes form them."""
    if scheme == "mbis":
        off = np.concatenate([[0], np.cumsum([int(get_nshell(z)) for z in mol.numbers])]).astype(np.int32)
        return off, np.concatenate([get_initial_mbis_propars(z) for z in mol.numbers]), None, None
    h = _basis()
    off = np.concatenate([[0], np.cumsum([h.get_nshell(z) for z in mol.numbers])]).astype(np.int32)
    init = np.concatenate([np.full(h.get_nshell(z), float(z) / h.get_nshell(z)) for z in mol.numbers])
    return (off, init, np.concatenate([h.get_order(z) for z in mol.numbers]),
            np.concatenate([h.get_exponent(z) for z in mol.numbers]))


def _job(case, mol):
    off, init, orders, exps = _shells(case["scheme"], mol)
    solver = {"mbis": "default", "gisa": "quadprog", "lisa": "sc", "glisa": "pnewton"}[case["scheme"]]
    inner = {"mbis": 2000, "lisa": 50}.get(case["scheme"], 0)
    return _lib.Job(_lib.default_context(0), case["scheme"], mol.coordinates, mol.pseudo_numbers, mol.grid.points,
                    mol.grid.weights, mol.density, off, init, shell_orders=orders, shell_exponents=exps,
                    solver=solver, precision=case["precision"], grid_type=3, threshold=case["threshold"],
                    inner_threshold=case["threshold"], maxiter=case.get("maxiter", 500), inner_maxiter=inner,
                    polish=True)


def _eval_points(case, mol, seed):
    """Populations at which the service is asked: positive, near the initial guess."""
    _, init, _, _ = _shells("glisa", mol)
    rng = np.random.default_rng(seed)
    x = init / init.sum() * float(mol.numbers.sum())
    return x * rng.uniform(0.5, 1.5, x.size), x * rng.uniform(0.8, 1.2, x.size)


def _wavefunction(case, mol, seed):
    shells = synthetic.contracted_basis(mol.numbers, mol.coordinates, seed=seed)
    nb = sum(s.nfunc for s in shells)
    nocc = min(nb, max(1, int(mol.numbers.sum()) // 2))
    mats = [synthetic.density_matrix(nb, nocc, seed=seed + 1)]
    if case["spin"]:
        mats.append(0.5 * synthetic.density_matrix(nb, 1, seed=seed + 2) - 0.25 * synthetic.density_matrix(nb, 1, seed=seed + 3))
    return shells, np.array(mats)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "steps":
        return {"case": case, "jobs": [_job(case, m) for m in _molecules(case, seed)]}
    mol = _molecule(case, seed)
    if kind == "call":
        return {"case": case, "mol": mol}
    if kind == "run":
        return {"case": case, "job": _job(case, mol)}
    if kind == "evaluate":
        return {"case": case, "job": _job(case, mol), "x": _eval_points(case, mol, seed)}
    shells, mats = _wavefunction(case, mol, seed)
    plan = DensityPlan(shells, mats, context=_lib.default_context(0))
    if case["host"]:
        return {"case": case, "plan": plan, "points": mol.grid.points}
    pts = torch.as_tensor(mol.grid.points, device="cuda")
    return {"case": case, "plan": plan, "points": pts,
            "out": torch.empty((plan.nmat, pts.shape[0]), dtype=torch.float64, device="cuda")}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "call":
        mol = state["mol"]
        extra = {} if case["scheme"] == "mbis" else {"basis_func": _basis()}
        if case["scheme"] == "gisa":
            extra = {"bs_helper": extra["basis_func"]}
        part = wpart_schemes(case["scheme"])(
            mol.coordinates, mol.numbers, mol.pseudo_numbers, mol.grid, mol.density, logger=LOG,
            grid_type=case["grid_type"], threshold=case["threshold"], precision=case["precision"], **extra)
        part.do_partitioning()
        return {"niter": int(part["niter"]), "charges": part["charges"], "propars": part["propars"],
                "promoldens": part["promoldens"],
                "at_weights": [part[f"at_weights_{i}"] for i in range(mol.natom)]}
    if kind == "run":
        job = state["job"]
        job.reset()
        job.run()
        out = job.results(histories=False)
        return {"niter": int(job.info().niter), **out}
    if kind == "steps":
        jobs = state["jobs"]
        for j in jobs:
            j.reset()
        for _ in range(case["steps"]):
            jobs[0].ctx.step(jobs)
        return [j.results(histories=False) for j in jobs]
    if kind == "evaluate":
        job, (x, y) = state["job"], state["x"]
        f, grad, hess, pop = job.evaluate(x, 2)
        f1, grad1, _, pop1 = job.evaluate(y, 1)
        return {"f": f, "grad": grad, "hess": hess, "pop": pop, "f1": f1, "grad1": grad1, "pop1": pop1}
    if case["host"]:
        return state["plan"].evaluate(state["points"])
    state["plan"].evaluate_device(state["points"], state["out"])
    return state["out"]


def work(case):
    """What a pass cannot do without. Iterations are data dependent: about 8 outer iterations for MBIS to its
    threshold, 20 for gLISA, 40 for GISA, 40 inner iterations per outer one (MBIS), 50 (aLISA)."""
    counts = _counts(case["formula"])
    npa = case["nrad"] * case["nang"]
    total = {"bytes": 0.0, "flops": 0.0}
    for m in range(case.get("molecules", 1)):
        f = max(0.1, 1.0 - m / 6.0) if case.get("molecules", 1) > 1 else 1.0
        c = {z: max(1, round(n * f)) for z, n in counts.items()}
        natom = sum(c.values())
        n = natom * npa
        if case["kind"] == "density":
            nb = sum(k * (5 if z == 1 else 14) for z, k in c.items())
            nmat = 2 if case["spin"] else 1
            total["bytes"] += n * (24.0 + 8.0 * nmat)
            total["flops"] += n * nmat * float(nb) * (nb + 1)
            continue
        total["bytes"] += n * (40.0 + 8.0) + (8.0 * natom * n if case["kind"] == "call" else 0.0)
        shells = {z: int(get_nshell(z)) if case["scheme"] == "mbis" else BASIS_SHELLS[z] for z in c}
        s = float(sum(k * shells[z] for z, k in c.items()))
        if case["scheme"] == "mbis":
            passes = 40.0 if case.get("grid_type") != 1 else 2.0
            total["flops"] += case.get("steps", 8) * passes * n * s * 25.0
        elif case["scheme"] == "lisa":
            total["flops"] += case["steps"] * 50.0 * n * s * 4.0
        elif case["scheme"] == "gisa":
            total["flops"] += 40.0 * n * s * 6.0
        elif case["kind"] == "evaluate":
            total["flops"] += n * (s * s + 8.0 * s)
        else:
            total["flops"] += 20.0 * n * (s * s + 6.0 * s)
    return total


# ---------------------------------------------------------------------------
# the same in 64 bits with torch and numpy alone
# ---------------------------------------------------------------------------

class _Inputs:
    """A molecule on the GPU in 64 bits: grid, density and the distances to every atom."""

    def __init__(self, mol):
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")  # noqa: E731
        self.pts, self.w, self.rho, self.xyz = t(mol.grid.points), t(mol.grid.weights), t(mol.density), t(mol.coordinates)
        self.numbers, self.natom, self.grid = mol.numbers, mol.natom, mol.grid

    def r(self, a):
        return ((self.pts - self.xyz[a]) ** 2).sum(dim=1).sqrt()

    def own(self, a):
        """Atom a's points, its radial nodes and weights 4 pi r^2 w (atom grids)."""
        ag = self.grid.atgrids[a]
        sl = slice(int(self.grid.indices[a]), int(self.grid.indices[a + 1]))
        rr = torch.as_tensor(ag.rgrid.points, device="cuda")
        ww = 4.0 * math.pi * rr * rr * torch.as_tensor(ag.rgrid.weights, device="cuda")
        return sl, torch.as_tensor(ag.sphere_weights, device="cuda"), rr, ww

    def on_atom(self, a, rho_a, local):
        """(radii, weights, AIM density) that atom a's inner solve integrates."""
        if not local:
            return self.r(a), self.w, rho_a
        sl, ws, rr, ww = self.own(a)
        return rr, ww, (ws * rho_a[sl]).reshape(rr.numel(), -1).sum(dim=1)


def _slater(p, r):
    return (p[0::2] * p[1::2] ** 3 / (8.0 * math.pi))[:, None] * torch.exp(-p[1::2][:, None] * r[None])


def _gaussians(alphas, r):
    a = torch.as_tensor(np.asarray(alphas, dtype=np.float64), device="cuda")
    return (a / math.pi).pow(1.5)[:, None] * torch.exp(-a[:, None] * (r * r)[None])


def _qp(P, q, total, x):
    """min x.Px/2 + q.x, x >= 0, sum x = total: primal active set from the feasible x."""
    n = len(q)
    work = x <= 0
    for _ in range(50 * n):
        f = np.flatnonzero(~work)
        K = np.zeros((len(f) + 1, len(f) + 1))
        K[:-1, :-1] = P[np.ix_(f, f)]
        K[:-1, -1] = K[-1, :-1] = 1.0
        y = np.linalg.solve(K, np.concatenate([-q[f], [total]]))
        z = np.zeros(n)
        z[f] = y[:-1]
        d = z - x
        neg = (d < 0) & (z < 0) & ~work
        if neg.any():
            step = np.where(neg, -x / np.where(neg, d, -1.0), np.inf)
            k = int(np.argmin(step))
            x = x + step[k] * d
            x[k], work[k] = 0.0, True
            continue
        x = z
        mu = P @ x + q + y[-1]
        mu[~work] = np.inf
        k = int(np.argmin(mu))
        if not mu[k] < -1e-12 * max(1.0, np.abs(P @ x + q).max()):
            return x
        work[k] = False
    return x


def _exact_iterstock(case, mol, steps=None):
    """MBIS, GISA or aLISA (sc): `steps` outer iterations, or as many as the threshold takes."""
    scheme, local = case["scheme"], case.get("grid_type") == 1
    off, init, _, exps = _shells(scheme, mol)
    m = _Inputs(mol)
    A = m.natom
    thr = case["threshold"]
    inner_thr = min(1e-8, thr) if case["kind"] == "call" else thr
    par = [torch.as_tensor(init[2 * off[a]:2 * off[a + 1]] if scheme == "mbis" else init[off[a]:off[a + 1]],
                           device="cuda").clone() for a in range(A)]
    if scheme != "mbis":
        scale = float(torch.dot(m.w, m.rho)) / float(init.sum())
        par = [p * scale for p in par]
        P = []
        for a in range(A):
            e = exps[off[a]:off[a + 1]]
            P.append(2.0 / math.pi ** 1.5 * (e[:, None] * e[None]) ** 1.5 / (e[:, None] + e[None]) ** 1.5)

    def shells(a, r):  # unit-population functions of a basis scheme
        return _gaussians(exps[off[a]:off[a + 1]], r)

    def pro(a, p, r):
        return _slater(p, r).sum(dim=0) if scheme == "mbis" else (p[:, None] * shells(a, r)).sum(dim=0)

    it = 0
    while True:
        it += 1
        old = [p.clone() for p in par]
        pros = [pro(a, par[a], m.r(a)) for a in range(A)]
        promol = torch.zeros_like(m.rho)
        for v in pros:
            promol = promol + v + 1e-100
        charges = np.zeros(A)
        msd = 0.0
        for a in range(A):
            r, w, rho_a = m.on_atom(a, (pros[a] / promol).clamp(0.0, 1.0) * m.rho, local)
            pop = float(torch.dot(w, rho_a))
            charges[a] = float(mol.pseudo_numbers[a]) - pop
            g = shells(a, r) if scheme != "mbis" else None
            if scheme == "gisa":
                q = -2.0 * (g @ (w * rho_a)).cpu().numpy()
                x0 = np.maximum(par[a].cpu().numpy(), 0.0)
                par[a] = torch.as_tensor(_qp(P[a], q, pop, x0 * (pop / x0.sum())), device="cuda")
            else:
                p, last = par[a], None
                for n in range(2000 if scheme == "mbis" or case["kind"] == "call" else 50):
                    t = _slater(p, r) if scheme == "mbis" else p[:, None] * g
                    y = t.sum(dim=0)
                    ratio = torch.where((rho_a < CUTOFF) | (y < CUTOFF), torch.zeros_like(y), w * rho_a / y)
                    m0 = t @ ratio
                    if scheme == "mbis":
                        p = torch.stack([m0, 3.0 * m0 / (t @ (ratio * r))], dim=1).reshape(-1)
                    else:
                        p = m0
                    if last is not None and math.sqrt(float(torch.dot(w, (last - y) ** 2))) < inner_thr:
                        break
                    last = y
                par[a] = p
            d = pro(a, par[a], r) - pro(a, old[a], r)
            msd += float(torch.dot(w, d * d))
        if steps is not None and it >= steps or steps is None and math.sqrt(msd) < thr:
            break
    out = {"charges": charges, "propars": torch.cat(par).cpu().numpy(), "promoldens": promol.cpu().numpy()}
    if case["kind"] == "call":
        out["at_weights"] = []
        for a in range(A):
            sl = slice(None) if not local else m.own(a)[0]
            out["at_weights"].append((pros[a] / promol).clamp(0.0, 1.0)[sl].cpu().numpy())
    return out


def _glisa_matrix(mol):
    off, init, _, exps = _shells("glisa", mol)
    m = _Inputs(mol)
    return m, off, init, torch.cat([_gaussians(exps[off[a]:off[a + 1]], m.r(a)) for a in range(m.natom)])


def _glisa_terms(m, G, c, nderiv):
    rho0 = G.T @ c
    ok = ~((m.rho < CUTOFF) | (rho0 < CUTOFF))
    inv = torch.where(ok, 1.0 / rho0, torch.zeros_like(rho0))
    wr = torch.where(ok, m.w * m.rho, torch.zeros_like(rho0))
    f = float((wr * torch.log(torch.where(ok, m.rho * inv, torch.ones_like(rho0)))).sum())
    grad = -(G @ (wr * inv)) if nderiv >= 1 else None
    hess = None
    if nderiv == 2:
        hess = torch.zeros((G.shape[0], G.shape[0]), dtype=torch.float64, device="cuda")
        for s in range(0, G.shape[1], 1 << 17):
            x = G[:, s:s + (1 << 17)]
            hess += (x * (wr * inv * inv)[None, s:s + (1 << 17)]) @ x.T
    return f, grad, hess, rho0


def _exact_glisa(case, mol):
    """The optimum of int rho ln(rho / rho0) + sum c over c >= 0: projected Newton, run on to its last digits."""
    m, off, init, G = _glisa_matrix(mol)
    c = torch.as_tensor(init, device="cuda") / float(init.sum()) * float(torch.dot(m.w, m.rho))
    for it in range(60):
        f, grad, H, _ = _glisa_terms(m, G, c, 2)
        dF = 1.0 + grad
        free = (c > 0) | (dF < 0)
        k = torch.nonzero(free)[:, 0]
        L = torch.linalg.cholesky(H[k][:, k])
        d = torch.zeros_like(c)
        d[k] = -torch.cholesky_solve(dF[k][:, None], L)[:, 0]
        F = f + float(c.sum())
        t, done = 1.0, False
        for _ in range(30):
            n = (c + t * d).clamp(min=0.0)
            fn = _glisa_terms(m, G, n, 0)[0] + float(n.sum())
            if fn <= F + 1e-4 * float(torch.dot(dF, n - c)) + 1e-13 * abs(F):
                break
            t *= 0.5
        done = float((n - c).abs().max()) < 1e-13
        c = n
        if done:
            break
    promol = torch.zeros_like(m.rho)
    pros = [G[off[a]:off[a + 1]].T @ c[off[a]:off[a + 1]] for a in range(m.natom)]
    for v in pros:
        promol = promol + v + 1e-100
    aw = [(v / promol).clamp(0.0, 1.0) for v in pros]
    charges = np.array([float(z) - float(torch.dot(m.w, v * m.rho)) for z, v in zip(mol.pseudo_numbers, aw)])
    out = {"charges": charges, "propars": c.cpu().numpy(), "promoldens": promol.cpu().numpy()}
    if case["kind"] == "call":
        own = [slice(None)] * m.natom if case["grid_type"] != 1 else [
            slice(int(mol.grid.indices[a]), int(mol.grid.indices[a + 1])) for a in range(m.natom)]
        out["at_weights"] = [v[o].cpu().numpy() for v, o in zip(aw, own)]
    return out


def _exact_density(case, mol, seed):
    shells, mats = _wavefunction(case, mol, seed)
    D = torch.as_tensor(mats, device="cuda")
    pts = torch.as_tensor(mol.grid.points, device="cuda")
    out = torch.empty((len(mats), pts.shape[0]), dtype=torch.float64, device="cuda")
    for s in range(0, pts.shape[0], 1 << 15):
        rows = []
        for sh in shells:
            d = pts[s:s + (1 << 15)] - torch.as_tensor(sh.center, device="cuda")
            x, y, z = d[:, 0], d[:, 1], d[:, 2]
            r2 = x * x + y * y + z * z
            e = torch.as_tensor(sh.exponents, device="cuda")
            norm = (2.0 * e / math.pi) ** 0.75 * (4.0 * e) ** (0.5 * sh.l) / math.sqrt({0: 1, 1: 1, 2: 3}[sh.l])
            rad = ((torch.as_tensor(sh.coeffs, device="cuda") * norm)[:, None] * torch.exp(-e[:, None] * r2[None])).sum(dim=0)
            s3 = math.sqrt(3.0)
            ang = {0: [torch.ones_like(x)], 1: [x, y, z],
                   2: [z * z - 0.5 * (x * x + y * y), s3 * x * z, s3 * y * z, 0.5 * s3 * (x * x - y * y), s3 * x * y]}[sh.l]
            rows += [rad * v for v in ang]
        phi = torch.stack(rows)
        for k in range(len(mats)):
            out[k, s:s + (1 << 15)] = (phi * (D[k] @ phi)).sum(dim=0)
    return out.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "steps":
        return [_exact_iterstock(case, m, case["steps"]) for m in _molecules(case, seed)]
    mol = _molecule(case, seed)
    if kind == "density":
        return _exact_density(case, mol, seed)
    if kind == "evaluate":
        m, _, _, G = _glisa_matrix(mol)
        out = {}
        for x, tag, nderiv in zip(_eval_points(case, mol, seed), ("", "1"), (2, 1)):
            f, grad, hess, rho0 = _glisa_terms(m, G, torch.as_tensor(x, device="cuda"), nderiv)
            out.update({"f" + tag: f, "grad" + tag: grad.cpu().numpy(), "pop" + tag: float(torch.dot(m.w, rho0))})
            if hess is not None:
                out["hess"] = hess.cpu().numpy()
        return out
    return _exact_glisa(case, mol) if case["scheme"] == "glisa" else _exact_iterstock(case, mol)
