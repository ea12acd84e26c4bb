"""FP64 kernels over the stored basis matrix: shell counts at the edges of the
Hessian's row groups, ragged grids, tiles on which shells or whole atoms
vanish, and jobs with and without the stored arrays."""

import numpy as np
import pytest

from horton_part_gb300 import _lib, synthetic
from horton_part_gb300.molgrid import MolecularGrid, becke_molecular_grid
from oracle import hp_oracle as O

pytestmark = pytest.mark.gpu


def _mol(numbers, coords, npoint=None, seed=3):
    numbers, coords = np.asarray(numbers), np.asarray(coords, dtype=float)
    grid = becke_molecular_grid(coords, 24, 50)
    rho = synthetic.slater_density(grid.points, coords, numbers, seed)
    if npoint is not None:
        keep = np.sort(np.random.default_rng(seed).permutation(grid.size)[:npoint])
        grid, rho = MolecularGrid(grid.points[keep], grid.weights[keep]), rho[keep]
    return synthetic.Molecule(coords, numbers, grid, rho)


def _far_chain(n):
    """n atoms 9 bohr apart: tight shells and far atoms vanish on most tiles."""
    return [6 if k % 2 == 0 else 1 for k in range(n)], [[9.0 * k, 0.3 * (k % 3), 0.0] for k in range(n)]


def _job(ctx, mol, scheme, shells, solver, amax=300.0, **kw):
    helper = synthetic.geometric_gaussian_basis(shells, 0.1, amax)
    off = np.concatenate([[0], np.cumsum([helper.get_nshell(z) for z in mol.numbers])]).astype(np.int32)
    init = np.concatenate([np.full(helper.get_nshell(z), z / helper.get_nshell(z)) for z in mol.numbers])
    exps = np.concatenate([helper.get_exponent(z) for z in mol.numbers])
    job = _lib.Job(ctx, scheme, mol.coordinates, mol.pseudo_numbers, mol.grid.points, mol.grid.weights,
                   mol.density, off, init, shell_orders=np.full(len(init), 2.0), shell_exponents=exps,
                   solver=solver, grid_type=3, **kw)
    return job, off, init, exps


# shells: one; edges of the 4-row groups, of one and two sets of accumulators (124 and 176 active rows, every
# row active with the small exponents) and of the kernel's 224 rows; beyond it
@pytest.mark.parametrize("natom,per,npoint,amax", [
    (1, 1, 700, 300.0), (1, 5, 17, 300.0), (8, 16, 2401, 300.0), (12, 10, 4000, 300.0), (31, 4, 900, 0.2),
    (25, 5, 801, 0.2), (22, 8, 700, 0.2), (14, 16, 3001, 0.2), (14, 16, 2200, 300.0), (15, 16, 2600, 300.0)])
def test_evaluation_against_numpy(natom, per, npoint, amax, gpu_context):
    numbers, coords = _far_chain(natom)
    mol = _mol(numbers, coords, npoint)
    job, off, init, exps = _job(gpu_context, mol, "glisa", {1: per, 6: per}, "newton", amax=amax, threshold=1e-8)
    x = np.random.default_rng(1).uniform(0.5, 1.5, init.size) * init
    f, grad, hess, pop = job.evaluate(x, 2)
    job.close()
    r = O.radial_distances(mol.grid.points, mol.coordinates)
    G = np.concatenate([O.basis_functions(np.full(per, 2.0), exps[off[a]:off[a + 1]], r[a])
                        for a in range(natom)])
    w, rho = mol.grid.weights, mol.density
    rho0 = G.T @ x
    ok = (rho >= 1e-15) & (rho0 >= 1e-15)
    inv = np.where(ok, 1.0 / np.where(ok, rho0, 1.0), 0.0)
    # sums of a few thousand terms of one sign: 1e-12 of the largest entry of a row leaves two digits over their rounding
    assert abs(f - np.sum((w * rho * np.log(np.where(ok, rho * inv, 1.0)))[ok])) < 1e-11 * max(1.0, abs(f))
    assert abs(pop - w @ rho0) < 1e-12 * abs(pop)
    want = -(G @ (w * rho * inv))
    np.testing.assert_allclose(grad, want, rtol=1e-12, atol=1e-12 * np.abs(want).max())
    want = (G * (w * rho * inv * inv)) @ G.T
    scale = np.sqrt(np.outer(np.diag(want), np.diag(want)))
    assert np.all(np.abs(hess - want) <= 1e-12 * scale + 1e-300)
    np.testing.assert_array_equal(hess, hess.T)


@pytest.mark.parametrize("scheme,solver", [("lisa", "sc"), ("gisa", "quadprog")])
@pytest.mark.parametrize("natom,per,npoint", [(1, 1, 300), (3, 9, 513), (5, 16, 2047)])
def test_outer_iterations_against_the_oracle(scheme, solver, natom, per, npoint, gpu_context):
    numbers, coords = _far_chain(natom)
    mol = _mol(numbers, coords, npoint)
    job, off, init, exps = _job(gpu_context, mol, scheme, {1: per, 6: per}, solver, threshold=1e-12,
                                inner_threshold=1e-8, maxiter=2, inner_maxiter=100000)
    job.run()
    res = job.results(at_weights=True)
    job.close()
    split = [slice(off[a], off[a + 1]) for a in range(natom)]
    ref = O.basis_scheme(scheme, mol.coordinates, mol.numbers, mol.pseudo_numbers, mol.grid.points,
                         mol.grid.weights, mol.density, [np.full(per, 2.0)] * natom,
                         [exps[s] for s in split], [init[s] for s in split], threshold=1e-12,
                         inner_threshold=1e-8, maxiter=2)
    # the parity bounds of the FP64 path: 1e-8 e, populations to 1e-7 of the atom's
    np.testing.assert_allclose(res["charges"], ref["charges"], rtol=0, atol=1e-8)
    np.testing.assert_allclose(res["propars"], ref["propars"], rtol=0, atol=1e-7 * np.max(numbers))
    np.testing.assert_allclose(res["at_weights"], ref["at_weights"], rtol=0, atol=1e-7)


def test_alisa_without_the_stored_pro_atoms_has_the_same_bits(gpu_context):
    mol = _mol(*_far_chain(4))
    opts = dict(threshold=1e-10, inner_threshold=1e-8, maxiter=2, inner_maxiter=200)
    pair = 8 * mol.natom * mol.npoint
    results, sizes = [], []
    # the second budget holds G and the job, and less than twice the pro-atoms beside them: they are not stored
    for budget in (0, None):
        if budget is None:
            budget = int(sizes[0] + 0.5 * pair)
        ctx = _lib.Context(0, hbm_budget=budget)
        job = _job(ctx, mol, "lisa", {1: 2, 6: 2}, "sc", **opts)[0]
        job.run()
        results.append(job.results(at_weights=True))
        sizes.append(job.info().device_bytes)
        job.close()
        ctx.close()
    assert sizes[0] - sizes[1] >= pair
    for key in results[0]:
        np.testing.assert_array_equal(results[0][key], results[1][key])
