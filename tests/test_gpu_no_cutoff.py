"""FP64 basis schemes without a density cutoff: where every shell underflows and the density does not, the quotient is
rho / 0, and 0 times it is NaN in every row, as in the reference, also on tiles where no shell is nonzero."""

import numpy as np
import pytest

from horton_part_gb300 import synthetic
from horton_part_gb300.molgrid import MolecularGrid
from oracle import hp_oracle as O
from test_gpu_fp64_basis import _far_chain, _job, _mol

pytestmark = pytest.mark.gpu


def _with_far_points(natom):
    """Points 200 bohr away, more than two tiles of them, behind those of a chain."""
    mol = _mol(*_far_chain(natom), 1200)
    far = np.random.default_rng(4).uniform(200.0, 210.0, (1300, 3))
    grid = MolecularGrid(np.concatenate([mol.grid.points, far]), np.concatenate([mol.grid.weights, np.full(1300, 1e-3)]))
    return synthetic.Molecule(mol.coordinates, mol.numbers, grid, np.concatenate([mol.density, np.full(1300, 1e-9)]))


@pytest.mark.parametrize("cutoff", [1e-15, 0.0, -1.0])
def test_evaluation(cutoff, gpu_context):
    mol = _with_far_points(3)
    job, off, init, exps = _job(gpu_context, mol, "glisa", {1: 5, 6: 5}, "newton", threshold=1e-8, density_cutoff=cutoff)
    _, grad, hess, _ = job.evaluate(init, 2)
    job.close()
    G = np.concatenate([O.basis_functions(np.full(5, 2.0), exps[off[a]:off[a + 1]], r)
                        for a, r in enumerate(O.radial_distances(mol.grid.points, mol.coordinates))])
    rho, rho0 = mol.density, G.T @ init
    with np.errstate(all="ignore"):
        sick = (rho < cutoff) | (rho0 < cutoff)
        ratio = np.where(sick, 0.0, mol.grid.weights * rho / rho0)
        want = -(G * ratio).sum(axis=1)
    assert np.isnan(want).all() == (cutoff <= 0.0)
    np.testing.assert_array_equal(np.isnan(grad), np.isnan(want))
    assert np.isnan(hess).all() == (cutoff <= 0.0) and np.isfinite(hess).all() == (cutoff > 0.0)


@pytest.mark.parametrize("cutoff", [1e-15, 0.0])
def test_alisa(cutoff, gpu_context):
    mol = _with_far_points(1)
    job, off, init, exps = _job(gpu_context, mol, "lisa", {1: 5, 6: 5}, "sc", threshold=1e-8, inner_threshold=1e-8,
                                maxiter=1, inner_maxiter=2, density_cutoff=cutoff)
    gpu_context.step([job])
    got = job.results()["propars"]
    job.close()
    assert np.isnan(got).all() == (cutoff <= 0.0) and np.isfinite(got).all() == (cutoff > 0.0)
