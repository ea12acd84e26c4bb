"""FP64 MBIS kernels: every shell count, ragged grids, and jobs with and
without the stored distances and pro-atoms (the same bits)."""

import numpy as np
import pytest

from horton_part_gb300 import _lib, synthetic
from horton_part_gb300.mbis import get_initial_mbis_propars, get_nshell
from horton_part_gb300.molgrid import MolecularGrid, becke_molecular_grid
from oracle import hp_oracle as O

pytestmark = pytest.mark.gpu


def _pair(z, npoint):
    """An element and a hydrogen: Slater densities of the initial parameters, the grid cut to npoint points."""
    coords = np.array([[0.0, 0.0, 0.0], [0.0, 0.3, 2.6]])
    numbers = np.array([z, 1])
    grid = becke_molecular_grid(coords, 24, 50)
    rho = np.zeros(grid.size)
    for c, n in zip(coords, numbers):
        r = np.linalg.norm(grid.points - c, axis=1)
        rho += O.mbis_proatom(get_initial_mbis_propars(n), r) * (1.0 + 0.05 * np.sin(r))
    keep = np.sort(np.random.default_rng(3).permutation(grid.size)[:npoint])
    return coords, numbers, MolecularGrid(grid.points[keep], grid.weights[keep]), rho[keep]


def _job(ctx, coords, numbers, grid, rho, maxiter, threshold=1e-12):
    nsh = [int(get_nshell(z)) for z in numbers]
    return _lib.Job(ctx, "mbis", coords, numbers.astype(float), grid.points, grid.weights, rho,
                    np.concatenate([[0], np.cumsum(nsh)]).astype(np.int32),
                    np.concatenate([get_initial_mbis_propars(z) for z in numbers]), grid_type=3,
                    threshold=threshold, inner_threshold=1e-8, inner_maxiter=2000, maxiter=maxiter)


# one element per shell count 1..7; points below, at and past tile edges (512 points a tile)
@pytest.mark.parametrize("z,npoint", [(1, 1), (6, 511), (14, 512), (30, 513), (50, 1025), (80, 2047), (92, 2400)])
def test_shell_counts_and_ragged_grids(z, npoint, gpu_context):
    coords, numbers, grid, rho = _pair(z, npoint)
    job = _job(gpu_context, coords, numbers, grid, rho, maxiter=2)
    job.run()
    res = job.results(at_weights=True)
    ref = O.mbis(coords, numbers, numbers.astype(float), grid.points, grid.weights, rho, threshold=1e-12,
                 inner_threshold=1e-8, maxiter=2)
    job.close()
    # the parity bounds of the FP64 path: 1e-8 e and 1e-7 relative parameters
    np.testing.assert_allclose(res["charges"], ref["charges"], rtol=0, atol=1e-8)
    np.testing.assert_allclose(res["propars"], ref["propars"], rtol=1e-7)
    np.testing.assert_allclose(res["at_weights"], ref["at_weights"], rtol=0, atol=1e-8)


def test_stored_pairs_are_given_back_and_change_no_bits():
    mol = synthetic.chain_molecule({6: 2, 1: 4, 8: 1}, 30, 50, seed=5)
    args = (mol.coordinates, mol.numbers, mol.grid, mol.density)

    def results(ctx, others):
        jobs = [_job(ctx, *args, maxiter=3) for _ in range(1 + others)]
        jobs[0].run()
        out, used = jobs[0].results(at_weights=True), jobs[0].info().device_bytes
        for j in jobs:
            j.close()
        return out, used

    big = _lib.Context(0)
    stored, kept = results(big, 0)
    big.close()
    # a budget that just holds two jobs without their stored arrays
    extra = 2 * 8 * mol.natom * mol.npoint
    plain = kept - extra
    small = _lib.Context(0, hbm_budget=int(2.05 * plain))
    recomputed, used = results(small, 1)
    assert small.memory()[0] == 0
    small.close()
    assert used < kept
    for key in stored:
        np.testing.assert_array_equal(stored[key], recomputed[key])


@pytest.mark.parametrize("npoint", [513, 2400])
def test_one_launch_solve_has_the_bits_of_the_stepwise_one(npoint, gpu_context):
    """A small job alone takes the cooperative inner solve; beside a large one, a launch per inner iteration."""
    small = _pair(8, npoint)
    mol = synthetic.chain_molecule({6: 6, 1: 8}, 40, 110, seed=9)
    results = []
    for others in (False, True):
        jobs = [_job(gpu_context, *small, maxiter=3, threshold=1e-14)]
        if others:
            jobs.append(_job(gpu_context, mol.coordinates, mol.numbers, mol.grid, mol.density, maxiter=3))
        for _ in range(3):
            gpu_context.step(jobs)
        results.append((jobs[0].results(at_weights=True), jobs[0].info().inner_iterations))
        for j in jobs:
            j.close()
    assert results[0][1] == results[1][1]
    for key in results[0][0]:
        np.testing.assert_array_equal(results[0][0][key], results[1][0][key])
