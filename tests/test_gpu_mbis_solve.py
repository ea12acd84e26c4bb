"""The one-launch MBIS inner solve at its tile edges, and the cutoff test of
the FP64 inner kernels at the ends of its range."""

import numpy as np
import pytest

from horton_part_gb300 import _lib, synthetic
from horton_part_gb300.mbis import get_initial_mbis_propars, get_nshell
from horton_part_gb300.molgrid import MolecularGrid, becke_molecular_grid
from oracle import hp_oracle as O

pytestmark = pytest.mark.gpu


def _hydride(z, nrad, nang, npoint):
    coords = np.array([[0.0, 0.0, 0.0], [0.0, 0.3, 2.6]])
    numbers = np.array([z, 1])
    grid = becke_molecular_grid(coords, nrad, nang)
    rho = np.zeros(grid.size)
    for c, n in zip(coords, numbers):
        r = np.linalg.norm(grid.points - c, axis=1)
        rho += O.mbis_proatom(get_initial_mbis_propars(n), r) * (1.0 + 0.05 * np.sin(r))
    assert grid.size >= npoint
    keep = np.sort(np.random.default_rng(7).permutation(grid.size)[:npoint])
    return coords, numbers, MolecularGrid(grid.points[keep], grid.weights[keep]), rho[keep]


def _job(ctx, coords, numbers, grid, rho, **kw):
    nsh = [int(get_nshell(z)) for z in numbers]
    args = dict(grid_type=3, threshold=1e-14, inner_threshold=1e-8, inner_maxiter=2000, maxiter=2)
    args.update(kw)
    return _lib.Job(ctx, "mbis", coords, numbers.astype(float), grid.points, grid.weights, rho,
                    np.concatenate([[0], np.cumsum(nsh)]).astype(np.int32),
                    np.concatenate([get_initial_mbis_propars(z) for z in numbers]), **args)


# 256-point tiles up to 2 x 152 blocks of two atoms (38912 points), 512-point
# tiles from there on, two tiles a block and more than 256 tiles at 140000
@pytest.mark.parametrize("npoint", [1, 257, 38912, 38913, 140000])
def test_same_bits_as_a_launch_per_iteration(npoint, gpu_context):
    small = _hydride(8, 240, 302, npoint)
    mol = synthetic.chain_molecule({6: 14, 1: 18}, 60, 194, seed=9)
    results = []
    for others in (False, True):
        jobs = [_job(gpu_context, *small)]
        if others:  # more blocks than are resident: a launch per inner iteration
            jobs.append(_job(gpu_context, mol.coordinates, mol.numbers, mol.grid, mol.density))
        for _ in range(2):
            gpu_context.step(jobs)
        results.append((jobs[0].results(at_weights=True), jobs[0].info().inner_iterations))
        for j in jobs:
            j.close()
    assert results[0][1] == results[1][1]
    for key in results[0][0]:
        np.testing.assert_array_equal(results[0][0][key], results[1][0][key])


@pytest.mark.parametrize("cutoff", [-1.0, 0.0, 1e-3])
def test_density_cutoff(cutoff, gpu_context):
    coords, numbers, grid, rho = _hydride(8, 30, 50, 2900)
    near = rho > 1e-60  # without a cutoff the quotients of underflowing pro-atoms are 0 / 0
    grid, rho = MolecularGrid(grid.points[near], grid.weights[near]), rho[near]
    job = _job(gpu_context, coords, numbers, grid, rho, density_cutoff=cutoff)
    job.run()
    res = job.results(at_weights=True)
    job.close()
    ref = O.mbis(coords, numbers, numbers.astype(float), grid.points, grid.weights, rho, threshold=1e-14,
                 inner_threshold=1e-8, maxiter=2, density_cutoff=cutoff)
    # the parity bounds of the FP64 path: 1e-8 e and 1e-7 relative parameters
    np.testing.assert_allclose(res["charges"], ref["charges"], rtol=0, atol=1e-8)
    np.testing.assert_allclose(res["propars"], ref["propars"], rtol=1e-7)
