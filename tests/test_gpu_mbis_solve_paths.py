"""Which kernels an FP64 MBIS step takes, by its launches: the one-launch inner solve with one to four tiles a block,
the same bits as a launch per inner iteration, and its wait that runs out."""

import ctypes

import numpy as np
import pytest

import device_checks
from horton_part_gb300 import _lib, synthetic
from horton_part_gb300.mbis import get_initial_mbis_propars, get_nshell
from horton_part_gb300.molgrid import MolecularGrid, becke_molecular_grid
from oracle import hp_oracle as O

pytestmark = pytest.mark.gpu


def _molecule(natom, npoint):
    """A chain O H H ...: Slater densities of the initial parameters on npoint points of its grid."""
    numbers = np.array([8] + [1] * (natom - 1))
    coords = np.array([[0.0, 0.3 * (a % 2), 1.9 * a] for a in range(natom)])
    nrad = 100
    while natom * nrad * 302 < npoint:
        nrad += 50
    grid = becke_molecular_grid(coords, nrad, 302)
    keep = np.sort(np.random.default_rng(npoint).permutation(grid.size)[:npoint])
    grid = MolecularGrid(grid.points[keep], grid.weights[keep])
    rho = np.zeros(npoint)
    for c, n in zip(coords, numbers):
        r = np.linalg.norm(grid.points - c, axis=1)
        rho += O.mbis_proatom(get_initial_mbis_propars(n), r) * (1.0 + 0.05 * np.sin(r))
    return coords, numbers, grid, rho


def _job(ctx, coords, numbers, grid, rho, **kw):
    args = dict(grid_type=3, threshold=1e-14, inner_threshold=1e-8, inner_maxiter=60, maxiter=10)
    args.update(kw)
    nsh = [int(get_nshell(z)) for z in numbers]
    return _lib.Job(ctx, "mbis", coords, numbers.astype(float), grid.points, grid.weights, rho,
                    np.concatenate([[0], np.cumsum(nsh)]).astype(np.int32),
                    np.concatenate([get_initial_mbis_propars(z) for z in numbers]), **args)


def _step(ctx, jobs):
    """Launches of inner kernels of one step."""
    ctx.profile()
    ctx.step(jobs)
    n = ctx.profile_get("inner")[1]
    ctx.profile(False)
    return n


@pytest.mark.parametrize("tiles", [1, 2, 3, 4])
def test_tiles_per_block(tiles, gpu_context):
    """Five atoms, so many points that a block takes `tiles` tiles; the last block of an atom takes fewer."""
    natom, cap = 5, device_checks.load().dc_solve_capacity()
    ntile = tiles * (cap // natom) - (tiles > 1)
    points = 512  # two points a thread up to 2 x 152 tiles
    assert ntile <= 304 and natom * -(-ntile // tiles) <= cap
    assert tiles == 1 or natom * -(-ntile // (tiles - 1)) > cap
    mol = _molecule(natom, ntile * points - 37)
    large = synthetic.chain_molecule({6: 14, 1: 18}, 60, 194, seed=9)
    results = []
    for others in (False, True):
        jobs = [_job(gpu_context, *mol, maxiter=1)]
        if others:
            jobs.append(_job(gpu_context, large.coordinates, large.numbers, large.grid, large.density))
        n = _step(gpu_context, jobs)
        assert n > 10 if others else n == 1
        results.append((jobs[0].results(at_weights=True), jobs[0].info().inner_iterations))
        for j in jobs:
            j.close()
    assert results[0][1] == results[1][1]
    for key in results[0][0]:
        np.testing.assert_array_equal(results[0][0][key], results[1][0][key])


def test_a_wait_that_runs_out():
    """One poll: some block's packets are not there yet. The step reports it, and a new context works."""
    mol = _molecule(2, 20000)
    ctx = _lib.Context(0)
    job = _job(ctx, *mol)
    assert _step(ctx, [job]) == 1
    want = job.results()["propars"]
    job.close()
    polls = _lib.lib().hp_test_solve_polls
    polls.argtypes = [ctypes.c_void_p, ctypes.c_int32]
    assert polls(ctx.handle, 1) == 0
    job = _job(ctx, *mol)
    ctx.step([job])
    info = job.info()
    assert info.done and info.status == 5  # HP_ERR_TIMEOUT
    job.close()
    job = _job(ctx, *mol)
    with pytest.raises(_lib.HPError) as e:
        job.run()
    assert e.value.code == 5
    ctx.close()
    ctx = _lib.Context(0)
    job = _job(ctx, *mol)
    ctx.step([job])
    np.testing.assert_array_equal(job.results()["propars"], want)
    ctx.close()
