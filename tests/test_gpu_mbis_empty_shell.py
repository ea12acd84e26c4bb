"""An MBIS shell of population zero: its exponent is 0 / 0 after an iteration, as in the reference, in every kernel that
forms the update, and the other shells are as they would be without it."""

import numpy as np
import pytest

from horton_part_gb300 import _lib, synthetic
from horton_part_gb300.mbis import get_initial_mbis_propars, get_nshell
from horton_part_gb300.molgrid import AtomGrid, MolecularGrid, atom_grid_arrays, radial_becke_gauss_chebyshev
from oracle import hp_oracle as O

pytestmark = pytest.mark.gpu


def _propars(numbers):
    init = np.concatenate([get_initial_mbis_propars(z) for z in numbers])
    z = int(np.flatnonzero(np.asarray(numbers) > 2)[0])
    empty = 2 * sum(int(get_nshell(n)) for n in numbers[:z])  # the first heavy atom's core shell
    init[empty] = 0.0
    return init, empty


def _job(ctx, mol, precision, local=None):
    init, _ = _propars(mol.numbers)
    off = np.concatenate([[0], np.cumsum([int(get_nshell(z)) for z in mol.numbers])]).astype(np.int32)
    return _lib.Job(ctx, "mbis", mol.coordinates, mol.numbers.astype(float), mol.grid.points, mol.grid.weights,
                    mol.density, off, init, grid_type=1 if local else 3, threshold=1e-8, inner_threshold=1e-8,
                    inner_maxiter=1, maxiter=10, precision=precision, local=local)


def _one_inner_iteration(mol):
    """Parameters after one outer iteration of one inner iteration each."""
    init, empty = _propars(mol.numbers)
    ends = np.concatenate([[0], np.cumsum([2 * int(get_nshell(z)) for z in mol.numbers])])
    rs = O.radial_distances(mol.grid.points, mol.coordinates)
    pros = [O.mbis_proatom(init[ends[a]:ends[a + 1]], rs[a]) for a in range(mol.natom)]
    _, at_weights = O.stockholder_weights(pros)
    new = [O.opt_mbis_propars(at_weights[a] * mol.density, init[ends[a]:ends[a + 1]].copy(), mol.grid.weights, rs[a],
                              1e-8, maxiter=1)[0] for a in range(mol.natom)]
    return np.concatenate(new), empty


# the small molecule alone takes the one-launch solve, the large one a launch per inner iteration
@pytest.mark.parametrize("precision", ["fp64", "ff", "mixed"])
@pytest.mark.parametrize("counts,nrad,nang", [({8: 1, 1: 2}, 20, 50), ({6: 14, 1: 18}, 40, 110)])
def test_exponent_of_an_empty_shell(counts, nrad, nang, precision, gpu_context):
    mol = synthetic.chain_molecule(counts, nrad, nang, seed=9)
    job = _job(gpu_context, mol, precision)
    gpu_context.step([job])
    got = job.results()["propars"]
    job.close()
    with np.errstate(invalid="ignore"):
        want, empty = _one_inner_iteration(mol)
    assert np.flatnonzero(np.isnan(want)).tolist() == [empty + 1] and want[empty] == 0.0
    # the parity bounds: 1e-7 relative parameters (FP64, float-float), 1e-4 for FP32 evaluation
    np.testing.assert_allclose(got, want, rtol=1e-4 if precision == "mixed" else 1e-7)


def test_exponent_of_an_empty_shell_on_atom_grids(gpu_context):
    mol = synthetic.water(30, 50, seed=2)
    r, wr = radial_becke_gauss_chebyshev(30)
    grid = MolecularGrid(mol.grid.points, mol.grid.weights, indices=mol.grid.indices,
                         atgrids=[AtomGrid(r, wr, 50) for _ in range(mol.natom)])
    job = _job(gpu_context, mol, "fp64", local=atom_grid_arrays(grid))
    gpu_context.step([job])
    got = job.results()["propars"]
    job.close()
    _, empty = _propars(mol.numbers)
    assert np.flatnonzero(np.isnan(got)).tolist() == [empty + 1] and got[empty] == 0.0
