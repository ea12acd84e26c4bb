"""Mixed-precision gLISA jobs with an odd number of shells: the fused passes
lay their shared-memory arrays out by the shell count, and the 16-byte loads
of the per-point values need that layout aligned for every count."""

import numpy as np
import pytest

from horton_part_gb300 import synthetic
from horton_part_gb300.utils import wpart_schemes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,shells", [({6: 1, 1: 2}, 21), ({6: 10, 8: 1, 1: 5}, 129)])
def test_odd_shell_counts_match_fp64(counts, shells, gpu_context):
    mol = synthetic.chain_molecule(counts, 24, 50, seed=17)
    helper = synthetic.geometric_gaussian_basis({1: 6, 6: 9, 8: 9}, 0.05, 300.0)
    assert sum(helper.get_nshell(z) for z in mol.numbers) == shells
    res = {}
    for precision in ("fp64", "mixed"):
        part = wpart_schemes("glisa")(mol.coordinates, mol.numbers, mol.pseudo_numbers, mol.grid,
                                      mol.density, grid_type=3, solver="cvxopt", basis_func=helper,
                                      threshold=1e-8, precision=precision)
        part.do_partitioning()
        res[precision] = part["charges"]
    # the bound of the mixed form against FP64 (float-float sums, the same optimum)
    assert np.abs(res["mixed"] - res["fp64"]).max() < 1e-7
