"""A batch of FP64 basis-scheme jobs of which some store the basis matrix and some have no room for it: each job has the
bits it has alone."""

import numpy as np
import pytest

from horton_part_gb300 import _lib
from test_gpu_fp64_basis import _far_chain, _job, _mol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
@pytest.mark.parametrize("scheme,solver", [("lisa", "sc"), ("gisa", "quadprog")])
def test_same_bits_as_alone(scheme, solver, order, gpu_context):
    mols = [_mol(*_far_chain(3), 1537), _mol(*_far_chain(4), 2200)]
    per = [9, 16]
    G = [8 * mol.natom * n * mol.npoint for mol, n in zip(mols, per)]
    opts = dict(threshold=1e-14, inner_threshold=1e-8, maxiter=3, inner_maxiter=300)

    def job(ctx, k):
        return _job(ctx, mols[k], scheme, {1: per[k], 6: per[k]}, solver, **opts)[0]

    def finish(jobs, ctx):
        for _ in range(3):
            ctx.step(jobs)
        return [j.results(at_weights=True) for j in jobs]

    big = _lib.Context(0)
    stored = job(big, 0)
    want = finish([stored], big)
    # a budget whose half is less than the matrix
    small = _lib.Context(0, hbm_budget=int(1.3 * G[1]))
    want += finish([job(small, 1)], small)
    both = _lib.Context(0, hbm_budget=stored.info().device_bytes + int(1.3 * G[1]))
    jobs = [job(both, 0), job(both, 1)]
    assert jobs[0].info().device_bytes > G[0] and jobs[1].info().device_bytes < G[1]
    got = finish([jobs[k] for k in order], both)
    for k, res in zip(order, got):
        for key in res:
            np.testing.assert_array_equal(res[key], want[k][key])
    for ctx in (big, small, both):
        ctx.close()
