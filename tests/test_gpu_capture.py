"""Contexts and jobs beside another stream that is being captured into a graph."""

import numpy as np
import pytest

import device_checks
from horton_part_gb300 import _lib
from test_gpu_fp64_basis import _far_chain, _job, _mol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme,solver", [("glisa", "newton"), ("gisa", "quadprog")])
def test_steps_while_another_stream_is_captured(scheme, solver, gpu_context):
    mol = _mol(*_far_chain(3), 1537)

    def run(capture):
        if capture:
            assert device_checks.load().dc_capture_begin() == 0
        try:
            ctx = _lib.Context(0)
            job = _job(ctx, mol, scheme, {1: 6, 6: 6}, solver, threshold=1e-14, maxiter=2)[0]
            ctx.step([job])
            ctx.step([job])
        finally:
            ended = device_checks.load().dc_capture_end() if capture else 0
        res = job.results()
        job.close()
        ctx.close()
        assert ended == 0  # the capture is whole
        return res

    want, got = run(False), run(True)
    for key in want:
        np.testing.assert_array_equal(got[key], want[key])
