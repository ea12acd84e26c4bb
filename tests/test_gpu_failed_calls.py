"""CUDA calls that fail (a fake in front of libcudart, fake_cudart.c): what the library makes of them."""

import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

SETUP = """
    import ctypes, sys
    sys.path[:0] = [{root!r}, {here!r}]
    import numpy as np
    from horton_part_gb300 import _lib, synthetic
    from horton_part_gb300.density import DensityPlan
    from test_gpu_memory import _job
    def fail(call, n, code=None):
        ctypes.c_int.in_dll(ctypes.CDLL(None), "fail_" + call).value = n
        if code is not None:
            ctypes.c_int.in_dll(ctypes.CDLL(None), "code_" + call).value = code
    ctx = _lib.Context(0)
"""


def _run(tmp_path, code):
    fake = str(tmp_path / "libfake.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", os.path.join(HERE, "fake_cudart.c"), "-o", fake, "-ldl"], check=True)
    setup = SETUP.format(root=os.path.dirname(HERE), here=HERE)
    res = subprocess.run([sys.executable, "-c", textwrap.dedent(setup) + textwrap.dedent(code)], capture_output=True,
                         text=True, timeout=300, env=dict(os.environ, LD_PRELOAD=fake))
    assert res.returncode == 0, res.stdout + res.stderr


def test_inner_solve_that_is_not_launched(tmp_path, gpu_context):
    """The step fails at once: no iteration is counted, and a later step goes on from the same parameters."""
    _run(tmp_path, """
        want = _job(ctx, 4000, maxiter=2)
        ctx.step([want])
        job = _job(ctx, 4000, maxiter=2)
        ctx.step([job])
        before = job.results()
        fail("cudaLaunchCooperativeKernel", 1, 701)  # cudaErrorLaunchOutOfResources
        try:
            ctx.step([job])
        except _lib.HPError as e:
            assert "inner solve" in str(e), e
        else:
            raise SystemExit("no error")
        after = job.results()
        assert job.info().niter == 1 and not job.info().done
        for key in set(before) - {"promoldens"}:  # (the begun iteration has formed its promolecule)
            np.testing.assert_array_equal(before[key], after[key])
        ctx.step([job]), ctx.step([want])
        for key, v in want.results(at_weights=True).items():
            np.testing.assert_array_equal(v, job.results(at_weights=True)[key])
    """)


def test_density_plan_whose_first_allocation_fails(tmp_path, gpu_context):
    """The context gives back what it can and asks again; only a second failure is reported."""
    _run(tmp_path, """
        mol = synthetic.water(10, 50, seed=1)
        shells = synthetic.contracted_basis(mol.numbers, mol.coordinates, seed=1)
        D = synthetic.density_matrix(sum(s.nfunc for s in shells), 5, seed=2)
        points = np.repeat(mol.grid.points, 30, axis=0)  # past a megabyte: device scratch
        plan = DensityPlan(shells, D, context=ctx)
        want = plan.evaluate(points)
        plan.close()
        job = _job(ctx, 4000)
        full = job.info().device_bytes
        fail("cudaMalloc", 1)
        plan = DensityPlan(shells, D, context=ctx)
        assert job.info().device_bytes < full
        fail("cudaMalloc", 1)
        np.testing.assert_array_equal(plan.evaluate(points), want)
        plan.close()
        fail("cudaMalloc", 2)
        try:
            DensityPlan(shells, D, context=ctx)
        except MemoryError:
            pass
        else:
            raise SystemExit("no error")
        fail("cudaMalloc", 0)
        plan = DensityPlan(shells, D, context=ctx)
        np.testing.assert_array_equal(plan.evaluate(points), want)
        plan.close()
        ctx.step([job])
    """)


@pytest.mark.parametrize("code", [720, 801])  # cudaErrorCooperativeLaunchTooLarge, cudaErrorNotSupported
def test_inner_solve_that_does_not_fit(code, tmp_path, gpu_context):
    """A launch per iteration instead, with the same bits."""
    _run(tmp_path, f"""
        results, launches = [], []
        for k in (0, 1):
            job = _job(ctx, 4000, maxiter=1)
            fail("cudaLaunchCooperativeKernel", k, {code})
            ctx.profile()
            ctx.step([job])
            launches.append(ctx.profile_get("inner")[1])
            results.append((job.results(at_weights=True), job.info().inner_iterations))
        assert launches[0] == 1 and launches[1] > 2, launches
        assert results[0][1] == results[1][1]
        for key in results[0][0]:
            np.testing.assert_array_equal(results[0][0][key], results[1][0][key])
    """)
