"""The device memory of a context: what FP64 jobs only keep to save recomputation (distances, pro-atoms, packets of the
inner solve) is given back when it makes room for something else, and stays where it does not."""

import numpy as np
import pytest

from horton_part_gb300 import _lib
from horton_part_gb300.mbis import get_initial_mbis_propars
from oracle import hp_oracle as O

pytestmark = pytest.mark.gpu

NUMBERS = np.array([1, 1])


def _job(ctx, npoint, maxiter=3):
    """Two hydrogens on `npoint` random points: the memory counts here, not the integral's accuracy."""
    rng = np.random.default_rng(npoint)
    coords = np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 1.5]])
    points = rng.uniform(-3.0, 3.0, (npoint, 3))
    rho = sum(O.mbis_proatom(get_initial_mbis_propars(1), np.linalg.norm(points - c, axis=1)) for c in coords)
    return _lib.Job(ctx, "mbis", coords, NUMBERS.astype(float), points, np.full(npoint, 216.0 / npoint), rho,
                    np.arange(3, dtype=np.int32), np.concatenate([get_initial_mbis_propars(1)] * 2), grid_type=3,
                    threshold=1e-12, inner_threshold=1e-8, inner_maxiter=50, maxiter=maxiter)


def _plain_job(ctx, scheme, natom, npoint, per, precision="fp64", solver="default"):
    rng = np.random.default_rng(1)
    coords = np.stack([np.zeros(natom), np.zeros(natom), 2.0 * np.arange(natom)], axis=1)
    points, n = rng.uniform(-3, 3, (npoint, 3)), per * natom
    extra = {} if scheme == "mbis" else dict(shell_orders=np.full(n, 2.0),
                                             shell_exponents=np.tile(np.geomspace(0.1, 10, per), natom))
    return _lib.Job(ctx, scheme, coords, np.ones(natom), points, np.full(npoint, 1.0 / npoint),
                    np.exp(-np.linalg.norm(points, axis=1)), np.arange(natom + 1, dtype=np.int32) * per,
                    np.tile([1.0, 2.0], n) if scheme == "mbis" else np.full(n, 1.0 / per), solver=solver,
                    precision=precision, grid_type=3, maxiter=3, threshold=1e-8, **extra)


@pytest.fixture(scope="module")
def sizes(gpu_context):
    """(device bytes of the 4000-point job with its kept arrays, without them)"""
    ctx = _lib.Context(0)
    job = _job(ctx, 4000)
    full = job.info().device_bytes
    ctx.close()
    ctx = _lib.Context(0, hbm_budget=full)
    job = _job(ctx, 4000)
    plain = job.info().device_bytes
    ctx.close()
    assert full - plain >= 2 * 8 * 2 * 4000  # the distances and the pro-atoms of every pair
    return full, plain


def test_a_refused_job_takes_nothing_from_a_live_one(sizes):
    full, plain = sizes
    budget = 32 * full
    ctx = _lib.Context(0, hbm_budget=budget)
    job = _job(ctx, 4000)
    assert job.info().device_bytes == full
    with pytest.raises(MemoryError):
        _job(ctx, 4000 * 64)  # more than the whole budget
    assert job.info().device_bytes == full
    ctx.close()


def _water_plan(ctx, nmat=1):
    from horton_part_gb300 import synthetic
    from horton_part_gb300.density import DensityPlan

    mol = synthetic.water(10, 50, seed=1)
    shells = synthetic.contracted_basis(mol.numbers, mol.coordinates, seed=1)
    nb = sum(s.nfunc for s in shells)
    mats = np.array([synthetic.density_matrix(nb, 5, seed=2)] * nmat)
    return DensityPlan(shells, mats, context=ctx), mol.grid.points


def test_a_small_host_density_call_needs_no_budget(sizes):
    full, plain = sizes
    ctx = _lib.Context(0)
    plan, points = _water_plan(ctx)
    plan_bytes = ctx.memory()[0]
    points = np.repeat(points, 20, axis=0)  # a little below a megabyte with the density
    want = plan.evaluate(points)
    plan.close()
    ctx.close()
    budget = 32 * full
    ctx = _lib.Context(0, hbm_budget=budget)
    plan, _ = _water_plan(ctx)
    jobs = [_job(ctx, 4000)]
    while budget - plan_bytes - sum(j.info().device_bytes for j in jobs) >= full:
        jobs.append(_job(ctx, 4000))
    held = [j.info().device_bytes for j in jobs]
    assert held[0] == full and budget - plan_bytes - sum(held) < 8 * 4 * len(points) < 1 << 20
    np.testing.assert_array_equal(plan.evaluate(points), want)
    assert [j.info().device_bytes for j in jobs] == held
    with pytest.raises(MemoryError):  # until nothing fits any more, not even by giving back
        while True:
            jobs.append(_job(ctx, 4000))
    np.testing.assert_array_equal(plan.evaluate(points), want)
    plan.close()
    ctx.close()


def test_memory_counts_what_only_closing_a_job_frees(sizes):
    full, plain = sizes
    ctx = _lib.Context(0, hbm_budget=32 * full)
    jobs = [_job(ctx, 4000)]
    assert jobs[0].info().device_bytes == full
    counted, budget = ctx.memory()
    assert 0.9 * plain < counted <= plain and budget == 32 * full
    # a job fits as long as used + its bytes stay within the budget, and no longer
    while ctx.memory()[0] + counted <= budget:
        jobs.append(_job(ctx, 4000))
        assert ctx.memory()[0] == counted * len(jobs)
    with pytest.raises(MemoryError):
        _job(ctx, 4000)
    for j in jobs:
        j.close()
    assert ctx.memory()[0] == 0
    ctx.close()


def test_kept_arrays_take_a_16th_of_the_budget_at_most(sizes):
    full, plain = sizes
    budget = 40 * full
    ctx = _lib.Context(0, hbm_budget=budget)
    jobs = [_job(ctx, 4000) for _ in range(40)]
    kept = [j.info().device_bytes - plain for j in jobs]
    assert set(kept) == {0, full - plain}
    assert kept[0] > 0 and sum(kept) <= budget // 16 < sum(kept) + full - plain
    ctx.close()


def test_given_back_arrays_return_when_there_is_room(sizes):
    """A job that had to give its arrays back has them again, and the one-launch inner solve, once the job that took
    the room is gone: the same launches and the same bits as a job that never lost them."""
    full, plain = sizes
    ctx = _lib.Context(0, hbm_budget=32 * full)
    runs = []
    for crowded in (False, True):
        job = _job(ctx, 4000)
        ctx.step([job])
        if crowded:
            others = []
            with pytest.raises(MemoryError):
                while True:
                    others.append(_job(ctx, 4000))
            assert job.info().device_bytes == plain
            ctx.step([job])  # without them, a launch per inner iteration
            for j in others:
                j.close()
        else:
            ctx.step([job])
        ctx.profile()
        ctx.step([job])
        runs.append((ctx.profile_get("inner")[1], job.info().device_bytes, job.results(at_weights=True)))
        ctx.profile(False)
        job.close()
    assert runs[0][:2] == runs[1][:2] == (1, full)
    for key in runs[0][2]:
        np.testing.assert_array_equal(runs[0][2][key], runs[1][2][key])
    ctx.close()


@pytest.mark.parametrize("when", ["create", "evaluate"])
def test_density_plans_take_the_room_that_jobs_give_back(when, sizes):
    full, plain = sizes
    ctx = _lib.Context(0)
    nmat = 40 if when == "create" else 1  # a plan larger than the small jobs below
    plan, points = _water_plan(ctx, nmat)
    plan_bytes = ctx.memory()[0]
    points = np.repeat(points, 30, axis=0)  # past a megabyte: device scratch
    want, want_few = plan.evaluate(points), plan.evaluate(points[:500])
    scratch = ctx.memory()[0] - plan_bytes
    assert scratch == 8 * (3 + nmat) * len(points) > 1 << 20
    plan.close()
    ctx.close()
    need = plan_bytes if when == "create" else scratch
    budget = 40 * full
    ctx = _lib.Context(0, hbm_budget=budget)
    if when == "evaluate":
        plan, _ = _water_plan(ctx, nmat)
    job = _job(ctx, 4000)
    ctx.step([job])
    jobs = []  # jobs that keep nothing, until what is left is below what the plan needs with the kept arrays, not without
    while budget - ctx.memory()[0] - (full - plain) >= need:
        jobs.append(_plain_job(ctx, "lisa", 1, 64, 2, "fp64", "newton"))
    assert job.info().device_bytes == full and budget - ctx.memory()[0] >= need
    if when == "create":
        plan, _ = _water_plan(ctx, nmat)
        np.testing.assert_array_equal(plan.evaluate(points[:500]), want_few)
    else:
        np.testing.assert_array_equal(plan.evaluate(points), want)
    assert job.info().device_bytes == plain
    ctx.step([job])  # and the job goes on
    plan.close()
    ctx.close()


# the bytes of the arrays that hold a job's inputs, parameters, pairs and partial sums (512-point tiles)
@pytest.mark.parametrize("spec,nbytes", [
    (("mbis", 2, 4000, 1), 298240), (("mbis", 3, 120000, 2), 9741568), (("mbis", 2, 4000, 1, "ff"), 538880),
    (("gisa", 3, 5000, 6), 1134592), (("lisa", 3, 5000, 6, "fp64", "sc"), 1134080),
    (("lisa", 3, 5000, 6, "fp64", "newton"), 1136384), (("glisa", 3, 5000, 6, "fp64", "newton"), 1316352)])
def test_a_budget_that_holds_a_job_is_enough(spec, nbytes, gpu_context):
    """GISA and aLISA store the basis matrix where it takes at most half of the budget: 2 x 720,000 bytes here."""
    budget = max(nbytes, 2 * 720000 if spec[0] in ("gisa", "lisa") else 0)
    ctx = _lib.Context(0, hbm_budget=budget)
    job = _plain_job(ctx, *spec)
    ctx.step([job])
    assert ctx.memory()[0] == nbytes
    job.close()
    assert ctx.memory()[0] == 0
    ctx.close()
    if budget == nbytes:
        ctx = _lib.Context(0, hbm_budget=nbytes - 1)
        with pytest.raises(MemoryError):
            _plain_job(ctx, *spec)
        ctx.close()
