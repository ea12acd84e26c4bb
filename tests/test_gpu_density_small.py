"""The density of small point sets: blocks of half a tile, and host arrays of
any size give the bits of device arrays."""

import numpy as np
import pytest

from horton_part_gb300 import synthetic
from horton_part_gb300.density import DensityPlan
from oracle import hp_density as H

pytestmark = pytest.mark.gpu


def _water():
    xyz = np.array([[0.0, 0.0, 0.2], [0.0, 1.4, -0.9], [0.0, -1.4, -0.9]])
    shells = synthetic.contracted_basis(np.array([8, 1, 1]), xyz)
    nb = sum(s.nfunc for s in shells)
    return shells, np.array([synthetic.density_matrix(nb, 5), 0.5 * synthetic.density_matrix(nb, 1, seed=3)])


# a block's 32 and a tile's 64 points; half tiles up to 76 tiles (4864 points),
# one block of 1024 threads a tile up to 152 (9728)
@pytest.mark.parametrize("npoint", [1, 31, 32, 33, 64, 65, 4864, 4865, 9728, 9729])
def test_against_the_oracle(npoint, gpu_context):
    shells, mats = _water()
    pts = np.random.default_rng(npoint).normal(scale=2.0, size=(npoint, 3))
    plan = DensityPlan(shells, mats, context=gpu_context)
    got = plan.evaluate(pts)
    stats = plan.stats()
    plan.close()
    for g, D in zip(got, mats):
        ref = H.density(D, shells, pts)
        assert np.abs(g - ref).max() <= 1e-13 * np.abs(ref).max()
    if npoint <= 65:  # the counters are those of whole tiles
        plan = DensityPlan(shells, mats, context=gpu_context)
        for t in range(0, npoint, 64):
            plan.evaluate(pts[t:t + 64])
        assert plan.stats() == stats
        plan.close()


@pytest.mark.parametrize("npoint", [7, 4500, 26214, 26215])
def test_host_arrays_give_the_bits_of_device_arrays(npoint, gpu_context):
    import torch

    shells, mats = _water()
    pts = np.random.default_rng(1).normal(scale=2.0, size=(npoint, 3))
    plan = DensityPlan(shells, mats, context=gpu_context)
    host = [plan.evaluate(pts), plan.evaluate(pts[::-1])]
    points = torch.tensor(pts, device=f"cuda:{gpu_context.device}")
    out = torch.empty((2, npoint), dtype=torch.float64, device=points.device)
    plan.evaluate_device(points, out)
    gpu_context.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), host[0])
    plan.evaluate_device(points.flip(0).contiguous(), out)
    gpu_context.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), host[1])
    plan.close()
