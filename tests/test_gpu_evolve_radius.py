"""Contacts of solids without a radius, and of ones whose radii's product is no FP32 number: the law goes by the bounding radii's sum
(collision.cpp:16-35), in the one-launch evolve as in the oracle; alone, among others, and for lists, fast solids and planes."""
import numpy as np
import pytest

from sdfibm_gb300 import abi
from sdfibm_gb300.host import make_shape, make_solid, mask_motion
from test_gpu_evolve import _compare, _evolve_pair

pytestmark = pytest.mark.gpu


def _sphere(i, r, at, radius_b, vel=(0, 0, 0)):
    d = make_solid(i, make_shape("Sphere", radius=r), 1.5, at, vel=vel)
    d.shape.radiusB = radius_b
    return d


@pytest.mark.parametrize("small", [0.0, 1e-40, 1e-25])
@pytest.mark.parametrize("mode", [abi.COLLISION_SPHERES, abi.COLLISION_REFERENCE])
def test_points_and_spheres(cuda_lib, torch_cuda, small, mode):
    mesh = abi.mesh_desc((16, 16, 16), (0.0, 0.0, 0.0), (1.0 / 16,) * 3)
    rng = np.random.default_rng(4)
    solids = [_sphere(0, 0.1, (0.5, 0.5, 0.5), 0.1), _sphere(1, 0.02, (0.53, 0.51, 0.5), small),   # inside the sphere
              _sphere(2, 0.02, (0.2, 0.2, 0.2), small), _sphere(3, 0.02, (0.2, 0.2, 0.2), small),  # one place: 0 >= 0, no direction
              _sphere(4, 0.02, (0.8, 0.2, 0.4), small, vel=(30.0, 0, 0)),                          # fast
              make_solid(5, make_shape("Plane"), 1.0, (0.5, 0.35, 0.5), (0, 0, 0), motion=mask_motion("b000000"))]
    for i in range(30):
        solids.append(_sphere(len(solids), 0.03, tuple(rng.uniform(0.4, 0.6, 3)), small if i % 2 else 0.03))
    sg, so, pairs = _evolve_pair(torch_cuda, mesh, solids, abi.options(rho_f=0.0, collision_mode=mode), 1e-5, 2)
    assert pairs > 30
    assert np.abs(np.array(so[1].force[:])).max() > 0
    _compare(sg, so)
