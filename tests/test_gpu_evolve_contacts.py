"""The one-launch evolve with contacts against the oracle at the sizes where its layout changes (a CTA holds 8 solids up to
8 per SM, then more), with solids fast enough that the neighbour lists are made again between sub-steps, neighbour lists
that overflow, forcers and fixed motions, and more plane-like solids than it takes (the launch-per-stage path)."""
import math

import numpy as np
import pytest

from oracle.oracle import OracleCloud
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_forcer, make_shape, make_solid, mask_motion
from test_gpu_evolve import _compare, _evolve_pair

pytestmark = pytest.mark.gpu


def _spheres(rng, n, r, box, speed):
    out = []
    for i in range(n):
        motion = mask_motion("b000000") if i % 7 == 3 else None
        forcer = make_forcer("Spring", 0.5, 0.5, 0.5, 2.0, 0.05) if i % 5 == 2 else None
        out.append(make_solid(i, make_shape("Sphere", radius=float(r * rng.uniform(0.5, 1.5))), 1.5,
                              rng.uniform(box[0], box[1], 3), vel=rng.normal(0, speed, 3), omega=rng.normal(0, 1, 3),
                              motion=motion, forcer=forcer))
    return out


@pytest.mark.parametrize("n,r,speed", [(2, 0.1, 0.1), (7, 0.15, 0.1), (8, 0.15, 0.1), (9, 0.15, 0.1), (33, 0.08, 40.0), (100, 0.06, 40.0),
                                       (257, 0.04, 0.1), (1217, 0.02, 10.0)])
def test_contacts_match_the_oracle(cuda_lib, torch_cuda, n, r, speed):
    rng = np.random.default_rng(n)
    mesh = abi.mesh_desc((12, 12, 12), (0.0, 0.0, 0.0), (1.0 / 12,) * 3)
    solids = _spheres(rng, n, r, (0.25, 0.75), speed)
    solids.append(make_solid(n, make_shape("Plane"), 1.0, (0.5, 0.3, 0.5), (0, 0, 10.0), motion=mask_motion("b000000")))
    # the contact law is stiff (1e4 per unit depth against masses of r^3): a step short of its period
    dt = 2e-3 * math.sqrt(4.19 * 1.5 * (0.5 * r) ** 3 / 1e4) * 20
    opt = abi.options(rho_f=0.0, collision_mode=abi.COLLISION_SPHERES, gravity=(0, -1.0, 0))
    sg, so, pairs = _evolve_pair(torch_cuda, mesh, solids, opt, dt, 2)
    assert n < 9 or pairs > 0
    _compare(sg, so)


def test_lists_that_overflow(cuda_lib, torch_cuda):
    """200 spheres that all touch each other: every list is longer than it can hold."""
    rng = np.random.default_rng(3)
    mesh = abi.mesh_desc((12, 12, 12), (0.0, 0.0, 0.0), (1.0 / 12,) * 3)
    solids = _spheres(rng, 200, 0.2, (0.45, 0.55), 0.1)
    opt = abi.options(rho_f=0.0, collision_mode=abi.COLLISION_SPHERES)
    # evolve alone: so many solids on one cell are more than a coupling pass takes
    gpu, orc = SolidCloud(mesh, solids, opt), OracleCloud(mesh, solids, opt, faithful=False)
    for i in range(2):
        gpu.evolve(1e-5 * i, 1e-5)
        orc.evolve(1e-5 * i, 1e-5)
    assert orc.last_pairs() > 200 * 150 // 2
    _compare(gpu.states(), orc.get_state())


@pytest.mark.parametrize("nplanes", [64, 65])
def test_many_planes(cuda_lib, torch_cuda, nplanes):
    """Ellipsoids under the reference's contact table act as planes: as many as one launch takes, and one more."""
    rng = np.random.default_rng(nplanes)
    mesh = abi.mesh_desc((12, 12, 12), (0.0, 0.0, 0.0), (1.0 / 12,) * 3)
    solids = [make_solid(i, make_shape("Ellipsoid", radiusa=0.05, radiusb=0.06, radiusc=0.04), 1.5,
                         rng.uniform(0.2, 0.8, 3), euler_deg=rng.uniform(0, 90, 3)) for i in range(nplanes)]
    for i in range(30):
        solids.append(make_solid(nplanes + i, make_shape("Sphere", radius=0.08), 1.5, rng.uniform(0.2, 0.8, 3),
                                 vel=rng.normal(0, 0.1, 3)))
    opt = abi.options(rho_f=0.0, collision_mode=abi.COLLISION_REFERENCE, gravity=(0, -1.0, 0))
    sg, so, _ = _evolve_pair(torch_cuda, mesh, solids, opt, 1e-4, 2)
    _compare(sg, so)
