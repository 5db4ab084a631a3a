"""Evolve with contacts where some solids cross several of their own sizes in a step: one of them, as many as the list of fast
solids holds, one more (every sub-step then lists the pairs anew), all; and on both sides of the largest cloud that is done in
one launch."""
import numpy as np
import pytest

from sdfibm_gb300 import abi
from sdfibm_gb300.host import make_shape, make_solid
from test_gpu_evolve import _compare, _evolve_pair

pytestmark = pytest.mark.gpu


def _cloud(n, fast, dt):
    rng = np.random.default_rng(n + fast)
    r = 0.3 * (1.0 / n) ** (1 / 3)
    return [make_solid(i, make_shape("Sphere", radius=float(r * rng.uniform(0.7, 1.3))), 1.5, rng.uniform(0.1, 0.9, 3),
                       vel=rng.normal(0, 1, 3) * (4 * r / dt if i % max(1, n // max(1, fast)) == 0 and i // max(1, n // max(1, fast)) < fast
                                                  else 0.01)) for i in range(n)]


@pytest.mark.parametrize("n,fast", [(300, 0), (300, 1), (300, 31), (300, 32), (300, 33), (300, 300), (40, 40), (1217, 40), (3040, 5),
                                    (3040, 200), (3041, 5)])
def test_fast_solids(cuda_lib, torch_cuda, n, fast):
    dt = 1e-6  # far below the contact law's period
    mesh = abi.mesh_desc((12, 12, 12), (0.0, 0.0, 0.0), (1.0 / 12,) * 3)
    solids = _cloud(n, fast, dt)
    opt = abi.options(rho_f=0.0, collision_mode=abi.COLLISION_SPHERES)
    sg, so, pairs = _evolve_pair(torch_cuda, mesh, solids, opt, dt, 2)
    assert pairs > 0
    _compare(sg, so)
