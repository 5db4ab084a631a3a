"""Evolve with contacts at the edges of the one-launch path on the SM count there is: one CTA, a last CTA of one solid, more than
eight solids a CTA, the largest cloud and one solid more."""
import pytest

from sdfibm_gb300 import abi
from test_gpu_evolve import _compare, _evolve_pair
from test_gpu_evolve_fast import _cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm,more", [(0, 1), (0, 8), (0, 9), (8, 1), (13, 0), (20, 0), (20, 1)])
def test_edges_of_one_launch(cuda_lib, torch_cuda, per_sm, more):
    n = per_sm * torch_cuda.cuda.get_device_properties(0).multi_processor_count + more
    dt = 1e-6
    mesh = abi.mesh_desc((12, 12, 12), (0.0, 0.0, 0.0), (1.0 / 12,) * 3)
    sg, so, pairs = _evolve_pair(torch_cuda, mesh, _cloud(n, 3, dt), abi.options(rho_f=0.0, collision_mode=abi.COLLISION_SPHERES), dt, 2)
    assert n < 100 or pairs > 0
    _compare(sg, so)
