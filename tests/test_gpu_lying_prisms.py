"""2-D shapes tilted so far that their prisms lie in the mesh layers (the local z axis more than 72 degrees from the mesh's): they cross
the whole mesh, and every cell of them is touched; against the oracle."""
import numpy as np
import pytest

from gpu_helpers import check_interact, run_pair
from sdfibm_gb300 import abi
from sdfibm_gb300.host import make_shape, make_solid
from sdfibm_gb300.workloads import Workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [abi.FRACTION_REFGEO, abi.FRACTION_SUBSAMPLE])
@pytest.mark.parametrize("e", [(90.0, 0, 0), (0, 90.0, 0), (75.0, 0, 0), (0, -80.0, 30.0), (88.0, 0, 45.0)])
@pytest.mark.parametrize("n", [(61, 20, 17), (18, 70, 9), (40, 33, 2)])
def test_prisms_that_lie(cuda_lib, torch_cuda, n, e, method):
    h = 1.0 / 64
    mid = 0.5 * h * np.array(n)
    rng = np.random.default_rng(sum(n))
    shapes = [make_shape("Circle", radius=2.3 * h), make_shape("Rectangle", radiusa=1.6 * h, radiusb=2.7 * h), make_shape("Ellipse", radiusa=3.1 * h, radiusb=1.2 * h)]
    solids = [make_solid(0, shapes[sum(n) % 3], 1.4, tuple(mid + rng.uniform(-0.4, 0.4, 3) * h), e, vel=(0.1, 0, 0.2), omega=(1, 2, -1))]
    mesh = abi.mesh_desc(n, (0.0, 0.0, 0.0), (h, h, h))
    w = Workload("lying", mesh, solids, abi.options(rho_f=1.0, fraction_method=method, subsample_n=6), 1e-3, (0.1, 0.0, 0.0), 0.05, 5)
    check_interact(w, run_pair(torch_cuda, w))
