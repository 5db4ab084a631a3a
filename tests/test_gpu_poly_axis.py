"""REF-GEO of elliptic prisms thinner than a cell whose axes run through the vertices of a polyMesh: the distance on the axis is no
number only where the reference's is none."""
import pytest

from oracle.oracle import OracleCloud
from polymesh_gen import uniform_block
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from test_gpu_ellipse_axis import TILTS, _check, _solids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", TILTS)
def test_polymesh(cuda_lib, torch_cuda, e):
    side, layers, h = 40, 9, 1.0 / 40
    pts, fo, fl, ow, nb, nc = uniform_block((side, side, layers), (0, 0, 0), (h,) * 3)
    solids, opt = _solids(side, layers, 0.0, e), abi.options(rho_f=1.0)
    gpu = SolidCloud.from_polymesh(pts, fo, fl, ow, nb, solids, opt)
    orc = OracleCloud(abi.mesh_desc((1, 1, 1), (0, 0, 0), (1, 1, 1)), solids, opt, faithful=False, polymesh=(pts, fo, fl, ow, nb))
    _check(gpu, orc, nc, torch_cuda)
    gpu.close()
