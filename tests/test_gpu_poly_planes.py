"""Half spaces through the vertices of a polyMesh: the distance there is zero or a rounding of it, and the fraction of the cells
beside it jumps by SMALL / h (the apex of calcApex, geometrictools.cpp:25-45) with its sign, so it has to be the reference's."""
import numpy as np
import pytest

from oracle.oracle import Lowering
from polymesh_gen import uniform_block
from sdfibm_gb300 import abi
from test_gpu_poly import _check, _pair

pytestmark = pytest.mark.gpu
L = Lowering


@pytest.mark.parametrize("h", [1e-3, 1.0 / 64])
@pytest.mark.parametrize("e", [(0, 0, 45.0), (0, 0, -45.0), (0, 0, 135.0), (45.0, 0, 0), (0, 0, 90.0), (0, 0, 180.0), (-90.0, 0, 0),
                               (30.0, 0, 45.0), (0, 0, 26.56505117707799)])
def test_planes_through_vertices(cuda_lib, torch_cuda, e, h):
    n = (16, 15, 14)
    poly = uniform_block(n, (0, 0, 0), (h,) * 3)
    rng = np.random.default_rng(3)
    U = rng.normal(0, 0.1, (3, poly[5]))
    for at in ((8, 8, 7), (4, 3, 2)):
        solids = [L.make_solid(0, L.make_shape("Plane"), 1.3, tuple(h * np.array(at)), e, vel=(0.1, 0.0, -0.1))]
        gpu, orc, fd, fo, FTg, FTo, Uo = _pair(torch_cuda, poly, solids, abi.options(rho_f=1.1), U, 0.01)
        _check(gpu, orc, fd, fo, FTg, FTo, Uo, 0.01, 1.1, 1, vol_mean=h ** 3)
        gpu.close()
