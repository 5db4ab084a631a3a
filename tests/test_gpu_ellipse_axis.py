"""REF-GEO of elliptic prisms thinner than a cell whose axes run through mesh vertices, along z, tilted and along the other axes: the
distance on the axis is -0.5 over the length of a rounding, and no number only where the reference's is none; on uniform meshes of
one layer, two and many."""
import numpy as np
import pytest

from oracle.oracle import OracleCloud
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid
from gpu_helpers import AS_REL

pytestmark = pytest.mark.gpu
TILTS = [(0, 0, 0), (0, 0, 30.0), (0, 0, 90.0), (10.0, 20.0, 30.0), (45.0, 0, 0), (30.0, 0, 0), (0, -60.0, 0)]


def _solids(side, layers, origin, e):
    """a few, far enough apart for their prisms to overlap little; more where they are parallel to z"""
    h = 1.0 / side
    upright = e[0] == 0 and e[1] == 0
    at = range(4, side - 3, 4) if upright else range(5, side - 4, 11)
    return [make_solid(0, make_shape("Ellipse", radiusa=0.7 * h, radiusb=0.8 * h), 1.4,
                       (origin + i / side, origin + j / side, origin + (0 if upright else (i + j) % (layers + 1)) / side), e)
            for i in at for j in at]


def _check(gpu, orc, N, torch):
    f, fo = gpu.new_fields(), orc.new_fields()
    gpu.interact(0.0, 1e-3, torch.zeros(3, N, device="cuda"), f)
    orc.interact(0.0, 1e-3, np.zeros(3 * N), fo)
    want, got = np.asarray(fo["Ts"]), f["Ts"].cpu().numpy()  # the fraction itself: As = min(Ts, 1) does not keep NaN
    ok = np.isfinite(want)
    assert np.all(np.isfinite(got[ok])), np.count_nonzero(~np.isfinite(got) & ok)
    # sums of FP32 terms below 1, of a few solids
    assert np.all(np.abs(got[ok] - want[ok]) <= AS_REL * np.abs(want[ok]) + 4 * 2.0 ** -24)


@pytest.mark.parametrize("side,origin,layers", [(40, 0.0, 1), (40, 0.0, 2), (40, 0.0, 9), (36, 0.1, 1), (48, -0.35, 8)])
@pytest.mark.parametrize("e", TILTS)
def test_uniform(cuda_lib, torch_cuda, side, origin, layers, e):
    h = 1.0 / side
    mesh, opt = abi.mesh_desc((side, side, layers), (origin,) * 3, (h,) * 3), abi.options(rho_f=1.0)
    solids = _solids(side, layers, origin, e)
    gpu, orc = SolidCloud(mesh, solids, opt), OracleCloud(mesh, solids, opt)
    _check(gpu, orc, side * side * layers, torch_cuda)
    gpu.close()
