"""REF-GEO of ellipsoids smaller than a cell with their centres on mesh vertices, to rounding: the distance there is -0.5 over the
rounding's own length, finite unless the offset is exactly zero, and so are the fractions of the cells around it, on meshes of many
layers and of two."""
import numpy as np
import pytest

from oracle.oracle import OracleCloud
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid
from gpu_helpers import AS_REL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,origin,layers", [(40, 0.0, 40), (36, 0.1, 36), (40, 0.0, 2), (56, 0.0, 2)])
def test_vertices_next_to_the_centre(cuda_lib, torch_cuda, side, origin, layers):
    h = 1.0 / side
    solids = []
    for i in range(4, side - 3, 4):
        for j in range(4, side - 3, 4):
            for k in range(4, side - 3, 4) if layers > 2 else (1,):
                s = make_shape("Ellipsoid", radiusa=0.7 * h, radiusb=0.8 * h, radiusc=0.75 * h)
                solids.append(make_solid(len(solids), s, 1.4, (origin + i / side, origin + j / side, origin + k / side)))
    mesh, opt = abi.mesh_desc((side, side, layers), (origin,) * 3, (h,) * 3), abi.options(rho_f=1.0)
    N = side * side * layers
    cloud, orc = SolidCloud(mesh, solids, opt), OracleCloud(mesh, solids, opt)
    f, fo = cloud.new_fields(), orc.new_fields()
    cloud.interact(0.0, 1e-3, torch_cuda.zeros(3, N, device="cuda"), f)
    orc.interact(0.0, 1e-3, np.zeros(3 * N), fo)
    want = np.asarray(fo["Ts"])  # the fraction itself: As = min(Ts, 1) does not keep NaN
    got, ok = f["Ts"].cpu().numpy(), np.isfinite(want)
    assert np.count_nonzero(ok & (want > 0)) > 0
    assert np.all(np.isfinite(got[ok]))
    # sums of FP32 terms below 1
    assert np.all(np.abs(got[ok] - want[ok]) <= AS_REL * np.abs(want[ok]) + 2.0 ** -24)
    cloud.close()
