"""Touched sets against the oracle in clouds of so many solids that several of them share a CTA: groups of 128 threads, and warps
with bitmaps up to their largest size, each with connected sets, sets that have to be flooded, solids outside the mesh, and
rows of every alignment."""
import numpy as np
import pytest

from oracle.oracle import OracleCloud
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid

pytestmark = pytest.mark.gpu


def _shape(rng, i, size):
    if i % 5 == 0:
        return make_shape("Sphere", radius=float(size * rng.uniform(0.3, 1.0)))
    if i % 5 == 1:  # thinner than a cell: not connected
        return make_shape("Box", radiusa=0.2, radiusb=float(0.6 * size), radiusc=float(0.6 * size * rng.uniform(0.3, 1)))
    if i % 5 == 2:
        return make_shape("Ellipsoid", radiusa=float(size), radiusb=float(0.3 * size), radiusc=float(0.5 * size))
    if i % 5 == 3:
        return make_shape("Box", radiusa=float(0.55 * size), radiusb=float(0.4 * size), radiusc=float(0.5 * size))
    return make_shape("Ellipsoid", radiusa=0.45, radiusb=float(0.9 * size), radiusc=0.6)


def _compare(torch, n, solids, which):
    mesh = abi.mesh_desc(n, (0, 0, 0), (1.0, 1.0, 1.0))
    opt = abi.options(rho_f=1.0)
    cloud, orc = SolidCloud(mesh, solids, opt), OracleCloud(mesh, [solids[s] for s in which], opt, faithful=False)
    U = torch.zeros(3, n[0] * n[1] * n[2], device="cuda")
    cloud.interact(0.0, 1e-3, U, cloud.new_fields())
    orc.interact(0.0, 1e-3, np.zeros(U.numel()), orc.new_fields())
    for i, s in enumerate(which):
        cg, tg = cloud.touched(s)
        co, to = orc.touched(i)
        assert np.array_equal(cg, co) and np.array_equal(tg, to), "solid %d: %d cells against %d" % (s, len(cg), len(co))
    cloud.close()


@pytest.mark.parametrize("size", [2.0, 4.0, 6.5, 9.0])
def test_groups(cuda_lib, torch_cuda, size):
    """up to 11, 100, 300 and 440 rows a solid: warps, and groups of 128 threads"""
    rng = np.random.default_rng(int(size * 2))
    step = 2 * size + 2.2
    at = [((i % 11) + 0.3, (i // 11 % 9) + 0.5, (i // 99) + 0.4) for i in range(800)]
    n = (int(11 * step), int(9 * step) + 1, int(8 * step) + 2)
    solids = [make_solid(i, _shape(rng, i, size), 1.4, tuple(step * np.array(p) + rng.uniform(-0.3, 0.3, 3)), tuple(rng.uniform(0, 360, 3)))
              for i, p in enumerate(at)]
    _compare(torch_cuda, n, solids, list(range(800)))


def test_largest_warps(cuda_lib, torch_cuda):
    """bitmaps of 129 to 256 words go to a warp in clouds of 64 solids an SM"""
    rng = np.random.default_rng(5)
    n = (72, 72, 110)
    solids = [make_solid(i, make_shape("Sphere", radius=0.4), 1.4, (3 * (i % 24) + 1.4, 3 * (i // 24 % 24) + 1.6, 3 * (i // 576) + 1.2))
              for i in range(16 * 576 + 576)]
    for j in range(50):
        solids.append(make_solid(len(solids), _shape(rng, j, 6.0), 1.4,
                                 (14.4 * (j % 5) + 7.2, 14.4 * (j // 5 % 5) + 7.2, 73 + 16 * (j // 25) + 1.0), tuple(rng.uniform(0, 360, 3))))
    _compare(torch_cuda, n, solids, list(range(0, 9792, 97)) + list(range(9792, len(solids))))
