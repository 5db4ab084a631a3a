"""The word lists of polyMesh contexts whose cells have one point count: touched cells where a solid's cells fill one word, part of a
word, many words of a CTA's share and more words than the grid takes at once; sets of which only the seed's part is kept; and the
memory a context takes for each solid and cell."""
import numpy as np
import pytest

from oracle.oracle import Lowering
from polymesh_gen import jiggle, uniform_block
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from test_gpu_poly import _check, _pair

pytestmark = pytest.mark.gpu
L = Lowering


@pytest.mark.parametrize("n,solids", [((32, 3, 1), [("Sphere", 0.4)]), ((64, 9, 1), [("Sphere", 4.0)]), ((17, 15, 13), [("Sphere", 6.0)] * 3),
                                      ((48, 40, 36), [("Sphere", 15.0)]), ((48, 40, 36), [("Sphere", 15.0), ("plates", 1.0)] * 8),
                                      ((20, 20, 20), [("plates", 1.0)] * 5)])
def test_touched_cells(cuda_lib, torch_cuda, n, solids):
    h = 1.0 / 16
    poly = list(uniform_block(n, (0, 0, 0), (h,) * 3))
    poly[0] = jiggle(poly[0], 0.2 * h, 5)
    rng = np.random.default_rng(sum(n) + len(solids))
    mid = 0.5 * h * np.array(n)
    out = []
    for i, (kind, r) in enumerate(solids):
        x, e = mid + rng.uniform(-0.6, 0.6, 3) * h, tuple(rng.uniform(0, 90, 3))
        shape = L.make_shape("Sphere", radius=r * h) if kind == "Sphere" else L.make_shape("Box", radiusa=0.15 * h, radiusb=6 * h, radiusc=5 * h)
        out.append(L.make_solid(i, shape, 1.3, tuple(x), e, vel=rng.normal(0, 0.1, 3), omega=rng.normal(0, 1, 3)))
    U = rng.normal(0, 0.1, (3, poly[5]))
    gpu, orc, fd, fo, FTg, FTo, Uo = _pair(torch_cuda, poly, out, abi.options(rho_f=1.1), U, 0.01, steps=2)
    _check(gpu, orc, fd, fo, FTg, FTo, Uo, 0.01, 1.1, len(out), vol_mean=h ** 3)
    gpu.close()


def test_memory_of_a_context(cuda_lib, torch_cuda):
    """At most 6 bytes for each solid and cell (the breadth-first search needs 5.1)."""
    n, count = (96, 96, 96), 150
    h = 1.0 / 96
    pts, fo, fl, ow, nb, nc = uniform_block(n, (0, 0, 0), (h,) * 3)
    rng = np.random.default_rng(1)

    def used(solids):
        torch_cuda.cuda.synchronize()
        free = torch_cuda.cuda.mem_get_info()[0]
        cloud = SolidCloud.from_polymesh(pts, fo, fl, ow, nb, solids, abi.options(rho_f=1.0))
        torch_cuda.cuda.synchronize()
        mem = free - torch_cuda.cuda.mem_get_info()[0]
        cloud.close()
        return mem

    solids = [L.make_solid(i, L.make_shape("Sphere", radius=4 * h), 1.3, tuple(rng.uniform(0.1, 0.9, 3))) for i in range(count)]
    used(solids[:1])  # what the first context of a process takes beside its own
    extra = used(solids) - used(solids[:1])
    assert extra <= 6 * (count - 1) * nc + (32 << 20), extra / ((count - 1) * nc)
