"""The connected set of a solid's cells against the oracle where its bitmaps can go wrong: sets that do not hang together (the
flood), rows of 8, 16, 32 and more cells, half spaces along and across the axes, solids cut by the mesh boundary, bitmaps of
a warp, of shared memory and of global memory, concave 2-D shapes; and several contexts alive at once, whose bitmaps need
different amounts of shared memory."""
import numpy as np
import pytest

from gpu_helpers import check_interact, run_pair
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid
from sdfibm_gb300.workloads import Workload

pytestmark = pytest.mark.gpu


def _case(name, rng):
    S = make_shape
    if name == "plates":  # thinner than a cell
        n = (40, 24, 20)
        return n, 0, [(S("Box", radiusa=0.2, radiusb=float(rng.uniform(3, 8)), radiusc=float(rng.uniform(3, 8))),
                       rng.uniform((8, 8, 8), (32, 16, 12)), tuple(rng.uniform(0, 90, 3))) for _ in range(12)]
    if name == "rows":  # boxes along x of 3 .. 70 cells
        n = (90, 12, 11)
        return n, 0, [(S("Box", radiusa=r, radiusb=2.3, radiusc=1.6), (45.2, 5.1, 5.3), (0, 0, 0))
                      for r in (1.4, 3.4, 4.6, 7.4, 8.6, 15.4, 16.6, 35.0)]
    if name == "planes":
        n = (37, 20, 9)
        return n, 0, [(S("Plane"), (0, 10, 4), (0, 0, -90)), (S("Plane"), (37, 10, 4), (0, 0, 90)),
                      (S("Plane"), (18, 7.3, 4), (0, 0, 0)), (S("Plane"), (18, 10, 4.4), (90, 0, 0)),
                      (S("Plane"), (18, 10, 4), (31, 17, 53)), (S("Plane"), (3, 2, 1), (100, 40, 20)),
                      (S("Plane"), (18, 40, 4), (0, 0, 0)), (S("Plane"), (18, 40, 4), (180, 0, 0))]
    if name == "boundary":
        n = (20, 18, 16)
        return n, 0, [(S("Sphere", radius=6.0), c, (0, 0, 0)) for c in ((0, 0, 0), (20, 18, 16), (10, -5.5, 8), (25.9, 9, 8),
                                                                       (10, 9, 22.5))]
    if name == "bitmaps":  # 7, 30 and 90 cells across
        n = (96, 96, 96)
        return n, 0, [(S("Sphere", radius=r), (48.3, 47.9, 48.1), (0, 0, 0)) for r in (2.0, 3.4, 13.0, 25.0, 44.0)]
    if name in ("flat1", "flat2"):  # one- and two-layer meshes: shapes that turn about z, and tilted ones
        n = (30, 26, int(name[4]))
        return n, 0, [(S("Circle", radius=5.2), (14.3, 12.1, 0.4), (0, 0, 20)), (S("Ellipse", radiusa=2.0, radiusb=7.5), (15, 13, 0), (0, 0, 33)),
                      (S("Rectangle", radiusa=6.0, radiusb=1.5), (15, 13, 0), (0, 0, 45)), (S("Circle", radius=1.1), (3, 3, 0), (0, 0, 0)),
                      (S("Plane"), (15, 13, 0), (0, 0, 37)), (S("Plane"), (15, 26, 0), (0, 0, 180)), (S("Plane"), (0, 13, 0), (0, 0, -90)),
                      (S("Circle", radius=4.0), (15, 13, 0.5), (10, 5, 0)), (S("Sphere", radius=4.0), (15, 13, 0.5), (0, 0, 0)),
                      (S("Plane"), (15, 13, 0.7), (60, 20, 10))]
    n = (60, 50, 1)  # "concave": 2-D tails, and one circle of a cell
    return n, 1, [(S("Circle_Tail", radius=4.0, ratio=3.0, thickness=0.4), (20, 20, 0), (0, 0, 25)),
                  (S("Circle_TwoTail", radius=4.0, ratio=3.0, thickness=0.8), (35, 30, 0), (0, 0, 70)),
                  (S("Rectangle", radiusa=15.0, radiusb=0.3), (30, 25, 0), (0, 0, 13)), (S("Circle", radius=0.8), (50, 8, 0), (0, 0, 0))]


@pytest.mark.parametrize("name", ["plates", "rows", "planes", "boundary", "bitmaps", "concave", "flat1", "flat2"])
def test_touched_sets_match_the_oracle(cuda_lib, torch_cuda, name):
    rng = np.random.default_rng(len(name))
    n, twod, shapes = _case(name, rng)
    solids = [make_solid(i, s, 1.4, tuple(np.asarray(x, float)), e, vel=rng.normal(0, 0.1, 3) * (1, 1, 1 - twod),
                         omega=rng.normal(0, 0.1, 3) * ((0, 0, 1) if twod else (1, 1, 1))) for i, (s, x, e) in enumerate(shapes)]
    mesh = abi.mesh_desc(n, (0, 0, -0.5 if twod else 0), (1.0, 1.0, 1.0), twod=twod)
    # one solid at a time: a cell of many solids at once is another test's matter
    for d in solids:
        d.id = 0
        w = Workload(name, mesh, [d], abi.options(rho_f=1.0), 1e-3, (0.1, 0.0, 0.0), 0.05, 5)
        check_interact(w, run_pair(torch_cuda, w, steps=2))


def test_contexts_with_different_shared_memory(cuda_lib, torch_cuda):
    """A context whose bitmaps take 90 KB of shared memory runs after one with 60 KB has been made."""
    torch = torch_cuda
    mesh = abi.mesh_desc((64, 64, 64), (0, 0, 0), (1.0, 1.0, 1.0))
    U = torch.zeros(3, 64 ** 3, device="cuda")
    clouds = [SolidCloud(mesh, [make_solid(0, make_shape("Sphere", radius=r), 1.4, (32, 32, 32))], abi.options(rho_f=1.0))
              for r in (24.5, 19.5, 5.0)]
    for c in clouds:
        c.interact(0.0, 1e-3, U, c.new_fields())
    assert [len(c.touched(0)[0]) > 0 for c in clouds] == [True] * 3
    for c in clouds:
        c.close()
