"""Work items of the classify pass: on one- and two-layer meshes the solids its first kernel does not take (tailed circles, tilted
prisms, 3-D shapes) against the oracle, few and many of them, and beside solids that kernel takes; their tiles go to as many warps
as there are; and the launches a call reports."""
import numpy as np
import pytest

from gpu_helpers import check_interact, run_pair
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid
from sdfibm_gb300.workloads import Workload

pytestmark = pytest.mark.gpu


def _flat(side, kinds, count, nz=1):
    h = 1.0 / side
    rng = np.random.default_rng(side + count)
    per = int(np.ceil(count ** 0.5))
    solids = []
    for i in range(count):
        kind, e = kinds[i % len(kinds)], (0.0, 0.0, float(rng.uniform(0, 360)))
        at = ((i % per + 0.5) / per, (i // per + 0.5) / per, 0.0)
        if kind in ("Circle_Tail", "Circle_TwoTail"):
            s = make_shape(kind, radius=6.3 * h, ratio=1.0, thickness=2.1 * h)
        elif kind == "tilted":
            s, e = make_shape("Circle", radius=5.2 * h), (20.0, 15.0, 0.0)
        elif kind == "Circle":
            s = make_shape("Circle", radius=5.2 * h)
        elif kind == "Sphere":
            s = make_shape("Sphere", radius=4.7 * h)
        else:
            s, e = make_shape("Box", radiusa=4 * h, radiusb=3 * h, radiusc=5 * h), tuple(rng.uniform(0, 90, 3))
        solids.append(make_solid(i, s, 1.4, at, e, vel=rng.normal(0, 0.1, 3), omega=rng.normal(0, 1, 3)))
    mesh = abi.mesh_desc((side, side, nz), (0.0, 0.0, -0.5 * h * nz), (h, h, h), twod=int(nz == 1 and "tilted" not in kinds
                                                                                       and "Sphere" not in kinds))
    return mesh, solids


@pytest.mark.parametrize("method", [abi.FRACTION_REFGEO, abi.FRACTION_SUBSAMPLE])
@pytest.mark.parametrize("kinds,count,nz", [(("Circle_Tail",), 1, 1), (("Circle_Tail", "Circle_TwoTail", "Circle"), 49, 1),
                                            (("tilted",), 1, 1), (("Circle", "tilted", "Sphere", "Box"), 36, 2)])
def test_flat_shapes_of_the_second_kernel(cuda_lib, torch_cuda, kinds, count, nz, method):
    mesh, solids = _flat(160, kinds, count, nz)
    w = Workload("flat", mesh, solids, abi.options(rho_f=1.0, fraction_method=method, subsample_n=8), 1e-3, (0.1, 0.0, 0.0), 0.05, 5)
    check_interact(w, run_pair(torch_cuda, w, steps=2))


def _classify_us(torch, mesh, solids):
    cloud = SolidCloud(mesh, solids, abi.options(rho_f=1.0, timing=1))
    f = cloud.new_fields()
    U = torch.zeros(3, mesh.nx * mesh.ny * mesh.nz, device="cuda")
    best = 1e9
    for _ in range(12):
        cloud.interact(0.0, 1e-3, U, f, want_ft=False)
        best = min(best, cloud.kernel_times()["classify_kernel"] * 1e3)
    items = cloud.stats()["work_items"]
    cloud.close()
    return best, items


def test_neighbouring_tiles_go_to_different_warps(cuda_lib, torch_cuda):
    """A tailed circle of some eighty one-tile items takes no longer than one of a few: a warp each (32 neighbours a warp would
    take several times as long)."""
    h = 1.0 / 400
    mesh = abi.mesh_desc((400, 400, 1), (0.0, 0.0, -0.5), (h, h, 1.0), twod=1)
    few, n_few = _classify_us(torch_cuda, mesh, [make_solid(0, make_shape("Circle_Tail", radius=h, ratio=0.5, thickness=0.5 * h), 1.4,
                                                            (0.5, 0.5, 0.0))])
    many, n_many = _classify_us(torch_cuda, mesh, [make_solid(0, make_shape("Circle_Tail", radius=14 * h, ratio=1.0, thickness=4 * h),
                                                              1.4, (0.5, 0.5, 0.0))])
    assert n_few <= 9 and n_many >= 64
    assert many <= 4 * few, (many, few)


@pytest.mark.parametrize("dims,shapes,classify", [((40, 40, 40), ("Sphere",), 1), ((40, 40, 40), ("Sphere", "Circle"), 2),
                                                  ((40, 40, 40), ("Circle",), 1), ((40, 40, 1), ("Circle",), 2),
                                                  ((40, 40, 1), ("Circle", "Circle_Tail"), 2), ((40, 40, 1), ("Circle_Tail",), 1)])
def test_launches_of_a_call(cuda_lib, torch_cuda, dims, shapes, classify):
    """plan, connect, claim, scan and reset, fractions, couple, finalize, and the classify kernels that have chunks"""
    kw = dict(Sphere=dict(radius=3.0), Circle=dict(radius=3.0), Circle_Tail=dict(radius=3.0, ratio=1.0, thickness=1.0))
    solids = [make_solid(i, make_shape(s, **kw[s]), 1.4, (12.0 + 15 * i, 20.0, 0.5 * dims[2])) for i, s in enumerate(shapes)]
    cloud = SolidCloud(abi.mesh_desc(dims, (0, 0, 0), (1.0, 1.0, 1.0)), solids, abi.options(rho_f=1.0))
    U = torch_cuda.zeros(3, dims[0] * dims[1] * dims[2], device="cuda")
    cloud.interact(0.0, 1e-3, U, cloud.new_fields())
    assert cloud.stats()["launches"] == 7 + classify
    cloud.close()


WALLS = [((0.0, 0.5, 0.5), (0, 0, -90.0)), ((1.0, 0.5, 0.5), (0, 0, 90.0)), ((0.5, 0.0, 0.5), (0, 0, 0.0)),
         ((0.5, 1.0, 0.5), (0, 0, 180.0)), ((0.5, 0.5, 0.0), (90.0, 0, 0)), ((0.5, 0.5, 1.0), (-90.0, 10.0, 0))]


@pytest.mark.parametrize("n,spheres", [((31, 33, 30), 1), ((64, 60, 57), 4), ((96, 40, 1), 2)])
def test_items_of_half_spaces(cuda_lib, torch_cuda, n, spheres):
    """Items of two tiles or more for the walls of a cloud of few solids, whose own items are single tiles."""
    h = 1.0 / max(n)
    flat = n[2] == 1
    walls = [w for w in WALLS if not flat or w[1][:2] == (0, 0)]
    solids = [make_solid(i, make_shape("Plane"), 1.4, tuple(np.array(p) * h * np.array(n)), e) for i, (p, e) in enumerate(walls)]
    for i in range(spheres):
        x = (np.array([0.3, 0.4, 0.5]) + 0.25 * (i % 2)) * h * np.array(n)
        solids.append(make_solid(len(solids), make_shape("Circle" if flat else "Sphere", radius=3.3 * h), 1.4, tuple(x)))
    mesh = abi.mesh_desc(n, (0.0, 0.0, 0.0), (h, h, h))
    w = Workload("walls", mesh, solids, abi.options(rho_f=1.0), 1e-3, (0.1, 0.0, 0.0), 0.05, 5)
    r = run_pair(torch_cuda, w, steps=2)
    check_interact(w, r)
    side, layers = (8, 2) if flat else (4, 4)
    tiles = [-(-d // t) for d, t in zip(n, (side, side, layers))]
    own = spheres * (4 if flat else 4 ** 3)  # 11 cells a side
    assert r["gpu"].stats()["work_items"] <= len(walls) * -(-int(np.prod(tiles)) // 2) + own


@pytest.mark.parametrize("dims,shape,items", [((400, 200, 1), dict(radius=5.0), 9), ((48, 48, 48), dict(radius=6.0), 125)])
def test_tuning_keeps_the_items_of_a_small_cloud(cuda_lib, torch_cuda, dims, shape, items):
    """One solid's tiles are an item each, with a warp for every one of them, and stay so when the autotuner has chosen."""
    s = make_shape("Circle" if dims[2] == 1 else "Sphere", **shape)
    cloud = SolidCloud(abi.mesh_desc(dims, (0, 0, 0), (1.0, 1.0, 1.0)), [make_solid(0, s, 1.4, tuple(0.47 * d for d in dims))],
                       abi.options(rho_f=1.0))
    U = torch_cuda.zeros(3, int(np.prod(dims)), device="cuda")
    f = cloud.new_fields()
    cloud.interact(0.0, 1e-3, U, f)
    assert cloud.stats()["work_items"] == items
    want = {k: v.clone() for k, v in f.items()}
    assert cloud.autotune(1e-3, U, f) in (2, 4, 8, 16, 32)
    cloud.interact(0.0, 1e-3, U, f)
    assert cloud.stats()["work_items"] == items
    assert all(torch_cuda.equal(want[k], f[k]) for k in f)
    cloud.close()


def test_tuning_knows_the_forcing(cuda_lib, torch_cuda):
    """The FP64 and the FP32 forcing are different kernels: a choice made for one is not taken for the other."""
    mesh = abi.mesh_desc((44, 43, 41), (0, 0, 0), (1.0, 1.0, 1.0))
    solids = [make_solid(0, make_shape("Sphere", radius=6.0), 1.4, (21.0, 20.0, 19.0))]
    U = torch_cuda.zeros(3, 44 * 43 * 41, device="cuda")
    cached = []
    for exact in (1, 0, 1, 0):
        cloud = SolidCloud(mesh, solids, abi.options(rho_f=1.0, exact_forcing=exact))
        cloud.autotune(1e-3, U, cloud.new_fields())
        cached.append(cloud.tuning()["from_cache"])
        cloud.close()
    assert cached == [0, 0, 1, 1]


def test_vertex_distances_are_reserved_where_they_are_listed(cuda_lib, torch_cuda):
    """REF-GEO in 3-D: 32 bytes a bbox cell for the vertex distances that the classify pass lists, which it does for none of the
    shapes of its first kernel."""
    h = 1.0 / 64

    def used(shapes):
        solids = [make_solid(i, s, 1.4, (0.5, 0.5, 0.5)) for i, s in enumerate(shapes)]
        torch_cuda.cuda.synchronize()
        free = torch_cuda.cuda.mem_get_info()[0]
        cloud = SolidCloud(abi.mesh_desc((64, 64, 64), (0, 0, 0), (h, h, h)), solids, abi.options(rho_f=1.0))
        torch_cuda.cuda.synchronize()
        mem = free - torch_cuda.cuda.mem_get_info()[0]
        cloud.close()
        return mem

    spheres = [make_shape("Sphere", radius=20 * h)] * 200
    cells = 200 * 45 ** 3
    used(spheres[:1])
    assert used(spheres + [make_shape("Circle", radius=2 * h)]) - used(spheres) >= 30 * cells
