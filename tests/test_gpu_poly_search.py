"""The block search and union-find enumeration of polyMesh contexts (meshes with one point count per cell) and the
breadth-first one (other meshes) against the oracle, at the sizes and shapes where they can go wrong: cell counts around a
block of 128 and a bitmap word of 32, solids that no cell's vertex lies in, solids whose cells do not hang together, half
spaces and tilted prisms, many solids on few cells."""
import numpy as np
import pytest

from oracle.oracle import Lowering
from polymesh_gen import jiggle, uniform_block
from sdfibm_gb300 import abi
from test_gpu_poly import _check, _pair

pytestmark = pytest.mark.gpu
L = Lowering


def _solids(kind, lo, hi, h, rng):
    """Solids of one kind across the box lo..hi of cells of size h."""
    mid = 0.5 * (lo + hi)
    at = lambda: rng.uniform(lo, hi)
    eu = lambda: tuple(rng.uniform(0, 90, 3))
    S = lambda t, **kw: L.make_shape(t, **kw)
    if kind == "spheres":
        return [(S("Sphere", radius=r * h), at(), eu()) for r in (2.2, 1.1, 0.8, 0.45, 0.2)]
    if kind == "outside":  # beyond the mesh, at its corner, and a seed cell without an inside vertex
        return [(S("Sphere", radius=2 * h), hi + 9 * h, (0, 0, 0)), (S("Sphere", radius=2 * h), hi, (0, 0, 0)),
                (S("Ellipsoid", radiusa=0.2 * h, radiusb=3 * h, radiusc=3 * h), mid + 0.45 * h, (0, 0, 0))]
    if kind == "plates":  # thinner than a cell: their cells need not hang together
        return [(S("Box", radiusa=0.15 * h, radiusb=3 * h, radiusc=3 * h), mid, eu()) for _ in range(6)]
    if kind == "planes":
        return [(S("Plane"), mid, eu()), (S("Plane"), lo, (0, 0, 0)), (S("Plane"), hi + 5 * h, (0, 0, 180.0))]
    if kind == "prisms":
        return [(S("Circle", radius=1.7 * h), mid, (0, 0, 30.0)), (S("Ellipse", radiusa=h, radiusb=2 * h), mid, eu()),
                (S("Rectangle", radiusa=1.3 * h, radiusb=0.7 * h), mid, (0, 0, 45.0))]
    return [(S("Sphere", radius=rng.uniform(0.3, 1.5) * h), at(), eu()) for _ in range(40)]  # "many"


def _run(torch, n, kind, seed, poly):
    h = 1.0 / 16
    rng = np.random.default_rng(seed)
    lo, hi = np.zeros(3), np.array(n) * h
    solids = [L.make_solid(i, s, 1.3, tuple(x), e, vel=rng.normal(0, 0.1, 3), omega=rng.normal(0, 1, 3))
              for i, (s, x, e) in enumerate(_solids(kind, lo, hi, h, rng))]
    U = rng.normal(0, 0.1, (3, poly[5]))
    gpu, orc, fd, fo, FTg, FTo, Uo = _pair(torch, poly, solids, abi.options(rho_f=1.1), U, 0.01, steps=2)
    _check(gpu, orc, fd, fo, FTg, FTo, Uo, 0.01, 1.1, len(solids), vol_mean=h ** 3)
    gpu.close()


@pytest.mark.parametrize("kind", ["spheres", "outside", "plates", "planes", "prisms", "many"])
@pytest.mark.parametrize("n", [(3, 3, 3), (31, 1, 1), (8, 4, 4), (43, 3, 1), (11, 10, 9)])
def test_poly_search_matches_the_oracle(cuda_lib, torch_cuda, n, kind):
    poly = list(uniform_block(n, (0, 0, 0), (1.0 / 16,) * 3))
    poly[0] = jiggle(poly[0], 0.2 / 16, 5)
    _run(torch_cuda, n, kind, 100 * sum(n) + len(kind), poly)


@pytest.mark.parametrize("kind", ["spheres", "outside", "planes"])
def test_poly_mixed_point_counts_keep_the_breadth_first_search(cuda_lib, torch_cuda, kind):
    """Two cells of a far corner merged into one of 12 points: the mesh no longer has one point count."""
    n = (9, 8, 7)
    pts, fo, fl, ow, nb, nc = uniform_block(n, (0, 0, 0), (1.0 / 16,) * 3)
    ni = len(nb)
    gone = [f for f in range(ni) if ow[f] == nc - 2 and nb[f] == nc - 1]
    assert len(gone) == 1
    keep = np.array([f for f in range(len(ow)) if f not in gone])
    faces = fl.reshape(-1, 4)[keep]
    ow2 = np.minimum(ow[keep], nc - 2).astype(np.int32)
    nb2 = np.minimum(nb[keep[keep < ni]], nc - 2).astype(np.int32)
    poly = (pts, np.arange(0, 4 * len(faces) + 1, 4, dtype=np.int32), faces.reshape(-1).copy(), ow2, nb2, nc - 1)
    h = 1.0 / 16
    rng = np.random.default_rng(7)
    lo = np.zeros(3)
    solids = [L.make_solid(i, s, 1.3, tuple(np.minimum(x, lo + 3 * h) if kind == "spheres" else x), e)
              for i, (s, x, e) in enumerate(_solids(kind, lo, lo + 4 * h, h, rng))]
    if kind == "planes":
        solids = solids[1:2]  # the half space below the mesh's corner
    U = rng.normal(0, 0.1, (3, nc - 1))
    gpu, orc, fd, fo_, FTg, FTo, Uo = _pair(torch_cuda, poly, solids, abi.options(rho_f=1.1), U, 0.01)
    _check(gpu, orc, fd, fo_, FTg, FTo, Uo, 0.01, 1.1, len(solids), vol_mean=h ** 3)
    gpu.close()
