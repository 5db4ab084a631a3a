"""SUBSAMPLE counts, exactly, where a cloud has cells enough that each lane counts one: shapes mixed in the lists (quadrics, boxes,
half spaces, prisms on a 3-D mesh), axis-aligned boxes whose faces lie on lattice planes, spheres far larger and smaller than a
cell, lattices of 5 to 17 samples, and a recheck list too short for the undecided points; and the same clouds small enough for a
warp per cell."""
import numpy as np
import pytest

from oracle.oracle import OracleCloud
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid

pytestmark = pytest.mark.gpu


def _shapes(kind, rng, count):
    S = make_shape
    out = []
    for i in range(count):
        e = tuple(rng.uniform(0, 360, 3))
        if kind == "mixed":
            s = [S("Sphere", radius=float(rng.uniform(0.3, 5))), S("Box", radiusa=float(rng.uniform(0.4, 5)), radiusb=2.5, radiusc=1.3),
                 S("Ellipsoid", radiusa=0.6, radiusb=float(rng.uniform(1, 6)), radiusc=3.0),
                 S("Circle", radius=float(rng.uniform(1, 4)))][i % 4]
            if i % 4 == 3:
                e = (0, 0, e[2])
        elif kind == "aligned":  # faces on sample planes (multiples of 1/20 of a cell), on cell faces, and between
            s, e = S("Box", radiusa=float(rng.integers(20, 100)) / 20, radiusb=float(rng.integers(20, 100)) / 20, radiusc=float(rng.integers(2, 9)) / 2), (0, 0, 0)
        elif kind == "boxes":
            s = S("Box", radiusa=float(rng.uniform(0.05, 6)), radiusb=float(rng.uniform(0.05, 6)), radiusc=float(rng.uniform(0.05, 6)))
        else:
            s = S("Ellipsoid", radiusa=float(rng.uniform(0.2, 8)), radiusb=float(rng.uniform(0.2, 8)), radiusc=float(rng.uniform(0.2, 8)))
        out.append((s, e))
    return out


def _run(torch, kind, n, count, dims, recheck_cap=0):
    rng = np.random.default_rng(n + count)
    side = np.array(dims)
    solids = []
    step = 13.0
    per = np.maximum(1, (side // step).astype(int))
    for i, (s, e) in enumerate(_shapes(kind, rng, count)):
        at = np.array([i % per[0], i // per[0] % per[1], i // (per[0] * per[1])]) * step + 6.5
        at = at + (rng.integers(-10, 10, 3) / 20 if kind == "aligned" else rng.uniform(-0.5, 0.5, 3))
        solids.append(make_solid(i, s, 1.4, tuple(at), e))
    if kind == "mixed":
        solids.append(make_solid(count, make_shape("Plane"), 1.4, (side[0] / 2, 1.3, side[2] / 2), (0, 0, 3.0)))
    mesh = abi.mesh_desc(dims, (0, 0, 0), (1.0, 1.0, 1.0))
    opt = abi.options(rho_f=1.0, fraction_method=abi.FRACTION_SUBSAMPLE, subsample_n=n)
    opt.recheck_cap = recheck_cap
    cloud, orc = SolidCloud(mesh, solids, opt), OracleCloud(mesh, solids, opt, faithful=False)
    N = int(np.prod(dims))
    f, fo = cloud.new_fields(), orc.new_fields()
    cloud.interact(0.0, 1e-3, torch.zeros(3, N, device="cuda"), f)
    orc.interact(0.0, 1e-3, np.zeros(3 * N), fo)
    cut = cloud.stats()["cut_cells"]
    # counts over n^3, summed where solids share a cell: both sides round sums of the same FP32 fractions
    got, want = f["As"].cpu().numpy().astype(np.float64), np.asarray(fo["As"], np.float64)
    assert np.abs(got - want).max() <= 2.0 ** -22 < 0.25 / n ** 3, np.abs(got - want).max() * n ** 3
    assert np.array_equal(f["Ct"].cpu().numpy(), fo["Ct"])
    cloud.close()
    return cut


LANES = 160 * 152  # cells from which the lanes count (152 SMs; fewer SMs: fewer)


@pytest.mark.parametrize("n", [5, 6, 10, 13, 17])
@pytest.mark.parametrize("kind", ["mixed", "aligned", "boxes", "ellipsoids"])
def test_counts_of_a_cell_per_lane(cuda_lib, torch_cuda, kind, n):
    assert _run(torch_cuda, kind, n, 420, (93, 93, 120)) > LANES


@pytest.mark.parametrize("n", [5, 10, 17])
@pytest.mark.parametrize("kind", ["mixed", "aligned", "boxes", "ellipsoids"])
def test_counts_of_a_cell_per_warp(cuda_lib, torch_cuda, kind, n):
    assert _run(torch_cuda, kind, n, 16, (40, 40, 40)) < LANES


@pytest.mark.parametrize("cap", [1, 40])
def test_short_recheck_list(cuda_lib, torch_cuda, cap):
    assert _run(torch_cuda, "aligned", 10, 420, (93, 93, 120), recheck_cap=cap) > LANES
