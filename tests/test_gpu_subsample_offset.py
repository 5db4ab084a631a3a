"""SUBSAMPLE counts, exactly, of boxes whose centre of mass lies many half extents away and whose faces are turned out of the lattice
planes by next to nothing to either side, and of lattices of more than 32 samples per axis; a lane and a warp per cell."""
import numpy as np
import pytest

from oracle.oracle import OracleCloud
from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid

pytestmark = pytest.mark.gpu


def _run(torch, solids, dims, n):
    mesh = abi.mesh_desc(dims, (0, 0, 0), (1.0, 1.0, 1.0))
    opt = abi.options(rho_f=1.0, fraction_method=abi.FRACTION_SUBSAMPLE, subsample_n=n)
    cloud, orc = SolidCloud(mesh, solids, opt), OracleCloud(mesh, solids, opt, faithful=False)
    N = int(np.prod(dims))
    f, fo = cloud.new_fields(), orc.new_fields()
    cloud.interact(0.0, 1e-3, torch.zeros(3, N, device="cuda"), f)
    orc.interact(0.0, 1e-3, np.zeros(3 * N), fo)
    cut = cloud.stats()["cut_cells"]
    got, want = f["As"].cpu().numpy().astype(np.float64), np.asarray(fo["As"], np.float64)
    # counts over n^3 of cells of one solid each: both sides round the same quotient
    assert np.abs(got - want).max() <= 2.0 ** -22 < 0.25 / n ** 3, np.abs(got - want).max() * n ** 3
    cloud.close()
    return cut


def _at(i, per, step):
    return np.array([i % per, i // per % per, i // (per * per)]) * step + 0.5 * step


def _lanes(torch):
    return 160 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("com", [0.0, 7.3, -61.0])
@pytest.mark.parametrize("turn", [0.0, 1e-7, -1e-7, 1e-5, -1e-5])
def test_boxes_off_their_centre_of_mass(cuda_lib, torch_cuda, com, turn):
    rng = np.random.default_rng(3)
    for per, many in ((7, True), (2, False)):
        solids = []
        for i in range(per ** 3):
            r = rng.integers(40, 100, 3) / 20
            c = np.array([com, -0.4 * com, 0.7 * com])
            s = make_shape("Box", com=tuple(c), radiusa=float(r[0]), radiusb=float(r[1]), radiusc=float(r[2]))
            # the box's own centre lies at -com in the local frame
            solids.append(make_solid(i, s, 1.4, tuple(_at(i, per, 13.0) + c + rng.integers(-10, 10, 3) / 20), (turn, 2 * turn, -turn)))
        side = int(13 * per)
        cut = _run(torch_cuda, solids, (side, side, side), 10)
        assert (cut >= _lanes(torch_cuda)) == many


def _shapes(rng, count, per, step):
    S = make_shape
    solids = []
    for i in range(count):
        s = [S("Sphere", radius=float(rng.uniform(2.5, 3.6))), S("Box", radiusa=2.4, radiusb=float(rng.uniform(1, 2.4)), radiusc=2.0),
             S("Ellipsoid", radiusa=3.0, radiusb=float(rng.uniform(2, 3.6)), radiusc=2.6)][i % 3]
        solids.append(make_solid(i, s, 1.4, tuple(_at(i, per, step) + rng.uniform(-0.4, 0.4, 3)), tuple(rng.uniform(0, 90, 3))))
    return solids


def _fractions(torch, solids, dims, n):
    opt = abi.options(rho_f=1.0, fraction_method=abi.FRACTION_SUBSAMPLE, subsample_n=n)
    cloud = SolidCloud(abi.mesh_desc(dims, (0, 0, 0), (1.0, 1.0, 1.0)), solids, opt)
    f = cloud.new_fields()
    cloud.interact(0.0, 1e-3, torch.zeros(3, int(np.prod(dims)), device="cuda"), f)
    cut = cloud.stats()["cut_cells"]
    cloud.close()
    return f["As"], cut


@pytest.mark.parametrize("n", [32, 33, 47])
def test_lattices_of_more_than_32(cuda_lib, torch_cuda, n):
    """Few solids (a warp per cell) against the oracle; many (a lane per cell) against the same solids a few at a time."""
    assert _run(torch_cuda, _shapes(np.random.default_rng(n), 8, 2, 9.0), (18, 18, 18), n) < _lanes(torch_cuda)
    solids = _shapes(np.random.default_rng(n), 729, 9, 9.0)
    got, cut = _fractions(torch_cuda, solids, (81, 81, 81), n)
    if cut < _lanes(torch_cuda):
        pytest.skip("more SMs than this cloud has cells for")
    want = torch_cuda.zeros_like(got)
    for i in range(0, 729, 81):  # a layer of solids; no cell has two
        part, c = _fractions(torch_cuda, solids[i:i + 81], (81, 81, 81), n)
        assert c < _lanes(torch_cuda)
        want += part
    assert torch_cuda.equal(got, want)
