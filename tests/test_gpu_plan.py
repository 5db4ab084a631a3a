"""The plan of a solid against the oracle: counts at the edges of a CTA's 32 solids, centres that are equally near to several
cells, solids outside the mesh, and elongated solids in mesh units from 1e-6 to 1e6 (their extents are bounded in FP32)."""
import numpy as np
import pytest

from gpu_helpers import check_interact, run_pair
from sdfibm_gb300 import abi
from sdfibm_gb300.host import make_shape, make_solid
from sdfibm_gb300.workloads import Workload

pytestmark = pytest.mark.gpu


def _run(torch, n, h, shapes, steps=2):
    rng = np.random.default_rng(3)
    solids = [make_solid(i, s, 1.4, tuple(np.asarray(x, float) * h), e, vel=rng.normal(0, 0.1, 3) * h, omega=rng.normal(0, 0.1, 3))
              for i, (s, x, e) in enumerate(shapes)]
    w = Workload("plan", abi.mesh_desc(n, (0, 0, 0), (h, h, h)), solids, abi.options(rho_f=1.0), 1e-3, (0.1 * h, 0.0, 0.0), 0.05 * h, 5)
    check_interact(w, run_pair(torch, w, steps=steps))


@pytest.mark.parametrize("count", [0, 1, 31, 32, 33, 65])
def test_solid_counts(cuda_lib, torch_cuda, count):
    rng = np.random.default_rng(count)
    _run(torch_cuda, (40, 36, 30), 1.0, [(make_shape("Sphere", radius=float(rng.uniform(0.4, 3))), rng.uniform(-2, 38, 3),
                                          (0, 0, 0)) for _ in range(count)])


@pytest.mark.parametrize("at", [(10, 10, 10), (10.5, 10, 10), (10, 10.5, 10.5), (0, 0, 0), (20, 18, 16), (20, 0, 8.5), (19.5, -1, 17)])
def test_centres_on_ties(cuda_lib, torch_cuda, at):
    """thin plates: which of the separate sets is kept depends on the cell taken as nearest"""
    for shape in (dict(radiusa=4, radiusb=4, radiusc=0.2), dict(radiusa=0.2, radiusb=5, radiusc=3), dict(radiusa=0.3, radiusb=0.3, radiusc=0.3)):
        for e in ((0, 0, 0), (20, 30, 40)):
            _run(torch_cuda, (20, 18, 16), 1.0, [(make_shape("Box", **shape), at, e)])


@pytest.mark.parametrize("h", [1e-6, 1.0, 1e6])
def test_elongated_in_any_unit(cuda_lib, torch_cuda, h):
    rng = np.random.default_rng(7)
    for name in ("Ellipsoid", "Box"):
        for r in ((9.3, 0.8, 0.7), (0.9, 7.7, 3.1), (1.1, 1.2, 11.9)):
            for _ in range(3):
                x, e = rng.uniform(8, 20, 3), tuple(rng.uniform(0, 360, 3))
                _run(torch_cuda, (30, 28, 26), h, [(make_shape(name, radiusa=r[0] * h, radiusb=r[1] * h, radiusc=r[2] * h), x, e)],
                     steps=1)
