"""apply_forcing and fix_internal bit for bit against the FP64 formulas rounded once: ragged meshes, with and without a
temperature, and values at the ends of the formats (zeros of both signs, denormals, overflow to infinity, infinities, NaN), which
the conversions treat apart."""
import numpy as np
import pytest

from sdfibm_gb300 import abi
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 1e-45, -3e-42, 1.1754942e-38, 1.17549435e-38, -1.2e-38, 3.4028235e38, -3.4e38, np.inf, -np.inf, np.nan],
                   np.float32)


def _setup(torch, n, solids):
    cloud = SolidCloud(abi.mesh_desc(n, (0, 0, 0), (1.0, 1.0, 1.0)), solids, abi.options(rho_f=1.0))
    N = n[0] * n[1] * n[2]
    U = torch.randn(3, N, device="cuda") * 0.1
    f = cloud.new_fields()
    cloud.interact(0.0, 1e-3, U, f)
    return cloud, U, f, N


@pytest.mark.parametrize("temperature", [False, True])
@pytest.mark.parametrize("dt", [1e-3, -0.7, 1e-40, 1e300])
@pytest.mark.parametrize("n", [(7, 5, 3), (31, 17, 9), (64, 48, 40)])
def test_apply_forcing_rounds_once(cuda_lib, torch_cuda, n, dt, temperature):
    torch = torch_cuda
    rng = np.random.default_rng(n[0])
    solids = [make_solid(i, make_shape("Sphere", radius=0.12 * n[2] + 1.0), 1.4, rng.uniform(0, n)) for i in range(5)]
    cloud, U, f, N = _setup(torch, n, solids)
    touched = np.flatnonzero(f["Ct"].cpu().numpy() != 0)
    assert len(touched) > 0
    Uh, Th = U.cpu().numpy().reshape(3, N), rng.normal(300, 10, N).astype(np.float32)
    Fh, Ah, Bh = f["Fs"].cpu().numpy().reshape(3, N), f["As"].cpu().numpy(), f["Ts"].cpu().numpy()
    for a in (Uh, Fh):
        for r in range(3):
            at = rng.choice(touched, max(1, len(touched) // 3))
            a[r, at] = rng.choice(SPECIAL, len(at))
    for a in (Th, Ah, Bh):
        at = rng.choice(touched, max(1, len(touched) // 3))
        a[at] = rng.choice(SPECIAL, len(at))
    U.copy_(torch.from_numpy(Uh).reshape(U.shape))
    f["Fs"].copy_(torch.from_numpy(Fh).reshape(f["Fs"].shape))
    f["As"].copy_(torch.from_numpy(Ah))
    f["Ts"].copy_(torch.from_numpy(Bh))
    T = torch.from_numpy(Th).cuda()
    cloud.apply_forcing(dt, f, U, T if temperature else None)
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        d = lambda x: x.astype(np.float64)
        want_U = (d(Uh) - d(Fh) * dt).astype(np.float32)
        want_T = ((1.0 - d(Ah)) * d(Th) + d(Bh)).astype(np.float32) if temperature else Th
    got_U, got_T = U.cpu().numpy().reshape(3, N), T.cpu().numpy()
    for got, want in ((got_U, want_U), (got_T, want_T)):
        same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
        assert same.all(), "%d values differ" % (~same).sum()
    cloud.close()


def test_fix_internal_rounds_once(cuda_lib, torch_cuda):
    """U inside is v + omega x (C - x): FP64, to the last place of FP32 or the next"""
    torch = torch_cuda
    n = (30, 26, 22)
    rng = np.random.default_rng(1)
    solids = [make_solid(i, make_shape("Sphere", radius=4.0), 1.4, c, vel=v, omega=o) for i, (c, v, o) in
              enumerate([((7, 8, 9), (0, 0, 0), (0, 0, 0)), ((20.3, 14.1, 11.7), rng.normal(size=3), rng.normal(size=3) * 5),
                         ((8, 20, 15), (1e-42, 0, 0), (0, 0, 0))])]
    cloud, U, f, N = _setup(torch, n, solids)
    cloud.fix_internal(f["Ct"], U)
    torch.cuda.synchronize()
    Ct, got = f["Ct"].cpu().numpy(), U.cpu().numpy().reshape(3, N)
    k, j, i = np.unravel_index(np.arange(N), n[::-1])
    C = np.stack([i, j, k], 1) + 0.5
    for s, d in enumerate(solids):
        at = np.flatnonzero(Ct == s + 4)
        assert len(at) > 0
        want = np.array(d.vel) + np.cross(np.array(d.omega), C[at] - np.array(d.pos))
        assert np.all(np.abs(got[:, at].T - want) <= 2.0 ** -23 * np.abs(want) + 1e-45)
    cloud.close()
