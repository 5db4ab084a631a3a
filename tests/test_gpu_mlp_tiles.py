"""Network kernels at the edges of their tiles and of their number formats, against the CPU oracle of the model: cell counts
around a tile and around one wave of CTAs, pre-activations far beyond the range of FP32's exponential (the units that share a
reciprocal must not spoil one another), and a gradient array at every FP32 alignment."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_oracle as MO
from sdfibm_gb300 import abi, learned
from sdfibm_gb300._lib import load

pytestmark = pytest.mark.gpu

FWD_ABS = 2e-5   # the model's contract, as in test_gpu_mlp
GRAD_REL = 2e-2


def _params(seed):
    p = learned.init_params(seed)
    rng = np.random.default_rng(seed + 100)
    p[MO.OFF_B1:MO.OFF_W2] = rng.normal(0, 0.1, 64)
    p[MO.OFF_B2:MO.OFF_W3] = rng.normal(0, 0.1, 64)
    return p


def _check(torch, p, feat, label):
    pd = torch.from_numpy(p).cuda()
    X, y = feat.cpu().numpy().T, label.cpu().numpy().astype(np.float64)
    assert np.abs(learned.forward(torch, pd, feat).cpu().numpy() - MO.forward(p, X)).max() <= FWD_ABS
    loss, g = learned.loss_grad(torch, pd, feat, label)
    lref, gref = MO.loss_grad(p, X, y)
    assert abs(loss - lref) <= 1e-4 * (1 + lref)
    assert np.linalg.norm(g - gref) <= GRAD_REL * np.linalg.norm(gref)


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 255, 128 * 304, 128 * 304 + 1, 128 * 608 + 77])
def test_cell_counts(cuda_lib, torch_cuda, n):
    feat, label, _ = learned.make_dataset(torch_cuda, n, seed=31, n_sub=4)
    _check(torch_cuda, _params(8), feat, label)


@pytest.mark.parametrize("z", [-60.0, -90.0, -1e4, 100.0])
def test_saturated_units(cuda_lib, torch_cuda, z):
    """every other pair of units has one saturated member, in both layers"""
    feat, label, _ = learned.make_dataset(torch_cuda, 500, seed=32, n_sub=4)
    p = _params(9)
    if z < 0:
        p[MO.OFF_B1:MO.OFF_W2][1::4] = z
        p[MO.OFF_B2:MO.OFF_W3][2::4] = z
        p[MO.OFF_B2:MO.OFF_W3][4:6] = z
    else:
        p[MO.OFF_B2:MO.OFF_W3][2] = z
        p[MO.OFF_W3 + 2] = 0.01
    _check(torch_cuda, p, feat, label)


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_gradient_alignment(cuda_lib, torch_cuda, offset):
    torch = torch_cuda
    feat, label, _ = learned.make_dataset(torch, 300, seed=33, n_sub=4)
    p = _params(10)
    pd = torch.from_numpy(p).cuda()
    g = torch.full((abi.MLP_NPARAM + 1 + 8,), 7.0, device="cuda")
    ptr = lambda t, o=0: C.c_void_p(t.data_ptr() + 4 * o)
    torch.cuda.synchronize()
    assert load().sdfibm_mlp_loss_grad(ptr(pd), ptr(feat), ptr(label), feat.stride(0), 300, ptr(g, offset), None) == 0
    g = g.cpu().numpy()
    gref = MO.loss_grad(p, feat.cpu().numpy().T, label.cpu().numpy().astype(np.float64))[1]
    got = g[offset:offset + abi.MLP_NPARAM]
    assert np.linalg.norm(got - gref) <= GRAD_REL * np.linalg.norm(gref)
    assert np.all(g[:offset] == 7.0) and np.all(g[offset + abi.MLP_NPARAM + 1:] == 7.0)
