"""Network units far from zero, further than the exponent that two units share a reciprocal over: below they are off, whatever their
distance, and above they are what they are beside one that is off; a unit that is no number says so.  Against the CPU oracle of the
model, in both layers."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO
from sdfibm_gb300 import learned
from test_gpu_mlp_tiles import FWD_ABS, GRAD_REL, _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layer", [1, 2])
@pytest.mark.parametrize("z,top", [(-41.6, 0.0), (-1e6, 0.0), (-1e20, 0.0), (-1e30, 0.0), (-3e38, 0.0), (-50.0, 1e12), (-1e30, 1e24)])
def test_units_far_from_zero(cuda_lib, torch_cuda, layer, z, top):
    feat, label, _ = learned.make_dataset(torch_cuda, 300, seed=34, n_sub=4)
    p = _params(11)
    first, end = (MO.OFF_B1, MO.OFF_W2) if layer == 1 else (MO.OFF_B2, MO.OFF_W3)
    p[first:end][1::4] = z       # beside units in the ordinary range
    p[first:end][4:6] = z        # and beside one another
    if top:
        p[first:end][8] = top
    pd = torch_cuda.from_numpy(p).cuda()
    X, y = feat.cpu().numpy().T, label.cpu().numpy().astype(np.float64)
    assert np.abs(learned.forward(torch_cuda, pd, feat).cpu().numpy() - MO.forward(p, X)).max() <= FWD_ABS
    loss, g = learned.loss_grad(torch_cuda, pd, feat, label)
    lref, gref = MO.loss_grad(p, X, y)
    assert abs(loss - lref) <= 1e-4 * (1 + lref)
    assert np.linalg.norm(g - gref) <= GRAD_REL * np.linalg.norm(gref)


def test_a_cell_that_is_no_number(cuda_lib, torch_cuda):
    feat, _, _ = learned.make_dataset(torch_cuda, 300, seed=35, n_sub=4)
    pd = torch_cuda.from_numpy(_params(12)).cuda()
    want = learned.forward(torch_cuda, pd, feat).cpu().numpy()
    feat[3, 130] = float("nan")
    got = learned.forward(torch_cuda, pd, feat).cpu().numpy()
    assert np.isnan(got[130]) and np.array_equal(np.delete(got, 130), np.delete(want, 130))
