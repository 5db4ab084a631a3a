"""Solid states read back through the staging of small clouds and by the plain copy of larger ones: the same states as were
set, on both sides of the limit; and gradient calls of several threads at once, each with sums of its own."""
import threading

import numpy as np
import pytest

from sdfibm_gb300 import abi, learned
from sdfibm_gb300.cloud import SolidCloud
from sdfibm_gb300.host import make_shape, make_solid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 255, 256, 257, 700])
def test_states_round_trip(cuda_lib, torch_cuda, count):
    cloud = SolidCloud(abi.mesh_desc((8, 8, 8), (0, 0, 0), (1, 1, 1)),
                       [make_solid(i, make_shape("Sphere", radius=0.5), 1.4, (4, 4, 4)) for i in range(count)], abi.options(rho_f=1.0))
    st = cloud.states()
    rng = np.random.default_rng(count)
    for s in st:
        s.pos[:] = rng.normal(size=3).tolist()
        s.forcer_torque_old[:] = rng.normal(size=3).tolist()
        s.first_fluid_step, s.first_forcer_step = int(rng.integers(2)), int(rng.integers(2))
    cloud.set_states(st)
    assert [bytes(s) for s in cloud.states()] == [bytes(s) for s in st]
    cloud.close()


def test_gradients_of_several_threads(cuda_lib, torch_cuda):
    torch = torch_cuda
    sets = [learned.make_dataset(torch, 2000 + 300 * i, seed=40 + i, n_sub=4)[:2] for i in range(4)]
    params = [torch.from_numpy(learned.init_params(i)).cuda() for i in range(4)]
    alone = [learned.loss_grad(torch, p, *d) for p, d in zip(params, sets)]
    out = [[] for _ in sets]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                out[i].append(learned.loss_grad(torch, params[i], *sets[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(4):
        assert len(out[i]) == 20
        for loss, g in out[i]:  # FP32 sums of the same addends in another order: 5e3 adds of 2^-24 each at most
            assert abs(loss - alone[i][0]) <= 1e-5 * alone[i][0]
            assert np.linalg.norm(g - alone[i][1]) <= 1e-4 * np.linalg.norm(alone[i][1])
