"""The batched NCP on batches whose problems have different contact counts, none included: a warp's
turns and rows end at the contacts of its own problems, and every problem has the impulses, the
residual, the sweeps and the gradient of its own size alone, bit for bit."""
import importlib

import numpy as np
import pytest

from conftest import cuda_ok
from test_bncp_lanes_gpu import _problems

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]


@pytest.mark.parametrize("wide,most", [(3, 1), (4, 1), (4, 4), (7, 2), (8, 2), (8, 3), (8, 8), (9, 9), (11, 4), (12, 12),
                                       (15, 14), (16, 1), (16, 16)])
def test_ragged_batch_has_the_bits_of_each_problem_alone(me, wide, most):
    import torch
    bn = importlib.import_module("motion_engine_b200.bncp")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    B, n = 41, 3 * wide
    rng = np.random.default_rng(10 * wide + most)
    nc = rng.integers(0, most + 1, B).astype(np.int32)
    nc[0] = most
    G, b, mu = _problems(B, wide, 7)
    beyond = np.arange(n)[None, :] >= 3 * nc[:, None]  # what a caller leaves there must not matter
    G[beyond[:, :, None] | beyond[:, None, :]] = np.nan
    b[beyond], mu[beyond[:, ::3]] = np.nan, np.nan
    g = rng.standard_normal((B, n))
    s = bn.BatchNCP(t(G), t(b), t(mu), torch.from_numpy(nc))
    lam = s.solve(400, 1e-9).cpu().numpy()
    gb, gmu = (x.cpu().numpy() for x in s.vjp(t(g)))
    for e in range(B):
        k, m = int(nc[e]), 3 * int(nc[e])
        assert not lam[e, m:].any() and not gb[e, m:].any() and not gmu[e, k:].any()
        if k == 0:
            assert int(s.iters[e]) == 0 and float(s.res[e]) == 0.0
            continue
        one = bn.BatchNCP(t(G[e:e + 1, :m, :m]), t(b[e:e + 1, :m]), t(mu[e:e + 1, :k]))
        assert one.solve(400, 1e-9).cpu().numpy()[0].tobytes() == lam[e, :m].tobytes()
        assert int(one.iters[0]) == int(s.iters[e]) and float(one.res[0]) == float(s.res[e])
        ob, om = (x.cpu().numpy()[0] for x in one.vjp(t(g[e:e + 1, :m])))
        assert np.array_equal(ob, gb[e, :m], equal_nan=True) and np.array_equal(om, gmu[e, :k], equal_nan=True)
