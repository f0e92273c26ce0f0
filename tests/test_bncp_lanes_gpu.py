"""The batched NCP solve at the contact counts where its layout changes (one lane a contact: 1, 2,
4, 8 or 16 lanes a problem; G in registers up to 8 contacts, in shared memory above), against the
oracle's PGS, and padded: a problem in a wider batch gives the bits it gives alone.

Tolerance: both iterate the same contraction to a natural residual of 1e-12; the impulses then
differ by at most the residual over the contraction's gap, 1e-9 as in test_bncp_gpu.py."""
import importlib

import numpy as np
import pytest

from conftest import cuda_ok

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]


@pytest.fixture(scope="module")
def bn(me):
    return importlib.import_module("motion_engine_b200.bncp")


def _problems(B, nc, seed):
    rng = np.random.default_rng(seed)
    n, nv = 3 * nc, 3 * nc + 6
    J = rng.normal(size=(B, n, nv))
    G = J @ J.transpose(0, 2, 1) / nv
    v = rng.normal(size=(B, nv)) * 0.3
    b = (J @ v[..., None])[..., 0]
    b[:, 0::3] -= 0.3
    return G, b, rng.uniform(0.2, 0.8, (B, nc))


@pytest.mark.parametrize("nc,B", [(1, 33), (2, 17), (3, 9), (4, 9), (5, 5), (7, 5), (8, 5), (9, 3), (16, 3)])
def test_every_layout_matches_the_oracle_and_its_padding(bn, oracle_mod, nc, B):
    import torch
    from oracle import oracle_bncp as OB
    G, b, mu = _problems(B, nc, nc)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    s = bn.BatchNCP(t(G), t(b), t(mu))
    lam = s.solve(20000, 1e-12).cpu().numpy()
    res = s.res.cpu().numpy()
    assert (s.iters.cpu().numpy() < 20000).all() and (res < 1e-12).all()
    for e in (0, B - 1):
        ref, _ = OB.pgs(G[e], b[e], mu[e], 20000, 1e-14)
        assert np.max(np.abs(lam[e] - ref)) < 1e-9, e
    gb, gmu = (x.cpu().numpy() for x in s.vjp(t(np.ones((B, 3 * nc)))))
    for wide in {min(nc + 1, 16), 8, 9, 16} - set(range(nc + 1)):
        Gw, bw, mw = np.zeros((B, 3 * wide, 3 * wide)), np.zeros((B, 3 * wide)), np.zeros((B, wide))
        Gw[:, :3 * nc, :3 * nc], bw[:, :3 * nc], mw[:, :nc] = G, b, mu
        q = bn.BatchNCP(t(Gw), t(bw), t(mw), torch.full((B,), nc, dtype=torch.int32))
        lw = q.solve(20000, 1e-12).cpu().numpy()
        assert lw[:, :3 * nc].tobytes() == lam.tobytes() and not lw[:, 3 * nc:].any()
        assert q.res.cpu().numpy().tobytes() == res.tobytes() and bool((q.iters == s.iters).all())
        gw, mwv = (x.cpu().numpy() for x in q.vjp(t(np.ones((B, 3 * wide)))))
        assert np.array_equal(gw[:, :3 * nc], gb, equal_nan=True) and np.array_equal(mwv[:, :nc], gmu, equal_nan=True)


def test_warm_start_iteration_limit_and_unchecked_solve(bn):
    import torch
    G, b, mu = _problems(11, 4, 1)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    s = bn.BatchNCP(t(G), t(b), t(mu))
    half = s.solve(7, 1e-12, check=0).clone()
    assert bool((s.iters == 7).all()) and bool((s.res > 0).all())
    both = s.solve(14, 1e-12, check=0).clone()
    assert torch.equal(s.solve(7, 1e-12, check=0, warm=half), both)
    s.solve(0, 1e-12, warm=both)
    assert bool((s.iters == 0).all()) and torch.equal(s.lam, both)
