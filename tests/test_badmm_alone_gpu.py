"""A problem of the batched ADMM alone = the same problem among others, bit for bit, where a warp's
problems do not take equally many Jacobi rotations: Delassus matrices with eigenvalues that occur
several times, stances without leg joints (rank 6) and random ones, side by side.  Bits: no
tolerance."""
import numpy as np
import pytest

from test_badmm_gpu import _badmm

pytestmark = pytest.mark.gpu
DT = 1 / 240


def _mixed(B, nc, nv, seed):
    from importlib import import_module
    import __graft_entry__ as ge
    ge.load_package()
    J, Minv, v, mu = import_module("motion_engine_b200.scenes").stance_batch(B=B, nv=nv, nc=nc, mu=0.5, seed=seed)
    rng = np.random.default_rng(seed)
    n = 3 * nc
    for e in range(B):
        if e % 3 == 0:  # G = Q diag(eigenvalues) Q^T, two or three distinct ones
            Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
            Minv[e] = np.eye(nv)
            Minv[e, :n, :n] = (Q * rng.choice(rng.uniform(0.1, 3.0, int(rng.integers(2, 4))), n)) @ Q.T
            Minv[e] = 0.5 * (Minv[e] + Minv[e].T)
            J[e] = np.eye(n, nv)
        elif e % 3 == 1:
            J[e, :, 6:] = 0.0
    return J, Minv, v, mu


@pytest.mark.parametrize("mode", ["sqrt", "regime"])
@pytest.mark.parametrize("nc,nv,B", [(1, 9, 288), (2, 12, 288), (4, 18, 384), (5, 21, 96)])
def test_a_problem_alone_has_its_bits_of_the_batch(nc, nv, B, mode):
    P = _mixed(B, nc, nv, 100 + nc)
    names = ("rho", "lam", "v_plus", "dlam_tau", "dv_tau", "dlam_mu")

    def solve(J, Minv, v, mu):
        s = _badmm().BatchProxADMM(len(v), nv, nc).upload(J, Minv, v, mu, DT).set_rho(mode)
        s.step_and_grad(20, 8, 4, 1e-8, n_calls=nc + 2, grad_cg=60)
        return [getattr(s, k).cpu().numpy() for k in names]

    batch = solve(*P)
    differ = {}
    for e in range(B):
        for k, one, all_ in zip(names, solve(*(a[e:e + 1] for a in P)), batch):
            if one[0].tobytes() != all_[e].tobytes():
                differ.setdefault(k, []).append(e)
    assert not differ, {k: len(v) for k, v in differ.items()}
