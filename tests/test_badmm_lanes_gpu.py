"""The batched ADMM at every contact count (one lane a contact: 1, 2, 4 or 8 lanes a problem, 32 to
4 problems a warp), on batches that leave a warp's last problems empty, against the ADMM oracle;
and G's spectrum, whose Jacobi rotations run in stages, where few sweeps are asked for.

The bar is the one the batched ADMM has in test_badmm_gpu.py: 1e-9 of each output's scale (the
two sum in another order).  The penalty is the spectrum's: rotations equal but for rounding, so
1e-10 of it."""
import numpy as np
import pytest

from test_badmm_gpu import _badmm

pytestmark = pytest.mark.gpu


def _problems(B, nc, per_leg, seed):
    from importlib import import_module
    import __graft_entry__ as ge
    ge.load_package()
    return import_module("motion_engine_b200.scenes").stance_batch(B=B, nv=6 + nc * per_leg, nc=nc, mu=0.5, seed=seed)


def _close(got, ref, what):
    got = got.cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-9 * max(1.0, np.abs(ref).max()), what


@pytest.mark.parametrize("nc,per_leg,B", [(1, 3, 33), (2, 4, 17), (3, 3, 9), (4, 4, 9), (5, 3, 5), (6, 4, 5),
                                          (7, 3, 3), (8, 3, 5)])
def test_every_contact_count_matches_the_oracle(nc, per_leg, B):
    from oracle.oracle_badmm import BatchADMMOracle
    J, Minv, v, mu = _problems(B, nc, per_leg, 20 + nc)
    s = _badmm().BatchProxADMM(B, v.shape[1], nc).upload(J, Minv, v, mu, 1 / 240).set_rho("regime")
    s.step_and_grad(60, 8, 4, 1e-8, n_calls=nc + 2, grad_cg=60, jdir=1)
    o = BatchADMMOracle(J, Minv, v, mu, 1 / 240).set_rho("regime").forward(60, 8, 4, 1e-8)
    o.gradient(n_calls=nc + 2, grad_cg=60, jdir=1)
    assert np.allclose(s.rho.cpu().numpy(), o.rho, rtol=1e-10, atol=0)
    assert np.array_equal(s.labels.cpu().numpy(), o.labels) and np.array_equal(s.mask.cpu().numpy(), o.mask)
    for name in ("lam", "u", "v_plus:vplus", "dlam_tau", "dv_tau", "dlam_mu"):
        mine, _, theirs = name.partition(":")
        _close(getattr(s, mine), getattr(o, theirs or mine), name)


@pytest.mark.parametrize("sweeps", [1, 2, 10])
@pytest.mark.parametrize("nc", [1, 2, 3, 4])
def test_few_jacobi_sweeps_give_the_cyclic_order_s_eigenvalues(nc, sweeps):
    from oracle.oracle_badmm import BatchADMMOracle
    J, Minv, v, mu = _problems(6, nc, 3, 40 + nc)
    s = _badmm().BatchProxADMM(6, v.shape[1], nc).upload(J, Minv, v, mu, 1 / 240, jacobi_sweeps=sweeps).set_rho("sqrt")
    s.forward(n_iter=4, chunk=4)
    o = BatchADMMOracle(J, Minv, v, mu, 1 / 240, jacobi_sweeps=sweeps).set_rho("sqrt")
    assert np.allclose(s.rho.cpu().numpy(), o.rho, rtol=1e-10, atol=0)


def test_one_direction_alone_and_a_frozen_batch():
    """do_mu=False leaves dlam_mu zero and dlam_tau as it is with it; a batch that converges early
    keeps, at every later iteration, the outputs it froze with."""
    J, Minv, v, mu = _problems(9, 4, 3, 3)
    outs = []
    for do_mu in (True, False):
        s = _badmm().BatchProxADMM(9, 18, 4).upload(J, Minv, v, mu, 1 / 240).set_rho("regime")
        s.step_and_grad(80, 8, 4, 1e-8, n_calls=6, grad_cg=60, do_mu=do_mu)
        outs.append((s.dlam_tau.cpu().numpy(), s.dlam_mu.cpu().numpy()))
    assert np.abs(outs[0][0] - outs[1][0]).max() <= 1e-12 * max(1.0, np.abs(outs[0][0]).max())
    assert not outs[1][1].any() and outs[0][1].any()
    s = _badmm().BatchProxADMM(9, 18, 4).upload(J, Minv, v, mu, 1 / 240).set_rho("regime")
    a = s.forward(n_iter=400, tol=1e-3, chunk=400)
    b = s.forward(n_iter=800, tol=1e-3, chunk=800)
    assert a.n_active == 0 and a.lam.tobytes() == b.lam.tobytes() and a.resenv.tobytes() == b.resenv.tobytes()
