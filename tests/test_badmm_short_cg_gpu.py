"""The batched ADMM's gradient after few CG steps, where a solve is not linear in its right-hand side
and the columns of the slip map depend on the direction, and on both sides of the step count from
which the directions share them (6 a contact): the oracle's gradient to 1e-9 of each output's
scale, the bar of test_badmm_gpu.py.  At these steps the oracle with its product summed in another
order moves by less than 5e-12."""
import numpy as np
import pytest

from test_badmm_gpu import _badmm
from test_badmm_lanes_gpu import _close, _problems

pytestmark = pytest.mark.gpu
DT = 1 / 240


@pytest.mark.parametrize("nc,per_leg,cg", [(1, 3, 1), (2, 3, 2), (2, 3, 11), (2, 3, 12), (4, 3, 3), (4, 3, 4), (4, 3, 23),
                                           (4, 3, 24), (5, 3, 4), (5, 3, 29), (8, 3, 5), (8, 3, 47), (8, 3, 48)])
def test_gradient_after_few_steps_matches_the_oracle(nc, per_leg, cg):
    from oracle.oracle_badmm import BatchADMMOracle
    J, Minv, v, mu = _problems(9, nc, per_leg, 60 + nc)
    o = BatchADMMOracle(J, Minv, v, mu, DT).set_rho("regime").forward(60, 8, 4, 1e-8)
    o.gradient(n_calls=nc + 2, grad_cg=cg)
    s = _badmm().BatchProxADMM(9, v.shape[1], nc).upload(J, Minv, v, mu, DT).set_rho("regime")
    s.step_and_grad(60, 8, 4, 1e-8, n_calls=nc + 2, grad_cg=cg)
    assert np.array_equal(s.labels.cpu().numpy(), o.labels)
    for name in ("dlam_tau", "dv_tau", "dlam_mu"):
        _close(getattr(s, name), getattr(o, name), name)
    # one direction given by the caller
    db = np.random.default_rng(nc).standard_normal((9, nc, 3))
    got = s.grad_given(o.lam, o.u, db, n_calls=nc + 2, cg=cg)
    ref = o.grad_db(o.lam, o.u, db, n_calls=nc + 2, cg=cg)
    assert np.abs(got - ref).max() <= 1e-9 * max(1.0, np.abs(ref).max())
