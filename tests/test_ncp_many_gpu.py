"""The exact-cone sweeps where a CTA takes many rounds of contacts a colour (the kernel with more
groups a CTA), with soft steps and without the de Saxce term, and the reverse sweeps at the final
iterate on both sides of the lines between one CTA, cluster and grid: every form has the bits of
every other."""
import importlib

import numpy as np
import pytest

from conftest import cuda_ok
from test_ncp_forms_gpu import _lattice

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]


@pytest.fixture(scope="module")
def ncp(me):
    return importlib.import_module("motion_engine_b200.ncp")


@pytest.mark.parametrize("desaxce,soft", [(True, True), (False, False), (False, True)])
@pytest.mark.parametrize("dtype,n", [("float64", 119), ("float64", 121), ("float64", 500), ("float32", 359), ("float32", 361),
                                     ("float32", 900)])
def test_many_rounds_have_the_bits_of_the_automatic_form(ncp, dtype, n, desaxce, soft):
    bs = _lattice(ncp, n)
    if soft:
        bs.sep = np.where(np.arange(bs.n_c) % 3 == 0, 1e-3, -2e-3)
    p = ncp.SoftStep().params(1 / 240) if soft else None
    ref = None
    for form in (0, 1, -2, 2, 148):
        s = ncp.NCPSolverB200(bs.n_b, bs.n_c, dtype=dtype, solve_blocks=form, desaxce=desaxce)
        r = s.solve(bs, iters=6, measure_residual=False, soft=p)
        out = (r.lam.tobytes(), r.v.tobytes())
        ref = ref or out
        assert out == ref, form


@pytest.mark.parametrize("n", [1, 8, 198, 202, 2390, 2410])
def test_the_implicit_adjoint_agrees_between_forms(ncp, n):
    bs = _lattice(ncp, n)
    g = np.random.default_rng(2).normal(size=(bs.n_c, 3))
    ref = None
    for form in (0, 1, -2, -16, 37):
        s = ncp.NCPSolverB200(bs.n_b, bs.n_c, dtype="float64", solve_blocks=form)
        s.solve(bs, iters=6)
        d = s.vjp_implicit(g, 4)
        ref = ref or d
        for k in ref:
            assert d[k].tobytes() == ref[k].tobytes(), (form, k)
