"""The exact-cone sweeps, their colouring and their reverse in every launch form (one CTA, a
cluster, a cooperative grid, and the automatic choice), at the sizes where a form changes how it
works: narrow and wide colours, more colours than a CTA's task table holds, more bodies than one
CTA keeps in shared memory, more contacts than the colouring keeps in registers.  Forms differ in
who updates a contact and never in the arithmetic, so impulses and velocities are equal bit for
bit, and equal to the oracle's where it is quick."""
import importlib

import numpy as np
import pytest

from conftest import cuda_ok

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]
FORMS = (0, 1, -4, -16, 37, 148)


@pytest.fixture(scope="module")
def ncp(me):
    return importlib.import_module("motion_engine_b200.ncp")


def _lattice(ncp, n, seed=0):
    d = importlib.import_module("motion_engine_b200.scenes").ncp_lattice(n=n)
    rng = np.random.default_rng(seed)
    d["v_free"] = d["v_free"] + rng.normal(0.0, 0.05, d["v_free"].shape)
    d["mu"] = rng.uniform(0.3, 0.8, d["mu"].shape)
    return ncp.BlockScene(**d)


def _hub(ncp, contacts, bodies):
    """`contacts` ground contacts of body 0 (a colour each), the other bodies one each while they last."""
    rng = np.random.default_rng(contacts)
    a = np.zeros(contacts, np.int32)
    a[::7] = 1 + np.arange(len(a[::7])) % max(bodies - 1, 1)
    r = rng.uniform(-0.3, 0.3, (contacts, 3))
    D = np.array([[0.0, 0.0, 1.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]])
    Ja = np.zeros((contacts, 3, 6))
    Ja[:, :, :3] = D
    Ja[:, :, 3:] = np.cross(r[:, None, :], D[None])
    Minv = np.zeros((bodies, 6, 6))
    Minv[:, np.arange(6), np.arange(6)] = [1, 1, 1, 8, 9, 10]
    vf = rng.normal(0.0, 0.1, (bodies, 6))
    vf[:, 2] -= 0.3
    return ncp.BlockScene(Ja=Ja, Jb=np.zeros_like(Ja), Minv=Minv, v_free=vf, mu=rng.uniform(0.2, 0.7, contacts),
                          body_pairs=np.stack([a, np.full(contacts, -1)], 1).astype(np.int32), dt=1 / 240,
                          bias=np.zeros((contacts, 3)), feature=np.arange(contacts, dtype=np.int32))


def _solve(ncp, bs, form, dtype, iters):
    s = ncp.NCPSolverB200(bs.n_b, bs.n_c, dtype=dtype, solve_blocks=form)
    r = s.solve(bs, iters=iters, measure_residual=False)
    again = s.solve(bs, iters=iters, measure_residual=False)  # through the colour cache
    assert again.cache_hit and again.lam.tobytes() == r.lam.tobytes()
    return r, s.coloring()[0]


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("scene", [("lattice", 1), ("lattice", 5), ("lattice", 6), ("lattice", 50), ("lattice", 700),
                                   ("hub", 210, 4), ("hub", 60, 3000)])
def test_every_form_matches_the_oracle(ncp, oracle_mod, scene, dtype):
    bs = _lattice(ncp, scene[1]) if scene[0] == "lattice" else _hub(ncp, *scene[1:])
    nt = np.float32 if dtype == "float32" else np.float64
    o = oracle_mod.ncp_solve(bs, 12, dtype=dtype)
    for form in FORMS:
        r, _ = _solve(ncp, bs, form, dtype, 12)
        assert r.n_colors == o["n_colors"], form
        assert np.array_equal(r.lam.astype(nt), o["lam"]) and np.array_equal(r.v.astype(nt), o["v"]), form


@pytest.mark.parametrize("n,dtype", [(1300, "float64"), (2100, "float32"), (17000, "float32")])
def test_wide_scenes_agree_between_forms(ncp, n, dtype):
    bs = _lattice(ncp, n)
    ref = None
    for form in (0, -16, 148):
        r, col = _solve(ncp, bs, form, dtype, 4)
        out = (r.lam.tobytes(), r.v.tobytes(), col.tobytes())
        ref = ref or out
        assert out == ref, form


@pytest.mark.parametrize("scene", [("lattice", 3), ("lattice", 40), ("lattice", 700), ("hub", 210, 4)])
def test_the_recorded_adjoint_agrees_between_forms(ncp, scene):
    """The same reverse updates in the same order; the sums over a contact's lanes are a fixed
    butterfly, so the forms agree to the last bits of the block adjoints' accumulation."""
    bs = _lattice(ncp, scene[1]) if scene[0] == "lattice" else _hub(ncp, *scene[1:])
    g = np.random.default_rng(1).normal(size=(bs.n_c, 3))
    ref = None
    for form in FORMS:
        d = ncp.NCPSolverB200(bs.n_b, bs.n_c, dtype="float64", solve_blocks=form).vjp_recorded(bs, g, 5)
        ref = ref or d
        for k in ref:
            assert np.abs(d[k] - ref[k]).max() <= 1e-13 * max(1.0, np.abs(ref[k]).max()), (form, k)
