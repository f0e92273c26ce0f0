"""b2c_box_candidates asked for alone: it leaves the contact slots of the last narrowphase as they
are, and its candidates are those of a whole substep over the same bodies, which keeps the
partners in those slots between count and emission.  Integers and bytes: no tolerance."""
import ctypes
import importlib

import pytest
import torch

from conftest import cuda_ok

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]


def _engine(me, n, scenes):
    sc = importlib.import_module("motion_engine_b200.scenes")
    if scenes > 1:
        return me.BatchedBoxEngine(sc.batched_scenes(n_scenes=scenes, nmin=n, nmax=2 * n, seed_mass=1, seed_boxes=2), mu=0.5)
    e = me.BoxContactEngine(mu=0.5)
    S = sc.random_boxes(n=n, box=(5.0, 5.0, 4.0))
    for c, d, m, de in zip(S["centers"], S["dims"], S["mu"], S["density"]):
        e.add_box(c, dims=d, density=de, mu=m)
    return e


@pytest.mark.parametrize("n,scenes", [(1, 1), (301, 1), (9, 7)])
def test_candidates_alone_keep_the_slots(me, n, scenes):
    e = _engine(me, n, scenes)
    for _ in range(120):
        e.step(1 / 240, 1)
    before = e.get_state_packed().clone()
    e.step(1 / 240, 1)
    torch.cuda.synchronize()
    keep = ("slot_p", "slot_n", "slot_f", "cont_count", "cont_offset", "pair_flag", "pair_offset")
    lists = ("cand_offset", "cand_a", "cand_b", "cand_count")
    slots = {k: e.bx_bufs[k].clone() for k in keep}
    cands = {k: e.bx_bufs[k].clone() for k in lists}
    e.set_state_packed(before)
    e.bx_bufs["cand_a"].fill_(-7)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    me._lib.check(e.L.b2c_box_candidates(ctypes.byref(e.c_bodies), ctypes.byref(e.c_boxes),
                                         ctypes.c_void_p(e.header.data_ptr()), stream), "b2c_box_candidates")
    torch.cuda.synchronize()
    m = int(cands["cand_offset"][e.N])
    assert (m > 0 or n == 1) and torch.equal(e.bx_bufs["cand_offset"], cands["cand_offset"])
    for k in ("cand_a", "cand_b"):
        assert torch.equal(e.bx_bufs[k][:m], cands[k][:m]), k
    for k in keep:
        assert torch.equal(e.bx_bufs[k], slots[k]), k
