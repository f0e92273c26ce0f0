"""The automatic form of the persistent pair solve on both sides of its line (pairs a colour): the
same bits as the cluster and the grid asked for, on the bead engine and on the box engine."""
import numpy as np
import pytest

from conftest import lattice

pytestmark = pytest.mark.gpu


def _bead(me, n):
    e = me.ColorCacheContactEngine(dims=(0.3, 0.3, 0.2), mu=0.5, vit=6, pit=3)
    for c in lattice(n):
        e.add_body(c)
    return e


def _boxes(me, n):
    e = me.BoxContactEngine(mu=0.5, vit=6, pit=3)
    for c in lattice(n):  # 0.5 mm above the ground and each other: inside the margin from the start
        e.add_box([c[0], c[1], 0.1005 if c[2] < 0.2 else 0.301], dims=(0.3, 0.3, 0.2), density=800.0)
    return e


@pytest.mark.parametrize("make", [_bead, _boxes])
@pytest.mark.parametrize("n,wide", [(3300, False), (3500, True)])  # two layers: about n / 2 pairs a colour
def test_automatic_form_gives_the_asked_forms_bits(me, make, n, wide):
    out = []
    for form in (0, -16, 148):
        e = make(me, n)
        e.set_solve_blocks(form)
        for _ in range(4):
            e.step(1 / 240, 2)
        h = e.header_dict()
        assert h["error"] == 0 and (h["n_pairs"] >= 1700 * h["n_colors"]) == wide
        out.append((e.get_state_packed().numpy().tobytes(), np.asarray(e.kept_contacts()["jn"]).tobytes()))
    assert out[0] == out[1] == out[2]
