"""The automatic form of the persistent pair solve where it launches cluster and grid and the
colouring decides (scenes of 3 400 boxes or 6 200 bead bodies on), and just below: the same bits
as the cluster and the grid asked for."""
import numpy as np
import pytest

from test_solve_forms_gpu import _bead

pytestmark = pytest.mark.gpu


def _packed(me, n):
    """Boxes side by side in a block of 15 by 15 columns: pairs in all three directions."""
    e = me.BoxContactEngine(mu=0.5, vit=6, pit=3)
    for i in range(n):
        z, r = divmod(i, 225)
        y, x = divmod(r, 15)
        e.add_box([0.3005 * x, 0.3005 * y, 0.1005 + 0.2005 * z], dims=(0.3, 0.3, 0.2), density=800.0)
    return e


@pytest.mark.parametrize("make,n,both,wide", [(_bead, 6190, False, False), (_bead, 6300, True, True),
                                              (_packed, 3390, False, False), (_packed, 3410, True, False)])
def test_automatic_form_gives_the_asked_forms_bits(me, make, n, both, wide):
    line, bodies = (3100, 6200) if make is _bead else (1700, 3400)
    out = []
    for form in (0, -16, 148):
        e = make(me, n)
        e.set_solve_blocks(form)
        for _ in range(3):
            e.step(1 / 240, 2)
        h = e.header_dict()
        assert h["error"] == 0 and (n >= bodies) == both and (n >= bodies and h["n_pairs"] >= line * h["n_colors"]) == wide
        out.append((e.get_state_packed().numpy().tobytes(), np.asarray(e.kept_contacts()["jn"]).tobytes()))
    assert out[0] == out[1] == out[2]
