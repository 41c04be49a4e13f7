"""Which form of a solve runs is settled when its context is made: the switch of the
line passes afterwards changes nothing, for every scheme and context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mde", ["RQM4", "OS2", "ETDRK4"])
@pytest.mark.parametrize("made", ["0", "1"])
def test_settled_at_construction(monkeypatch, mde, made):
    import polystring_b200 as ps
    shape, cell = (32, 48, 1), ps.make_cell(2, "RECTANGULAR", 3.9, 4.4)
    w = np.random.default_rng(4).uniform(-1, 1, (2,) + shape)
    up = {"RQM4": ps.RQM4, "OS2": ps.PseudoSpectral, "ETDRK4": ps.Etdrk4_PBC}[mde]
    out = []
    for later in (made, "10"[int(made)]):
        monkeypatch.setenv("PS_B200_LINE_PASSES", made)
        m, u = ps.ModelAB(2, shape, cell, (9, 13), 18.0, mde=mde), up(cell, *shape, 0.02)
        monkeypatch.setenv("PS_B200_LINE_PASSES", later)
        m.set_fields(*w)
        m.update(2)
        qs = np.ones((7,) + shape)
        out.append((m.H(), m.get("qB"), u.solve(qs, w[0])))
        assert (m.launches_per_propagate() == 1) == (made == "0")
    for a, b in zip(*out):
        assert np.array_equal(a, b)
