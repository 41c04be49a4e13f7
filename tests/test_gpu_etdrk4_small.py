"""ETDRK4 solves that run in one CTA (1D and 2D grids up to 1536 points) at the
edges of their kernels' ranges, both chains, against the line passes: the same
operations on the same values, other radix schedules."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ps():
    import polystring_b200
    return polystring_b200


@pytest.mark.parametrize("shape", [(2, 1, 1), (64, 1, 1), (128, 1, 1), (352, 1, 1), (2, 2, 1), (12, 24, 1), (32, 32, 1),
                                   (48, 24, 1), (128, 12, 1), (32, 48, 1)])
def test_small_grids_match_line_passes(ps, monkeypatch, shape):
    dim = 1 if shape[1] == 1 else 2
    rng = np.random.default_rng(4)
    wA, wB = rng.uniform(-1, 1, (2,) + shape)
    cell = ps.make_cell(dim, ("LAMELLAR", "RECTANGULAR")[dim - 1], *(3.9, 4.4)[:dim])
    out = []
    for line_passes in ("0", "1"):
        monkeypatch.setenv("PS_B200_LINE_PASSES", line_passes)
        m = ps.ModelAB(dim, shape, cell, (9, 13), 18.0, mde="ETDRK4")
        assert (m.launches_per_propagate() == 1) == (line_passes == "0")
        m.set_fields(wA, wB)
        m.update(2)
        up = ps.Etdrk4_PBC(cell, *shape, 0.02)
        qs = np.ones((7,) + shape)
        up.solve(qs, wA)
        out.append((m.get("qB"), m.get("qAc"), m.get("wA"), qs))
    for a, b in zip(*out):
        # 20 steps of 8 transforms, each a few eps of the largest value
        assert np.abs(a - b).max() < 1e-12 * np.abs(b).max()
