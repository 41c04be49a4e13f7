"""The adjoint where the Boltzmann factors underflow or vanish (walls: w of 1e6, the
type's largest value, infinity) against the one on line passes, which forms no quotient of
them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wall", [4.0e4, 1.0e6, 1.7e308, np.inf])
@pytest.mark.parametrize("dim,shape", [(2, (32, 24, 1)), (2, (96, 16, 1)), (3, (16, 12, 24))])
def test_walls(monkeypatch, dim, shape, wall):
    import polystring_b200 as ps
    cell = ps.make_cell(dim, ("RECTANGULAR", "ORTHORHOMBIC")[dim - 2], *(3.9, 4.3, 4.1)[:dim])
    rng = np.random.default_rng(8)
    w = rng.uniform(-1, 1, (2,) + shape)
    w[:, :4] = wall      # e^{-w ds/4}, ds = 1 / 20: 7e-218 at 4e4, zero from there on
    w[1, 4:6] = wall     # and for one block only
    a, b = rng.standard_normal((2,) + shape)
    out = []
    for line_passes in ("0", "1"):
        monkeypatch.setenv("PS_B200_LINE_PASSES", line_passes)
        m = ps.ModelAB(dim, shape, cell, (9, 13), 18.0)
        m.set_fields(w[0], w[1])
        out.append((m.stress(), *m.grad_w(a, b, 0.7)))
    # as without walls: sums of some 40 terms with 50 roundings each, the largest term less
    # than 1e2 times the sum
    for x, y in zip(*out):
        assert np.isfinite(y).all()
        assert np.abs(x - y).max() < 1e-10 * np.abs(y).max()
