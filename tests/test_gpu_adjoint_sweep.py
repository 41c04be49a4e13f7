"""The adjoint on the persistent sweeps against the one on line passes: the same
discrete derivative, at line lengths whose orbits and tiles are not full, one
block much longer than the other, and chunks of steps that end unevenly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ps():
    import polystring_b200
    return polystring_b200


CASES = [(2, (24, 48, 1), (3.9, 4.3), (8, 30)), (2, (64, 12, 1), (4.9, 4.3), (33, 17)), (2, (8, 8, 1), (3.9, 4.3), (18, 9)),
         (3, (24, 12, 16), (3.8, 4.0, 4.2), (9, 34)), (3, (8, 48, 32), (3.8, 4.0, 4.2), (17, 18)),
         (3, (96, 8, 12), (5.8, 4.0, 4.2), (13, 21))]


@pytest.mark.parametrize("dim,shape,L,Ms", CASES)
def test_gradient_and_stress_match_line_passes(ps, monkeypatch, dim, shape, L, Ms):
    rng = np.random.default_rng(21)
    wA, wB = rng.uniform(-1, 1, (2,) + shape)
    a, b = rng.standard_normal((2,) + shape)
    cell = ps.make_cell(dim, ("RECTANGULAR", "ORTHORHOMBIC")[dim - 2], *L)
    out = []
    for line_passes in ("0", "1"):
        monkeypatch.setenv("PS_B200_LINE_PASSES", line_passes)
        m = ps.ModelAB(dim, shape, cell, Ms, 18.0)
        m.set_fields(wA, wB)
        gA, gB = m.grad_w(a, b, 0.7)
        s = m.stress()
        # twice on one model: nothing of a call is left for the next
        assert np.array_equal(m.grad_w(a, b, 0.7)[0], gA) and np.array_equal(m.stress(), s)
        out.append((gA, gB, s, m.get("phiA"), m.Q()))
    (gA, gB, s, phi, Q), (lA, lB, ls, lphi, lQ) = out
    # both forms sum about 2 Ns terms a point, each with some 50 roundings of
    # values up to the largest term; the largest terms exceed their sum by less
    # than 1e2 here: 1e2 x 80 x 50 eps < 1e-10
    assert np.abs(gA - lA).max() < 1e-10 * np.abs(lA).max() and np.abs(gB - lB).max() < 1e-10 * np.abs(lB).max()
    assert np.abs(s - ls).max() < 1e-10 * np.abs(ls).max()
    assert np.abs(phi - lphi).max() < 1e-12 and abs(Q - lQ) < 1e-12 * abs(lQ)
