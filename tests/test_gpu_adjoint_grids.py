"""The adjoint by the number of axes longer than a point, whatever the cell's
dimension: one such axis is refused (the propagators still run), two or three agree with
the line passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ps():
    import polystring_b200
    return polystring_b200


def _model(ps, dim, shape):
    cell = ps.make_cell(dim, ("LAMELLAR", "RECTANGULAR", "ORTHORHOMBIC")[dim - 1], *(3.9, 4.3, 4.1)[:dim])
    w = np.random.default_rng(4).uniform(-1, 1, (2,) + shape)
    m = ps.ModelAB(dim, shape, cell, (9, 13), 18.0)
    m.set_fields(w[0], w[1])
    return m


@pytest.mark.parametrize("dim,shape", [(1, (64, 1, 1)), (2, (64, 1, 1)), (2, (1, 64, 1)), (3, (64, 1, 1)),
                                       (3, (352, 1, 1)), (3, (1, 1, 64))])
def test_one_long_axis_is_refused(ps, dim, shape):
    m = _model(ps, dim, shape)
    a, b = np.random.default_rng(5).standard_normal((2,) + shape)
    for call in (lambda: m.grad_w(a, b, 0.7), m.stress):
        with pytest.raises(ps.PSError) as e:
            call()
        assert e.value.code == -2 and "2D or 3D grid" in str(e.value)
    m.update(2)
    # the refused calls leave the model as it was
    n = _model(ps, dim, shape)
    n.update(2)
    assert m.H() == n.H() and np.array_equal(m.get("phiA"), n.get("phiA"))


@pytest.mark.parametrize("shape", [(24, 16, 1), (96, 16, 1), (16, 1, 24), (1, 24, 16), (8, 12, 16)])
def test_two_and_three_long_axes_in_a_3d_cell(ps, monkeypatch, shape):
    a, b = np.random.default_rng(5).standard_normal((2,) + shape)
    out = []
    for line_passes in ("0", "1"):
        monkeypatch.setenv("PS_B200_LINE_PASSES", line_passes)
        m = _model(ps, 3, shape)
        out.append((*m.grad_w(a, b, 0.7), m.stress()))
    # sums of some 2 Ns = 40 terms a point with 50 roundings each, the largest term less
    # than 1e2 times the sum: 1e2 x 40 x 50 eps < 1e-10
    for x, y in zip(*out):
        assert np.abs(x - y).max() < 1e-10 * np.abs(y).max()
