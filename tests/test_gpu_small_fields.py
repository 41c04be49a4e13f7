"""Q and the densities on both sides of the sizes where their launches change (fields
of up to 1024 points reduced by one block, densities of grids below 32768 points in
one launch) against the contour sums of the returned propagators."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 1, 1), (256, 1, 1), (32, 32, 1), (48, 24, 1), (16, 16, 4), (16, 16, 24),
                                   (32, 32, 24), (32, 32, 32)])
@pytest.mark.parametrize("blocks", [2, 3])
def test_Q_and_densities(shape, blocks):
    import polystring_b200 as ps
    dim = 1 if shape[1] == 1 else 2 if shape[2] == 1 else 3
    cell = ps.make_cell(dim, ("LAMELLAR", "RECTANGULAR", "ORTHORHOMBIC")[dim - 1], *(3.9, 4.4, 4.1)[:dim])
    w = 0.5 * np.random.default_rng(2).standard_normal((3,) + shape)
    if blocks == 2:
        m = ps.ModelAB(dim, shape, cell, (9, 13), 18.0)
        m.set_fields(w[0], w[1])
        m.update(1)
        # Simpson's weights of 8 and 12 intervals, ds = 1 / 20
        for L, q, qc, phi in ((8, "qA", "qAc", "phiA"), (12, "qB", "qBc", "phiB")):
            c = np.ones(L + 1)
            c[1:-1:2], c[2:-1:2] = 4.0, 2.0
            a, b = m.get(q), m.get(qc)
            ref = np.tensordot(c / 3.0, a * b[::-1], 1) / 20.0 / m.Q()
            # sums of 13 products: a few eps of the largest value each
            assert np.abs(m.get(phi) - ref).max() < 1e-14 * 50 * np.abs(ref).max()
        Q = m.get("qB")[-1].mean()
        assert abs(m.Q() - Q) < 1e-13 * Q
    else:
        m = ps.ModelABC(dim, shape, cell, (9, 13, 7), (18.0, 20.0, 22.0))
        m.set_fields(*w)
        m.update(1)
        total = sum(m.get("phi" + x).mean() for x in "ABC")
        # every block's contour integral of a constant, exact under Simpson's rule up
        # to its error at ds = 1 / 26 (1e-4 of the integrand's variation)
        assert abs(total - 1.0) < 1e-3
