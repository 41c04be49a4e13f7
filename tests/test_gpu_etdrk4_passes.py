"""ETDRK4 on grids of several axes, whose passes hold a stage's transforms along one
axis together with its spectral or real part, against the oracle: the smallest and
largest lines, tiles of one line and of many, uneven lines; and both chains of a
solve, whose blocks change at different steps, against two updaters' solves."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ps():
    oracle.build()
    import polystring_b200
    return polystring_b200


@pytest.mark.parametrize("shape", [(64, 32, 1), (8, 352, 1), (352, 8, 1), (128, 96, 1), (2, 2, 2), (4, 2, 192), (256, 4, 2),
                                   (12, 24, 48), (48, 32, 16), (32, 32, 32)])
def test_updater_matches_oracle(ps, shape):
    dim = 2 if shape[2] == 1 else 3
    L = (3.9, 4.4, 4.1)[:dim]
    rng = np.random.default_rng(6)
    w = 0.5 * rng.standard_normal(shape)
    qs = np.zeros((14,) + shape)
    qs[0] = 1.0 + 0.2 * rng.standard_normal(shape)
    cell = ps.make_cell(dim, ("RECTANGULAR", "ORTHORHOMBIC")[dim - 2], *L)
    ref = oracle.Updater("ETDRK4", oracle.k2_orthogonal(dim, L, shape), shape, 0.01).solve(w, qs.copy())
    out = ps.Etdrk4_PBC(cell, *shape, 0.01).solve(qs.copy(), w)
    # 13 steps of 8 transforms, each a few eps of the largest value
    assert np.abs(out - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("shape", [(96, 64, 1), (16, 24, 32)])
def test_chains_match_updaters(ps, shape):
    dim = 2 if shape[2] == 1 else 3
    rng = np.random.default_rng(7)
    wA, wB = 0.5 * rng.standard_normal((2,) + shape)
    cell = ps.make_cell(dim, ("RECTANGULAR", "ORTHORHOMBIC")[dim - 2], *(3.9, 4.4, 4.1)[:dim])
    LA, LB = 8, 12
    m = ps.ModelAB(dim, shape, cell, (LA + 1, LB + 1), 18.0, mde="ETDRK4")
    m.set_fields(wA, wB)
    m.update(1)
    up = ps.Etdrk4_PBC(cell, *shape, 1.0 / (LA + LB))
    def run(first, n1, second, n2):
        a = np.ones((n1 + 1,) + shape)
        up.solve(a, first)
        b = np.empty((n2 + 1,) + shape)
        b[0] = a[-1]
        up.solve(b, second)
        return b
    # 20 steps of 8 transforms, each a few eps of the largest value
    for got, ref in ((m.get("qB"), run(wA, LA, wB, LB)), (m.get("qAc"), run(wB, LB, wA, LA))):
        got = got.reshape((-1,) + shape)
        assert np.abs(got[-1] - ref[-1]).max() < 1e-12 * np.abs(ref[-1]).max()
