"""The 1D and 2D sweeps at the edges of their line lengths (orbits and output
tiles not full, lines not a multiple of eight, the longest of each) against the
oracle's propagators; 2D solves in a batch and a string against single ones."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ps():
    oracle.build()
    import polystring_b200
    return polystring_b200


SHAPES = [(n, 1, 1) for n in (4, 8, 12, 24, 48, 64, 96, 128, 192, 256, 352)] + \
    [(4, 8, 1), (12, 64, 1), (64, 4, 1), (24, 48, 1), (16, 12, 1), (64, 64, 1)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("scheme", ["RQM4", "OS2"])
def test_every_line_length_matches_oracle(ps, shape, scheme):
    dim = 1 if shape[1] == 1 else 2
    L = (3.7, 4.1)[:dim]
    rng = np.random.default_rng(12)
    ds = 0.01
    w = 0.5 * rng.standard_normal(shape)
    qs = np.zeros((14,) + shape)
    qs[0] = 1.0 + 0.2 * rng.standard_normal(shape)
    cell = ps.make_cell(dim, ("LAMELLAR", "RECTANGULAR")[dim - 1], *L)
    g, l = oracle.unit_cell(dim, cell.system, *L)
    if scheme == "RQM4":
        ref = oracle.Updater("RQM4", oracle.k2_orthogonal(dim, l, shape), shape, ds).solve(w, qs.copy())
        up = ps.RQM4(cell, *shape, ds)
    else:
        ref = oracle.Updater("OS2", oracle.k_laplacian(g, shape, ds), shape, ds).solve(w, qs.copy())
        up = ps.PseudoSpectral(cell, *shape, ds)
    out = up.solve(qs.copy(), w)
    # 13 steps of at most 8 line operators, each a few eps of the largest value
    assert np.abs(out - ref).max() < 1e-12 * np.abs(ref).max()


def test_batch_and_string_members_equal_single_solves(ps):
    shape, cell = (48, 32, 1), ps.make_cell(2, "RECTANGULAR", 4.1, 3.6)
    spec = lambda k: dict(dim=2, shape=shape, cell=cell, Ms=(9 + 2 * k, 13), chiN=17.0)
    n = 4
    rng = np.random.default_rng(5)
    fields = [0.5 * rng.uniform(-1, 1, (2,) + shape) for _ in range(n)]
    b = ps.BatchAB([spec(k) for k in range(n)])
    for k in range(n):
        b.set_fields(k, *fields[k])
    b.update(2)
    for k in range(n):
        m = ps.ModelAB(**spec(k))
        m.set_fields(*fields[k])
        m.update(2)
        assert b.H(k) == m.H()
        assert np.array_equal(b.get(k, "qAc"), m.get("qAc")) and np.array_equal(b.get(k, "wA"), m.get("wA"))
    g = ps.StringAB(n, 2, shape, cell, (9, 13), 17.0, max_iter=2)
    g.set_images(np.stack([f[0] for f in fields]), np.stack([f[1] for f in fields]))
    g.iterate(1)
    phi = g.get("phiA")
    for k in range(n):
        m = ps.ModelAB(2, shape, cell, (9, 13), 17.0)
        m.set_fields(*fields[k])
        m.update(2)
        assert np.array_equal(phi[k], m.get("phiA")), k
