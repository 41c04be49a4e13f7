"""2D sweeps in tiles of lines over many CTAs, at the edges of their line lengths
(orbits and output tiles not full, partial tiles of lines, fragments and parts,
long rows in parts and whole) against the oracle's propagators; batch members
against single solves; the adjoint against the line passes."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ps():
    oracle.build()
    import polystring_b200
    return polystring_b200


SHAPES = [(64, 64), (48, 64), (64, 96), (96, 12), (12, 128), (128, 128), (192, 4), (4, 192), (24, 256), (256, 8),
          (12, 352), (352, 12), (352, 256)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("scheme", ["RQM4", "OS2"])
def test_every_line_length_matches_oracle(ps, shape, scheme):
    shape, L = shape + (1,), (3.7, 4.1)
    rng = np.random.default_rng(12)
    ds = 0.01
    w = 0.5 * rng.standard_normal(shape)
    qs = np.zeros((14,) + shape)
    qs[0] = 1.0 + 0.2 * rng.standard_normal(shape)
    cell = ps.make_cell(2, "RECTANGULAR", *L)
    g, l = oracle.unit_cell(2, cell.system, *L)
    if scheme == "RQM4":
        ref = oracle.Updater("RQM4", oracle.k2_orthogonal(2, l, shape), shape, ds).solve(w, qs.copy())
        up = ps.RQM4(cell, *shape, ds)
    else:
        ref = oracle.Updater("OS2", oracle.k_laplacian(g, shape, ds), shape, ds).solve(w, qs.copy())
        up = ps.PseudoSpectral(cell, *shape, ds)
    out = up.solve(qs.copy(), w)
    # 13 steps of at most 8 line operators, each a few eps of the largest value
    assert np.abs(out - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("extra", [0, 12])   # solves up to 64 x 64: with clusters for all of them, and with more
def test_batch_members_equal_single_solves(ps, extra):
    shapes = [(64, 64, 1), (96, 128, 1), (128, 128, 1), (96, 16, 1), (128, 128, 1), (128, 64, 1), (48, 64, 1)]
    shapes += extra * [(64, 64, 1)]
    specs = [dict(dim=2, shape=s, cell=ps.make_cell(2, "RECTANGULAR", 4.1, 3.6), Ms=(9 + 2 * (k % 3), 13), chiN=17.0)
             for k, s in enumerate(shapes)]
    rng = np.random.default_rng(5)
    fields = [0.5 * rng.uniform(-1, 1, (2,) + s) for s in shapes]
    b = ps.BatchAB(specs)
    for k in range(len(specs)):
        b.set_fields(k, *fields[k])
    b.update(2)
    for k, spec in enumerate(specs):
        m = ps.ModelAB(**spec)
        m.set_fields(*fields[k])
        m.update(2)
        assert b.H(k) == m.H()
        assert np.array_equal(b.get(k, "qAc"), m.get("qAc")) and np.array_equal(b.get(k, "wA"), m.get("wA"))


@pytest.mark.parametrize("shape", [(64, 64, 1), (12, 96, 1), (16, 256, 1), (256, 12, 1)])
def test_adjoint_matches_line_passes(ps, shape, monkeypatch):
    rng = np.random.default_rng(3)
    w = 0.5 * rng.standard_normal((2,) + shape)
    bar = rng.standard_normal((2,) + shape)
    out = []
    for lines in ("0", "1"):
        monkeypatch.setenv("PS_B200_LINE_PASSES", lines)
        m = ps.ModelAB(2, shape, ps.make_cell(2, "RECTANGULAR", 4.1, 3.6), (13, 21), 16.0)
        m.set_fields(*w)
        out.append(m.grad_w(bar[0], bar[1], 0.3) + (m.stress(),))
        del m
    # both sum about 2 Ns = 64 terms a point, each with some 50 roundings of values up
    # to the largest term, which exceeds the sum by less than 1e2: 1e2 x 64 x 50 eps < 1e-10
    for a, b in zip(*out):
        assert np.abs(a - b).max() < 1e-10 * np.abs(b).max()


@pytest.mark.parametrize("shape,mde", [((96, 64, 1), "RQM4"), ((12, 128, 1), "RQM4"), ((128, 96, 1), "OS2")])
def test_string_images_equal_single_solves(ps, shape, mde):
    n, cell = 5, ps.make_cell(2, "RECTANGULAR", 4.1, 3.6)
    fields = 0.5 * np.random.default_rng(8).uniform(-1, 1, (2, n) + shape)
    g = ps.StringAB(n, 2, shape, cell, (9, 13), 17.0, max_iter=2, mde=mde)
    assert g.launches_per_iteration() < 30
    g.set_images(*fields)
    g.iterate(1)
    phi = g.get("phiA")
    for k in range(n):
        m = ps.ModelAB(2, shape, cell, (9, 13), 17.0, mde=mde)
        m.set_fields(fields[0, k], fields[1, k])
        m.update(2)
        assert np.array_equal(phi[k], m.get("phiA")), k
