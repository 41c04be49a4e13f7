"""The 3D sweep on real line operators at the edges of its line lengths (every
length, orbits and output tiles not full, columns and rows not a multiple of
eight, more slabs than CTAs) against the oracle's propagators, and shared
launches against single ones."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ps():
    oracle.build()
    import polystring_b200
    return polystring_b200


SHAPES = [(4, 4, 8), (8, 12, 4), (12, 4, 12), (24, 8, 16), (16, 48, 24), (8, 64, 32), (64, 24, 48),
          (96, 12, 32), (4, 96, 12), (12, 8, 96), (128, 4, 8), (4, 128, 12), (8, 4, 128)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("scheme", ["RQM4", "OS2"])
def test_every_line_length_matches_oracle(ps, shape, scheme):
    L = (3.7, 4.1, 4.6)
    rng = np.random.default_rng(11)
    ds = 0.01
    w = 0.5 * rng.standard_normal(shape)
    qs = np.zeros((14,) + shape)
    qs[0] = 1.0 + 0.2 * rng.standard_normal(shape)
    cell = ps.make_cell(3, "ORTHORHOMBIC", *L)
    g, l = oracle.unit_cell(3, cell.system, *L)
    if scheme == "RQM4":
        ref = oracle.Updater("RQM4", oracle.k2_orthogonal(3, l, shape), shape, ds).solve(w, qs.copy())
        up = ps.RQM4(cell, *shape, ds)
    else:
        ref = oracle.Updater("OS2", oracle.k_laplacian(g, shape, ds), shape, ds).solve(w, qs.copy())
        up = ps.PseudoSpectral(cell, *shape, ds)
    out = up.solve(qs.copy(), w)
    # 13 steps of at most 12 line operators, each a few eps of the largest value
    assert np.abs(out - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("shape", [(24, 16, 32), (64, 16, 12), (96, 16, 24)])
def test_shared_launches_equal_single_ones(ps, monkeypatch, shape):
    """Solves of one shape with different Ns, cells and fields share launches
    with few CTAs each; results do not depend on the spread over CTAs."""
    if 12 in shape:
        shape = (64, 16, 16)
    spec = lambda k: dict(dim=3, shape=shape, cell=ps.make_cell(3, "ORTHORHOMBIC", 3.8, 4.0 + 0.1 * k, 4.2),
                          Ms=(7 + 2 * k, 9), chiN=18.0, scft="Anderson" if k % 2 else "EM", n_anderson=3)
    n = 7
    b = ps.BatchAB([spec(k) for k in range(n)])
    rng = np.random.default_rng(2)
    fields = [0.5 * rng.uniform(-1, 1, (2,) + shape) for _ in range(n)]
    for k in range(n):
        b.set_fields(k, *fields[k])
    b.update(3)
    for k in range(n):
        m = ps.ModelAB(**spec(k))
        m.set_fields(*fields[k])
        m.update(3)
        assert b.H(k) == m.H()
        for f in ("phiA", "wB", "qB", "qAc"):
            assert np.array_equal(b.get(k, f), m.get(f)), (k, f)
