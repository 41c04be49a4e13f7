"""A sweep that gives up at a grid barrier is reported by the calls that wait for its
results, and by the next iteration, until fields are set again.  PS_B200_BARRIER_GIVE_UP=1
lets a CTA give up as soon as it finds another one not yet there; every wait ends, and the
context stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ps():
    import polystring_b200
    return polystring_b200


GRIDS = [(3, (32, 16, 24), ("ORTHORHOMBIC", 3.9, 3.7, 4.1)), (2, (128, 192, 1), ("RECTANGULAR", 8.0, 11.0))]


def _fields(shape, n=2):
    return 0.5 * np.random.default_rng(3).standard_normal((n,) + shape)


def _given_up(ps, call):
    with pytest.raises(ps.PSError) as e:
        call()
    assert e.value.code == -3 and "barrier" in str(e.value)


@pytest.mark.parametrize("dim,shape,cell", GRIDS)
def test_model_reports_it(ps, monkeypatch, dim, shape, cell):
    monkeypatch.setenv("PS_B200_AUTOTUNE", "0")
    c = ps.make_cell(dim, *cell)
    w = _fields(shape)
    monkeypatch.setenv("PS_B200_BARRIER_GIVE_UP", "1")
    m = ps.ModelAB(dim, shape, c, (9, 13), 18.0, scft="Anderson", n_anderson=3)
    m.set_fields(w[0], w[1])
    m.update(2)
    for call in (m.synchronize, m.H, m.residual_error, m.Q, lambda: m.get("phiA"), lambda: m.update(1), m.forward):
        _given_up(ps, call)
    m.set_fields(w[0], w[1])   # a new start: no error is left
    m.synchronize()
    for call in (lambda: m.grad_w(w[0], w[1]), m.stress):
        _given_up(ps, call)
        m.set_fields(w[0], w[1])
    monkeypatch.delenv("PS_B200_BARRIER_GIVE_UP")
    n = ps.ModelAB(dim, shape, c, (9, 13), 18.0, scft="Anderson", n_anderson=3)
    n.set_fields(w[0], w[1])
    n.update(2)
    assert np.isfinite(n.H()).all()


def test_triblock_and_batch_report_it(ps, monkeypatch):
    monkeypatch.setenv("PS_B200_AUTOTUNE", "0")
    monkeypatch.setenv("PS_B200_BARRIER_GIVE_UP", "1")
    dim, shape, cell = GRIDS[0]
    c = ps.make_cell(dim, *cell)
    w = _fields(shape, 3)
    t = ps.ModelABC(dim, shape, c, (9, 13, 7), (18.0, 20.0, 22.0))
    t.set_fields(*w)
    t.update(1)
    for call in (t.synchronize, t.H, t.Q, t.residual_error, lambda: t.get("phiC"), lambda: t.update(1)):
        _given_up(ps, call)
    # a shared launch of three, and a solve alone
    shapes = [shape] * 3 + [(64, 64, 64)]
    b = ps.BatchAB([dict(dim=3, shape=s, cell=c, Ms=(9, 13), chiN=18.0) for s in shapes])
    f = [_fields(s) for s in shapes]
    for k in range(4):
        b.set_fields(k, *f[k])
    b.update(1)
    for call in (lambda: b.H(0), lambda: b.get(3, "phiA"), lambda: b.update(1)):
        _given_up(ps, call)
    for k in range(4):
        b.set_fields(k, *f[k])
    b.synchronize()


def test_updater_reports_it(ps, monkeypatch):
    import torch
    monkeypatch.setenv("PS_B200_BARRIER_GIVE_UP", "1")
    dim, shape, cell = GRIDS[0]
    u = ps.RQM4(ps.make_cell(dim, *cell), *shape, 0.01)
    w = _fields(shape, 1)[0]
    qs = np.zeros((9,) + shape)
    qs[0] = 1.0
    _given_up(ps, lambda: u.solve(qs, w))
    u.check()   # once
    tw, tq = torch.tensor(w, device="cuda"), torch.tensor(qs, device="cuda")
    torch.cuda.synchronize()
    u.solve(tq, tw)
    torch.cuda.synchronize()
    _given_up(ps, u.check)
    u.solve(tq, tw)
    torch.cuda.synchronize()
    _given_up(ps, lambda: u.solve(tq, tw))
    torch.cuda.synchronize()
    monkeypatch.delenv("PS_B200_BARRIER_GIVE_UP")
    v = ps.RQM4(ps.make_cell(dim, *cell), *shape, 0.01)
    out = v.solve(qs.copy(), w)
    v.check()
    assert np.isfinite(out).all()
