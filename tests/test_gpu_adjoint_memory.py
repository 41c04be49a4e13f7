"""The adjoint's kept fields where the device has little room: the line passes serve,
nothing of the attempt stays allocated, and what others need is left to them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE, MS = (48, 48, 48), (33, 41)
KEPT = 8 * 72 * 48 ** 3   # bytes of one kept field of all steps


def _free():
    import torch
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _model(ps, w):
    m = ps.ModelAB(3, SHAPE, ps.make_cell(3, "CUBIC", 4.0), MS, 18.0)
    m.set_fields(*w)
    return m


def test_little_room(monkeypatch):
    import torch
    import polystring_b200 as ps
    rng = np.random.default_rng(6)
    w = rng.uniform(-1, 1, (2,) + SHAPE)
    a, b = rng.standard_normal((2,) + SHAPE)
    monkeypatch.setenv("PS_B200_LINE_PASSES", "1")
    ref = _model(ps, w).grad_w(a, b, 0.7)
    monkeypatch.delenv("PS_B200_LINE_PASSES")
    m = _model(ps, w)
    swept = (*m.grad_w(a, b, 0.7), m.stress())

    def check(m, grad, stress):
        """which form served: the sweeps' results are the same bit for bit"""
        gA, gB = m.grad_w(a, b, 0.7)
        assert np.array_equal(gA, swept[0]) == grad and np.array_equal(gB, swept[1]) == grad
        for x, y in zip((gA, gB), ref):
            # sums of some 2 Ns terms, 50 roundings each, as in the comparison with room
            assert np.abs(x - y).max() < 1e-10 * np.abs(y).max()
        assert np.array_equal(m.stress(), swept[2]) == stress

    m = _model(ps, w)
    total = torch.cuda.mem_get_info()[1]
    # room for neither beside the sixteenth: about two kept fields' bytes beyond it
    hold = torch.empty(_free() - total // 16 - 2 * KEPT, dtype=torch.uint8, device="cuda")
    before = _free()
    check(m, False, False)
    check(m, False, False)
    assert before - _free() < KEPT
    # room for the stress's four, not for the gradient's: the stress's stay
    del hold
    hold = torch.empty(_free() - total // 16 - 7 * KEPT, dtype=torch.uint8, device="cuda")
    before = _free()
    check(m, False, True)
    assert 3.9 * KEPT < before - _free() < 4.5 * KEPT
    check(m, False, True)
    assert 3.9 * KEPT < before - _free() < 4.5 * KEPT
    # room for all
    del hold
    before = _free()
    check(m, True, True)
    assert 5.9 * KEPT < before - _free() < 7.5 * KEPT
    before = _free()
    del m
    assert _free() - before > 9.9 * KEPT
