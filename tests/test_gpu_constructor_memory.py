"""A model that does not fit on the device is refused, and nothing of it stays allocated."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,mde", [("ModelAB", "RQM4"), ("ModelAB", "ETDRK4"), ("ModelABC", "RQM4"),
                                      ("StringAB", "RQM4")])
def test_refused_model_leaves_nothing(kind, mde):
    import torch
    import polystring_b200 as ps
    # histories of 2 x 240 001 slices of 2 MiB: 1 TB
    shape, n = ((64, 64, 64), 120001) if kind != "StringAB" else ((128, 64, 1), 960001)

    def make(n):
        if kind == "ModelABC":
            return ps.ModelABC(3, shape, ps.make_cell(3, "CUBIC", 4.0), (n, n, 7), (18.0, 18.0, 18.0))
        if kind == "StringAB":
            return ps.StringAB(12, 2, shape, ps.make_cell(2, "RECTANGULAR", 4.0, 4.0), (n, n), 18.0)
        return ps.ModelAB(3, shape, ps.make_cell(3, "CUBIC", 4.0), (n, n), 18.0, mde=mde)

    make(9)   # kernels, tables of the process, the tuner's choice
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(4):
        with pytest.raises(ps.PSError) as e:
            make(n)
        assert e.value.code == -3 and "out of memory" in str(e.value)
    # four attempts; their work fields are 16 fields each at least.  Less than one may stay
    assert before - torch.cuda.mem_get_info()[0] < 8 * shape[0] * shape[1] * shape[2] + (4 << 20)
