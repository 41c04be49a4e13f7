"""An updater holds one form of its solve only: the persistent sweep's work fields and
factors where the grid has one."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,shape", [(3, (64, 64, 64)), (2, (256, 352, 1))])
def test_updater_holds_one_form(dim, shape):
    import torch
    import polystring_b200 as ps
    cell = ps.make_cell(dim, ("RECTANGULAR", "ORTHORHOMBIC")[dim - 2], *(4.0, 4.2, 4.4)[:dim])
    make = lambda: ps.RQM4(cell, *shape, 0.01)   # noqa: E731
    make()   # kernels loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    held = [make() for _ in range(4)]
    field = 8 * shape[0] * shape[1] * shape[2]
    # four factors and two work fields, each allocation rounded up to 2 MiB, and 8 MiB for the small ones
    assert before - torch.cuda.mem_get_info()[0] <= len(held) * (6 * (field + (2 << 20))) + (8 << 20)
