"""What the engine's objects keep on the device, by the free memory before and
after: no more than the arrays that their later use needs."""
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_boundary_keeps_no_scratch(cuda):
    """A sample: records and masses 16 + 16 bytes, keys, slots, order and marks
    13; a cell: counts, prefix and flag 9. A second mass buffer would be 16 more
    a sample. The slack is a sixth of that: allocations come in 2 MB pieces."""
    import torch

    import reyn_b200 as rb
    side, spacing, h = 1400, 0.25, 1.0
    n = side * side
    g = torch.arange(side, device="cuda", dtype=torch.float32) * spacing
    x, y = (t.contiguous().view(-1) for t in torch.meshgrid(g, g, indexing="ij"))
    z = torch.zeros(n, device="cuda")
    rb.Boundary(x[:1000], y[:1000], z[:1000], None, h=h, rho0=1.0).close()  # kernels loaded
    before = _free()
    bd = rb.Boundary(x, y, z, None, h=h, rho0=1.0)
    held = before - _free()
    cells = 1
    for extent in ((side - 1) * spacing, (side - 1) * spacing, 0.0):
        cells *= int((extent + 8 * h) / h) + 2  # a margin of 4 h on each side, cells of h
    bd.close()
    assert held <= 45 * n + 9 * cells + 16 * n // 6, held / n
