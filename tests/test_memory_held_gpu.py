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


@pytest.mark.parametrize("scheme,precision,extra", [
    ("SESPH", "FP32", 0), ("PCISPH", "FP32", 0), ("IISPH", "FP32", 16), ("IISPH", "MIXED", 40),
    ("IISPH", "MIXED_POS16", 48)])
def test_solver_holds_what_its_passes_need(cuda, scheme, precision, extra):
    """A particle: eight scalars (density, pressure and its spare, diagonal,
    source, accelerations) 32 bytes, predicted velocity and boundary sums 32, 68
    list rows (64 entries, four of padding) and a count 276. IISPH adds packed accelerations 16 and MIXED
    the FP16 records 24, or MIXED_POS16 two records and the gradient moment 48. The
    slack is a sixth of a float4 a particle."""
    import torch

    import reyn_b200 as rb
    side, h = 128, 0.02
    n = side ** 3
    st = rb.Particles(n, 1000.0)
    rb.scene_fluid_block(st, (side,) * 3, (0.01,) * 3, h)
    box = ((0.0,) * 3, (side * h + 0.02,) * 3)
    grid = rb.Grid(*box, 2 * h)
    prm = rb.reference_params(getattr(rb, scheme), rb.C2, h, 1000.0, 0.01)
    prm.precision = getattr(rb, "PRECISION_" + precision)
    prm.max_iter = 3

    def step(sv):
        try:
            sv.step(st, grid, None, 1e-4)
        except rb.ReynError as e:  # three sweeps are enough here
            assert "max_iter" in str(e)

    for _ in range(2):  # kernels loaded, the state's own arrays in place
        grid.construct_and_reorder(st)
        sv = rb.Solver(getattr(rb, scheme), prm, n)
        step(sv)
        sv.close()
    grid.construct_and_reorder(st)
    before = _free()
    sv = rb.Solver(getattr(rb, scheme), prm, n)
    step(sv)
    held = before - _free()
    for o in (sv, grid, st):
        o.close()
    assert held <= (340 + extra) * n + 16 * n // 6, held / n
