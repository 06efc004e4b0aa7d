"""The traversal, build and query paths at the sizes where they can go wrong:
odd and tiny particle counts (warps and blocks that are partly empty, states
spread over more warps), cells split across runs of lanes and crowded ones,
cell counts that are no multiple of the scan's rows, boundaries of a few
samples, particles with more neighbours than a list row holds, and query
batches around the size from which they are ordered."""
import numpy as np
import pytest

import oracle
from reyn_b200 import meshes, scenes
from tests.helpers import STEP_TOL, assert_close, compare_steps, run_engine, run_oracle


def _chord_window(f, dy, dz, R):
    """The x-cells of one row the device code visits, in float32: the floors
    come from rounded-down additions of 1.5 * 2^23, whose results are floors."""
    eps = np.float32(1e-3)
    fx, fy, fz = (np.float32(v) for v in f)

    def gap2(d, v):
        g = max(np.float32(d) - v, np.float32(0)) if d > 0 else (
            max(v - np.float32(d + 1), np.float32(0)) if d < 0 else np.float32(0))
        return np.float32(g * g)

    rr = np.float32(R * R) * np.float32(1.001) + eps
    t = np.float32(rr - gap2(dz, fz) - gap2(dy, fy))
    if t < 0:
        return None
    w = np.sqrt(t, dtype=np.float32)
    a = int(np.floor(max(np.float32(fx - eps - w), np.float32(-R))))
    b = int(np.floor(min(np.float32(fx + eps + w), np.float32(R))))
    return a, b


@pytest.mark.parametrize("R", [1, 2])
def test_row_windows_cover_the_sphere(R):
    """Every point within r = R cells lies in the window of its row."""
    rng = np.random.Generator(np.random.PCG64(R))
    for k in range(4000):
        f = rng.random(3).astype(np.float32)
        if k % 8 == 0:  # on cell faces
            f[rng.integers(3)] = np.float32(rng.choice([0.0, 1.0 - 2.0 ** -24]))
        d = rng.normal(size=3)
        d *= R * rng.random() ** (1 / 3) / np.linalg.norm(d)
        if k % 5 == 0:
            d *= R / np.linalg.norm(d)  # on the sphere
        c = np.floor(f.astype(np.float64) + d).astype(int)
        if np.abs(c).max() > R:  # beyond the cells searched: at distance >= r
            continue
        win = _chord_window(f, c[1], c[2], R)
        assert win is not None and win[0] <= c[0] <= win[1], (f, d, c, win)


@pytest.mark.gpu
@pytest.mark.parametrize("ratio", [0.5, 1.0])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 4097])
def test_grid_paths_agree(cuda, ratio, n):
    """XYZ order (trimmed rows) and Z-order (the general traversal) see the same
    neighbours; each cell's particles ascend whatever the caller's order; builds
    with and without a reorder agree, one after the other on one grid."""
    import torch

    import reyn_b200 as rb
    rng = np.random.Generator(np.random.PCG64(n))
    p = rng.random((3, n)).astype(np.float32) * np.float32([[0.5], [0.3], [0.9]])
    p[:, : n // 3] = p[:, :1] + rng.random((3, n // 3)).astype(np.float32) * 0.01  # a crowd
    r = 0.11
    box = ((0.0, 0.0, 0.0), (0.5, 0.3, 0.9))
    x, y, z = (torch.tensor(v, device="cuda") for v in p)
    m = torch.ones(n, device="cuda")
    want = None
    for order in (rb.ORDER_XYZ, rb.ORDER_ZORDER):
        grid = rb.Grid(*box, r, ratio, order)
        g = oracle.geometry(*box, r, ratio, order)
        prefix, ordered = oracle.grid_build(g, *p)[:2]
        st = rb.Particles(n, 1.0)
        for _ in range(2):
            grid.construct(x, y, z)
            info = grid.info()
            np.testing.assert_array_equal(
                rb.device_to_numpy(grid.permutation_ptr(), n, np.uint32), ordered)
            np.testing.assert_array_equal(
                rb.device_to_numpy(info.prefix, info.n_keys + 1, np.uint32), prefix)
            count, len2, rho = grid.neighbour_stats(x, y, z, m, rb.C2)
            st.upload(dict(zip("xyz", p)))
            grid.construct_and_reorder(st)
            np.testing.assert_array_equal(
                rb.device_to_numpy(grid.permutation_ptr(), n, np.uint32), ordered)
            np.testing.assert_array_equal(st.download()["y"], p[1][ordered])
        got = [t.cpu().numpy() for t in (count, len2, rho)]
        if want is None:
            want = got
        np.testing.assert_array_equal(got[0], want[0])
        # sums of up to n terms in another order: n / 2 roundings at most
        for a, b in zip(got[1:], want[1:]):
            assert_close(a, b, 6e-8 * max(8, n), 0.0, f"order {order}")
        grid.close()
        st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [1, 2, 300])
def test_boundary_reach(cuda, nb):
    """Few samples anywhere: every fluid particle within 2h sees them (the flags
    of the cells within reach), and the masses match the oracle's."""
    import torch

    import reyn_b200 as rb
    rng = np.random.Generator(np.random.PCG64(nb))
    h = 0.05
    b = rng.random((3, nb)).astype(np.float32)
    f = rng.random((3, 3000)).astype(np.float32)
    tb = [torch.tensor(v, device="cuda") for v in b]
    tf = [torch.tensor(v, device="cuda") for v in f]
    bd = rb.Boundary(*tb, None, h=h, rho0=1000.0)
    ptrs, k = bd.arrays()
    arr = [rb.device_to_numpy(q, k) for q in ptrs]
    mass = oracle.boundary_masses(*b, h, 1000.0, 5)
    i = np.lexsort(b[::-1])
    j = np.lexsort(np.stack(arr[:3])[::-1])
    assert_close(arr[3][j], np.asarray(mass)[i], 1e-5, 0.0, "masses")
    grid = rb.Grid((0, 0, 0), (1, 1, 1), 2 * h)
    grid.construct(*tf)
    zero = torch.zeros(3000, device="cuda")
    rho = grid.compute_densities(*tf, zero, bd, rb.B3).cpu().numpy()
    d = np.linalg.norm(f.T.astype(np.float64)[:, None] - np.stack(arr[:3], 1)[None], axis=2)
    q = np.minimum(d / (2 * h), 1.0)
    w = 16 / np.pi / (2 * h) ** 3 * ((1 - q) ** 3 - 4 * np.clip(0.5 - q, 0, 1) ** 3)
    ref = w @ arr[3].astype(np.float64)
    # W near the support's edge cancels to (1 - q)^3: absolute error of q
    assert_close(rho, ref, 1e-5, 1e-6, "boundary density")
    for o in (grid, bd):
        o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [(1, 1, 1), (3, 1, 1), (11, 3, 1), (7, 5, 13), (20, 20, 20)])
@pytest.mark.parametrize("scheme", [0, 1, 2])
def test_small_states_vs_oracle(cuda, counts, scheme):
    import reyn_b200 as rb
    sc = scenes.dam_break(counts, 0.02, np.asarray(counts) * 0.02 + 0.2, velocity_noise=0.05,
                          seed=3)
    bdy = dict(sc.bdy, m=oracle.boundary_masses(sc.bdy["x"], sc.bdy["y"], sc.bdy["z"], sc.h,
                                                sc.rho0, 5))
    prm = rb.reference_params(scheme, 1, sc.h, sc.rho0, 0.01)
    args = (scheme, 1, sc.fluid, bdy, sc.box_min, sc.box_max, sc.h, sc.rho0, 0.01, 5e-4, 1)
    got, want = run_engine(*args, params=prm), run_oracle(*args)
    assert got["iters"] == want["iters"]
    compare_steps(got, want, scheme, STEP_TOL, f"{counts} scheme {scheme}")


@pytest.mark.gpu
@pytest.mark.parametrize("precision,spacing", [("FP32", 0.02), ("MIXED", 0.02),
                                               ("MIXED_POS16", 0.02), ("FP32", 0.0125),
                                               ("MIXED", 0.0125)])
@pytest.mark.parametrize("warmstart", [0, 1])
def test_iisph_lists_and_overflow(cuda, precision, warmstart, spacing):
    """Ordinary and crowded states (at 0.0125 up to 136 neighbours, beyond the
    list) with and without warm start: one step of three sweeps (any error is
    within a tolerance of 20 %) on the lists and on the cell traversal against
    the oracle, the mixed modes at twenty times the FP32 tolerance."""
    import reyn_b200 as rb
    sc = scenes.dam_break((11, 10, 9), spacing, (0.4, 0.4, 0.4), velocity_noise=0.05, seed=9)
    h = 0.02
    bdy = dict(sc.bdy, m=oracle.boundary_masses(sc.bdy["x"], sc.bdy["y"], sc.bdy["z"], h,
                                                sc.rho0, 5))
    prm = rb.reference_params(rb.IISPH, rb.C2, h, sc.rho0, 0.01)
    ref = oracle.reference_params(2, 0, h, sc.rho0, 0.01)
    prm.warmstart = ref.warmstart = warmstart
    prm.eta = ref.eta = 0.2
    prm.precision = getattr(rb, "PRECISION_" + precision)
    args = (2, 0, sc.fluid, bdy, sc.box_min, sc.box_max, h, sc.rho0, 0.01, 5e-4, 1)
    got, want = run_engine(*args, params=prm), run_oracle(*args, params=ref)
    assert got["iters"] == want["iters"]
    f = 1 if precision == "FP32" else 20
    compare_steps(got, want, 2, {k: (f * r, f * a) for k, (r, a) in STEP_TOL.items()},
                  f"{precision} {spacing} warm {warmstart}")


@pytest.mark.gpu
@pytest.mark.parametrize("n,spread", [(32767, 1.0), (32768, 1.0), (32769, 1.0), (40000, 0.0),
                                      (33000, 3.0)])
def test_query_order_does_not_matter(cuda, n, spread):
    """Batches around the size from which queries are ordered, all in one cell
    of the order, and mostly outside the mesh's box."""
    import torch

    import reyn_b200 as rb
    v, f = meshes.icosphere(3)
    v = meshes.perturb(v, 0.01, 2)
    rng = np.random.Generator(np.random.PCG64(n))
    p = (rng.uniform(-1, 1, (3, n)) * spread + 0.1).astype(np.float32)
    mesh = rb.Mesh(v, f)
    t = [torch.tensor(c, device="cuda") for c in p]
    mesh.project(*t)
    want = oracle.lbvh_project(v, f, *p)
    for a, b in zip(t, want):
        np.testing.assert_array_equal(a.cpu().numpy(), np.asarray(b))
    inside = mesh.inside(*(torch.tensor(c, device="cuda") for c in p)).cpu().numpy()
    np.testing.assert_array_equal(inside, oracle.lbvh_inside(v, f, *p))
    mesh.close()
