"""Batches of mesh queries beyond the size from which they are ordered: results
whatever the order's cells are (points spread, gathered, coincident), the scratch
that a mesh keeps from one batch for the next, and the time of a batch that is
gathered in a small part of the mesh's box."""
import numpy as np
import pytest

import oracle
from reyn_b200 import meshes

pytestmark = pytest.mark.gpu


def _points(n, seed):
    """A third all over the box and beyond, a third gathered in 1/300 of its
    edges, the rest at one point, shuffled."""
    rng = np.random.Generator(np.random.PCG64(seed))
    p = rng.uniform(-1.3, 1.3, (3, n))
    k = n // 3
    p[:, k:2 * k] = 0.7 + rng.uniform(-1, 1, (3, k)) / 300
    p[:, 2 * k:] = np.array([[0.31], [-0.2], [0.9]])
    return p[:, rng.permutation(n)].astype(np.float32)


def test_one_mesh_many_batches(cuda):
    """The scratch grows, serves a smaller batch with fewer cells, and the larger
    one again."""
    import torch

    import reyn_b200 as rb
    v, f = meshes.icosphere(2)
    v = meshes.perturb(v, 0.01, 2)
    mesh = rb.Mesh(v, f)
    for k, n in enumerate((40000, 300001, 33000, 300001)):
        p = _points(n, k)
        t = [torch.tensor(c, device="cuda") for c in p]
        inside = mesh.inside(*t).cpu().numpy()
        np.testing.assert_array_equal(inside, oracle.lbvh_inside(v, f, *p))
        mesh.project(*t)
        for a, b in zip(t, oracle.lbvh_project(v, f, *p)):
            np.testing.assert_array_equal(a.cpu().numpy(), np.asarray(b))
    mesh.close()


@pytest.mark.parametrize("n", [(1 << 21) + 12345, (1 << 22) - 1, (1 << 22) + 12345, 5_000_001])
def test_large_batches_equal_small_ones(cuda, n):
    """Around and above the size from which a point has fewer cells: the same points
    in pieces that run in the caller's order."""
    import torch

    import reyn_b200 as rb
    v, f = meshes.icosphere(2)
    v = meshes.perturb(v, 0.01, 2)
    mesh = rb.Mesh(v, f)
    t = [torch.tensor(c, device="cuda") for c in _points(n, 3)]
    w = [c.clone() for c in t]
    step = (1 << 15) - 1
    parts = [mesh.inside(*(c[a:a + step] for c in t)) for a in range(0, n, step)]
    assert bool((mesh.inside(*t) == torch.cat(parts)).all())
    mesh.project(*t)
    for a in range(0, n, step):
        mesh.project(*(c[a:a + step] for c in w))
    for a, b in zip(t, w):
        assert bool((a == b).all())
    mesh.close()


@pytest.mark.parametrize("part", [64, 512, 2048])
def test_gathered_batches_are_ordered(cuda, part):
    """2.5M shuffled points in a small part of the box take about as long as the
    same points already in order. A batch whose points fall into one cell, or
    wait for the counters of a few, takes two to three times as long."""
    import torch

    import reyn_b200 as rb
    v, f = meshes.icosphere(6)
    v = meshes.perturb(v, 0.002, 1)
    n = 2_500_000
    rng = np.random.Generator(np.random.PCG64(5))
    c = np.array([[0.5], [0.6], [0.62]])
    u = rng.uniform(-1, 1, (3, n))
    p = (c / np.linalg.norm(c) + u / part).astype(np.float32)
    cell = ((u + 1) * 128).astype(np.int64)  # 256 cells an axis of the points' box
    code = np.zeros(n, np.int64)
    for b in range(8):
        for a in range(3):
            code |= ((cell[a] >> b) & 1) << (3 * b + 2 - a)
    mesh = rb.Mesh(v, f)

    def best(q):
        t = [torch.tensor(np.ascontiguousarray(a), device="cuda") for a in q]
        ms = []
        for _ in range(12):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            mesh.inside(*t)
            e[1].record()
            torch.cuda.synchronize()
            ms.append(e[0].elapsed_time(e[1]))
        return min(ms)

    shuffled, ordered = best(p), best(p[:, np.argsort(code, kind="stable")])
    mesh.close()
    assert shuffled < 1.5 * ordered, f"{shuffled} ms, in order {ordered} ms"
