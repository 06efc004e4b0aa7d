"""SESPH's viscous quotient (SESPH.cu:43-46) keeps the precision of a division:
isolated pairs whose other operands are exact or can be repeated on the host,
so that the quotient's own rounding is what is left."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 0.0625
SIDE = 16  # pairs along an axis, 0.5 apart: far beyond the support of 0.125
DX = 2.0 ** -5


def _pairs():
    """Pairs at (dx, dy), dx a power of two, dy = k 2^-13: positions, squares
    and their sum are exact in 32 bits. Velocities +-1 along x, mass 2^-12."""
    rng = np.random.Generator(np.random.PCG64(12))
    g = np.arange(SIDE, dtype=np.float64) * 0.5 + 0.25
    c = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    k = rng.integers(1, 960, len(c))
    a, b = c.copy(), c.copy()
    b[:, 0] += DX
    b[:, 1] += k * 2.0 ** -13
    p = np.concatenate([a, b]).astype(np.float32)
    n = len(p)
    fluid = {q: p[:, i].copy() for i, q in enumerate("xyz")}
    fluid.update(vx=np.where(np.arange(n) < n // 2, -1, 1).astype(np.float32),
                 vy=np.zeros(n, np.float32), vz=np.zeros(n, np.float32),
                 m=np.full(n, 2.0 ** -12, np.float32), id=np.arange(n, dtype=np.float32))
    l2 = (DX ** 2 + (k * 2.0 ** -13) ** 2).astype(np.float32)
    assert (l2.astype(np.float64) == DX ** 2 + (k * 2.0 ** -13) ** 2).all()
    return fluid, np.concatenate([l2, l2])


RUNS = 64


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_viscous_quotient_is_a_division(cuda, kind):
    """The acceleration of a pair from pressure alone is m prs g dx and from
    viscosity alone m (N / D) g dx, with the same g; m and dx are powers of two,
    and prs, N and D are formed here with the device's 32-bit operations. Over 64
    viscosities and 64 stiffnesses the mean of each quotient's error shows what
    is the same for every N at one D. A division leaves nothing: three roundings
    of at most u / sqrt(3) rms each (u = 2^-24), so an rms of sqrt(3 / 64) u /
    sqrt(3) = 0.125 u, and 0.14 u with five standard errors over the 900 values
    of D. A product with 1 / D keeps the reciprocal's own rounding, about 0.4 u
    even if that were correctly rounded."""
    import torch

    import reyn_b200 as rb
    f32 = np.float32
    fluid, l2 = _pairs()
    n = len(l2)
    rho0 = 2.0 ** -10
    rng = np.random.Generator(np.random.PCG64(kind))
    D = (l2 + f32(0.01 * H * H)).astype(np.float64)
    half = n // 2
    mean = {}
    for what in ("pressure", "viscosity"):
        total = np.zeros(n)
        for c in rng.uniform(1.0, 4.0, RUNS).astype(f32):
            prm = rb.reference_params(rb.SESPH, kind, H, rho0, 0.0)
            prm.g[0] = prm.g[1] = prm.g[2] = 0.0
            prm.nu = 0.0 if what == "pressure" else float(c)
            prm.k_sesph = float(c) if what == "pressure" else 0.0
            st = rb.Particles(n, rho0)
            st.upload(fluid)
            ids = torch.arange(n, device="cuda", dtype=torch.float32)
            grid = rb.Grid((0, 0, 0), (8.25, 8.25, 8.25), 2 * H)
            sv = rb.Solver(rb.SESPH, prm, n)
            grid.construct_and_reorder(st, [ids])
            sv.step(st, grid, None, 2.0 ** -20)
            torch.cuda.synchronize()
            at = np.argsort(ids.cpu().numpy())
            a, rho = (rb.device_to_numpy(getattr(sv.buffers(), k), n)[at] for k in ("ax", "rho"))
            for o in (sv, grid, st):
                o.close()
            inv = f32(1) / rho
            other = np.concatenate([inv[half:], inv[:half]])
            if what == "viscosity":
                q = (f32(10) * c * other * f32(2 * DX)).astype(np.float64) / D
            else:  # (k / rho0) w (1 - rho0 w), the bracket by one fused operation

                def term(w):
                    return c / f32(rho0) * w * (1.0 - rho0 * w.astype(np.float64)).astype(f32)

                q = (term(inv) + term(other)).astype(np.float64)
            assert (a != 0).all()
            total += np.abs(a.astype(np.float64)) / q
        mean[what] = total / RUNS
    err = (mean["viscosity"] / mean["pressure"] - 1.0) * 2.0 ** 24
    rms = float(np.sqrt(np.mean(err ** 2)))
    assert rms <= 0.14, f"rms {rms} u"
