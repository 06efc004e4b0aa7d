"""The record passes (MIXED_POS16) on particles with more neighbours than a list
row holds: the cell traversal in their place, with and without warm start."""
import numpy as np
import pytest

import oracle
from reyn_b200 import scenes
from tests.helpers import STEP_TOL, assert_close, by_id, run_engine, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warmstart", [0, 1])
@pytest.mark.parametrize("kind", [0, 2])
def test_crowded_records_vs_oracle(cuda, warmstart, kind):
    """Spacing 0.0125 at support 0.04: up to 144 neighbours. The mode's other tests
    allow twenty times the FP32 tolerances. A position is x + dt v, so it is held to
    dt times what v is held to, and three roundings."""
    import reyn_b200 as rb
    h, dt = 0.02, 5e-4
    sc = scenes.dam_break((11, 10, 9), 0.0125, (0.4, 0.4, 0.4), velocity_noise=0.05, seed=9)
    p = np.stack([sc.fluid[k] for k in "xyz"], 1).astype(np.float64)
    near = (np.linalg.norm(p[:, None] - p[None], axis=2) < 2 * h).sum(1) - 1
    assert (near > 64).sum() > 400 and (near <= 64).sum() > 100  # both paths
    bdy = dict(sc.bdy, m=oracle.boundary_masses(sc.bdy["x"], sc.bdy["y"], sc.bdy["z"], h,
                                                sc.rho0, 5))
    prm = rb.reference_params(rb.IISPH, kind, h, sc.rho0, 0.01)
    ref = oracle.reference_params(2, kind, h, sc.rho0, 0.01)
    prm.warmstart = ref.warmstart = warmstart
    prm.eta = ref.eta = 0.2
    prm.precision = rb.PRECISION_MIXED_POS16
    args = (2, kind, sc.fluid, bdy, sc.box_min, sc.box_max, h, sc.rho0, 0.01, dt, 1)
    got, want = run_engine(*args, params=prm), run_oracle(*args, params=ref)
    assert got.pop("iters") == want.pop("iters")
    g, w = by_id(got, got["id"]), by_id(want, want["id"])
    for k in ("vx", "vy", "vz", "m", "rho", "ax", "ay", "az", "p", "aii", "sii"):
        assert_close(g[k], w[k], *(20 * t for t in STEP_TOL[k]), k)
    for k in "xyz":
        rtol, af = (20 * t for t in STEP_TOL["v" + k])
        v = np.abs(w["v" + k].astype(np.float64))
        tol = dt * (rtol * v + af * v.max()) + 3 * 2.0 ** -24 * np.abs(w[k])
        err = np.abs(g[k].astype(np.float64) - w[k])
        assert (err <= tol).all(), (k, float((err / tol).max()))
