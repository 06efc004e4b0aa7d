"""A step that ends early leaves a state that the next step reads correctly:
the pressure passes take the packed velocities' memory, so the packed copies
must not count as valid after it."""
import ctypes

import pytest

from reyn_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP32", "MIXED", "MIXED_POS16"])
def test_step_after_a_failed_one_packs_again(cuda, precision):
    """The failure is the readback's wait for the stream, which a stream under
    capture refuses (its launches are recorded and never run)."""
    import torch

    import reyn_b200 as rb
    rt = ctypes.CDLL("libcudart.so.12")
    sc = scenes.dam_break((9, 8, 7), 0.02, (0.4, 0.4, 0.4), velocity_noise=0.05, seed=4)
    prm = rb.reference_params(rb.IISPH, rb.C2, sc.h, sc.rho0, 0.01)
    prm.warmstart = 0
    prm.precision = getattr(rb, "PRECISION_" + precision)
    side = torch.cuda.Stream()
    s = side.cuda_stream
    out = {}
    for fails in (False, True):
        st = rb.Particles(sc.n, sc.rho0)
        st.upload(sc.fluid)
        grid = rb.Grid(sc.box_min, sc.box_max, 2 * sc.h)
        sv = rb.Solver(rb.IISPH, prm, sc.n)
        for _ in range(2):  # every buffer is there and written
            grid.construct_and_reorder(st, stream=s)
            sv.step(st, grid, None, 1e-3, stream=s)
        grid.construct_and_reorder(st, stream=s)
        if fails:
            side.synchronize()
            graph = ctypes.c_void_p()
            assert rt.cudaStreamBeginCapture(ctypes.c_void_p(s), 2) == 0  # relaxed
            try:
                with pytest.raises(rb.ReynError):
                    sv.step(st, grid, None, 1e-3, stream=s)
            finally:
                assert rt.cudaStreamEndCapture(ctypes.c_void_p(s), ctypes.byref(graph)) != 0
                rt.cudaGetLastError()
        rb.profile_reset()
        sv.step(st, grid, None, 1e-3, stream=s)
        side.synchronize()
        packs = rb.profile_read().get("k_pack", (0, 0.0))[0]
        assert packs == int(fails)
        out[fails] = st.download()
        for o in (sv, grid, st):
            o.close()
    for k in out[False]:
        assert (out[False][k] == out[True][k]).all(), k
