"""Plain levels in 16-bit halves (one warp per scanline, D = 64, 128 and 256) against the oracle, stage by
stage: sizes around the staged chunks (32 steps, 16 at D = 256), penalties at the edges of the 16-bit
form (P1 = 127 is its last, P1 = 128 takes the 32-bit form), ranges that start below and above zero."""
import numpy as np
import pytest

from fasterstereocuda_b200 import scenes

pytestmark = pytest.mark.gpu

SIZES = [(12, 11), (33, 16), (64, 33), (97, 47), (131, 64)]


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("p1,p2", [(0, 0), (10, 150), (127, 127), (127, 16383), (128, 300)])
@pytest.mark.parametrize("k,size", list(enumerate(SIZES)))
def test_paths_and_disparities(engine_lib, oracle_mod, D, p1, p2, k, size):
    import fasterstereocuda_b200 as fsc
    O = oracle_mod
    W, H = size
    M, cs = (0, 3, -5, 0, 2)[k], k % 2
    L, R, _ = scenes.planar_pair(300 + k, W, H, dmin=0.0, dmax=W / 3)
    s = fsc.StereoCuda()
    assert s.Init(W, H, M, D, fsc.CuSGMOption(p1=p1, p2_init=p2, cs_type=cs, num_paths=4, do_lr_check=True,
                                              do_median_filter=True, lr_threshold=1.0, unique_threshold=0.95,
                                              using_constant_p2=True)), s.last_error()
    if D != 256:  # the warp-per-scanline kernels; D = 256 takes its own by default
        assert s.set_tuning(fsc.Tuning(4, 0, 4, 0, 0)), s.last_error()
    disp = np.empty((H, W), np.float32)
    right = np.empty((H, W), np.float32)
    assert s.Match(L, R, disp, right), s.last_error()
    ref = O.match(O.Config(width=W, height=H, min_disp=M, disp_range=D, cs_type=cs, p1=p1, p2=p2), L, R, dump=True,
                  want_right=True)
    x0 = max(0, M)
    assert np.array_equal(s.debug_read("cost")[:, x0:], ref["cost"][:, x0:])
    for name, i in (("lr", 1), ("rl", 3), ("bt", 2)):
        assert np.array_equal(s.debug_read(name)[:, x0:], ref["paths"][i][:, x0:]), name
    for got, want in ((s.debug_read("wta", 0), ref["wta_l"]), (s.debug_read("wta", 1), ref["wta_r"]),
                      (disp, ref["disp"]), (right, ref["disp_r"])):
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert engine_lib.sgm_debug_wait_timeouts() == 0
