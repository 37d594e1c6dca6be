"""32-disparity levels whose chunks have no INVALID base (the short form of the warp-per-scanline scans'
step), mixed with chunks that have some, at sizes around the 32-step chunks and the groups of 8 steps
read ahead; shifts within and beyond the range; penalties beyond 22 bits."""
import numpy as np
import pytest

from fasterstereocuda_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p1,p2", [(10, 150), (0, 0), (127, 16383), (5_000_000, 9_000_000)])
@pytest.mark.parametrize("k,size", list(enumerate([(64, 64), (65, 71), (95, 97), (104, 39), (129, 128)])))
def test_paths_and_disparities(engine_lib, oracle_mod, k, size, p1, p2):
    import fasterstereocuda_b200 as fsc
    O = oracle_mod
    W, H = size
    cs = k % 2
    L, R, _ = scenes.planar_pair(500 + k, W, H, dmin=0.0, dmax=W / 4)
    rng = np.random.default_rng(k)
    init = rng.integers(-2, 5, (H, W)).astype(np.int16)
    init[::5, ::7] = 60            # realignments beyond the range
    init[H // 2, 3:40] = -32768    # INVALID bases in some chunks of the rows ...
    init[40:60, W // 2] = -32768   # ... and of the columns
    s = fsc.StereoCuda()
    assert s.Init(W, H, 0, 32, fsc.CuSGMOption(p1=p1, p2_init=p2, cs_type=cs, num_paths=4, do_lr_check=True,
                                               do_median_filter=True, lr_threshold=1.0, unique_threshold=0.95,
                                               using_constant_p2=True)), s.last_error()
    assert s.set_tuning(fsc.Tuning(4, 0, 4, 0, 0)), s.last_error()
    disp = np.empty((H, W), np.float32)
    assert s.Match(L, R, disp, None, init), s.last_error()
    ref = O.match(O.Config(width=W, height=H, disp_range=32, cs_type=cs, p1=p1, p2=p2, do_lr_check=1, do_median=1), L, R,
                  init, dump=True, want_right=True)
    valid = init != -32768
    for name, i in (("lr", 1), ("rl", 3), ("bt", 2)):
        assert np.array_equal(s.debug_read(name)[valid], ref["paths"][i][valid]), name
    for got, want in ((s.debug_read("wta", 0), ref["wta_l"]), (s.debug_read("wta", 1), ref["wta_r"]),
                      (disp, ref["disp"])):
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert engine_lib.sgm_debug_wait_timeouts() == 0
