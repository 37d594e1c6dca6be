"""Small-region removal joins horizontal runs of pixels: maps of many short, ragged regions against the
oracle at widths around the 32 pixels of a step and the 128 read at once, strips of one and more rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strips", [1, 6, 60])
@pytest.mark.parametrize("W", [64, 95, 96, 97, 127, 128, 129, 161, 256])
def test_removal_matches_oracle(engine_lib, oracle_mod, W, strips):
    import fasterstereocuda_b200 as fsc
    O = oracle_mod
    H = 61
    rng = np.random.default_rng(W)
    L = np.repeat(np.repeat(rng.integers(0, 256, (H // 2 + 1, W // 3 + 1)), 2, 0), 3, 1)[:H, :W].astype(np.uint8)
    L = np.ascontiguousarray(L)
    shift = np.repeat(np.repeat(rng.integers(1, 16, (H // 5 + 1, W // 7 + 1)), 5, 0), 7, 1)[:H, :W]
    R = np.take_along_axis(L, np.minimum(np.arange(W) + shift, W - 1), 1)
    ratio = 30.0 / (W * (H // strips))  # regions under 30 pixels go
    s = fsc.StereoCuda()
    assert s.Init(W, H, 0, 64, fsc.CuSGMOption(p1=10, p2_init=150, cs_type=1, num_paths=4, unique_threshold=0.95,
                                               using_constant_p2=True, do_remove_peaks=True,
                                               peaks_ratio_threshold=ratio)), s.last_error()
    assert s.set_ext_options(fsc.ExtOptions(tie_rule=4, init_tie_rule=4, peaks_strips=strips, peaks_abs_mode=0))
    disp = np.empty((H, W), np.float32)
    assert s.Match(L, R, disp), s.last_error()
    cfg = O.Config(width=W, height=H, disp_range=64, cs_type=1, p1=10, p2=150, uniqueness=0.95, do_lr_check=0,
                   do_median=0, do_remove_peaks=1, peaks_ratio=ratio, peaks_strips=strips, tie_rule=4, init_tie_rule=4)
    want = O.match(cfg, L, R)["disp"]
    assert np.array_equal(disp.view(np.uint32), want.view(np.uint32))
