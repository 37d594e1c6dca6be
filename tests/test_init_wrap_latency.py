"""The warp-per-scanline scans of 32-disparity levels where the reference's uint32 recurrence wraps
(see test_init_wrap): both column forms, penalties up to the largest the options hold."""
import numpy as np
import pytest

from fasterstereocuda_b200 import scenes
from tests.test_init_wrap import STRIPS, adversarial_init

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p1,p2", [(10, 150), (10, 9000), (2147483647, 2147483647)])
@pytest.mark.parametrize("kind", ["cols", "rows", "random"])
def test_wrapping_paths_match_oracle(engine_lib, oracle_mod, kind, p1, p2):
    import torch
    import fasterstereocuda_b200 as fsc
    O = oracle_mod
    W, H = {"cols": (720, 40), "rows": (48, 600), "random": (300, 200)}[kind]
    L, R, _ = scenes.planar_pair(73, W, H)
    init = adversarial_init(kind, W, H, seed=5)
    opt = fsc.CuSGMOption(p1=p1, p2_init=p2, cs_type=1, num_paths=4, do_median_filter=True, do_lr_check=True,
                          lr_threshold=1.0, unique_threshold=0.95, using_constant_p2=True)
    cfg = O.Config(width=W, height=H, disp_range=32, cs_type=1, p1=p1, p2=p2, uniqueness=0.95, do_lr_check=1,
                   do_median=1, peaks_strips=STRIPS)
    ref = O.match(cfg, L, R, init, dump=True, want_right=True)
    valid = init != -32768

    def check(s, got):
        for name, i in (("lr", 1), ("rl", 3), ("bt", 2)):
            neq = (s.debug_read(name) != ref["paths"][i]).any(-1) & valid
            assert not neq.any(), (name, int(neq.sum()), np.argwhere(neq)[:3].tolist())
        assert np.array_equal(s.debug_read("wta", 0).view(np.uint32), ref["wta_l"].view(np.uint32))
        assert np.array_equal(s.debug_read("wta", 1).view(np.uint32), ref["wta_r"].view(np.uint32))
        assert np.array_equal(got.view(np.uint32), ref["disp"].view(np.uint32))
    s = fsc.StereoCuda()
    assert s.Init(W, H, 0, 32, opt), s.last_error()
    assert s.set_ext_options(fsc.ExtOptions(peaks_strips=STRIPS))
    out = torch.zeros(H, W, device="cuda")
    dl, dr, di = (torch.from_numpy(a).cuda() for a in (L, R, init))
    torch.cuda.synchronize()
    assert s.match_device(dl, dr, out, None, di), s.last_error()  # the column scan with the WTA in it
    torch.cuda.synchronize()
    check(s, out.cpu().numpy())
    disp = np.empty((H, W), np.float32)
    assert s.Match(L, R, disp, None, init), s.last_error()  # both column scans, then the WTA
    check(s, disp)
    assert engine_lib.sgm_debug_wait_timeouts() == 0
