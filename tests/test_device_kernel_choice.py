"""The device API's kernel choice by the number of initialised matchers: the same bits with few matchers
(latency kernels) and with many (default kernels), after a change of that number, and for a first match
recorded into the caller's own CUDA graph."""
import numpy as np
import pytest

from fasterstereocuda_b200 import scenes

pytestmark = pytest.mark.gpu

W, H = 322, 187


def _plain(fsc, D):
    s = fsc.StereoCuda()
    assert s.Init(W, H, 0, D, fsc.CuSGMOption(p1=10, p2_init=150, cs_type=1, num_paths=4, do_lr_check=True,
                                              do_median_filter=True, lr_threshold=1.0, unique_threshold=0.95,
                                              using_constant_p2=True)), s.last_error()
    return s


def _pyramid(fsc):
    p = fsc.FasterStereoCuda()
    assert p.Init(fsc.StereoOption1(width=W, height=H, min_disp=0, max_disp=64, num_layers=2, do_lr_check=True,
                                    do_rm_peaks=True), fsc.LevelOverride(1, 10, 150), fsc.ExtOptions(peaks_strips=6))
    return p


def _references(O, L, R):
    out = {D: O.match(O.Config(width=W, height=H, disp_range=D, do_lr_check=1, do_median=1), L, R)["disp"]
           for D in (64, 128, 256)}
    out["pyramid"] = O.pyr_match(O.PyrConfig(width=W, height=H, min_disp=0, max_disp=64, num_layers=2,
                                             override_enable=1, cs_type=1, p1=10, p2=150, peaks_strips=6), L, R)
    return out


def test_few_and_many_matchers_give_the_same_bits(engine_lib, oracle_mod):
    import torch
    import fasterstereocuda_b200 as fsc
    L, R, _ = scenes.kitti_like(91, W, H)
    ref = _references(oracle_mod, L, R)
    dl, dr = torch.from_numpy(L).cuda(), torch.from_numpy(R).cuda()
    torch.cuda.synchronize()
    mine = {D: _plain(fsc, D) for D in (64, 128, 256)}
    mine["pyramid"] = _pyramid(fsc)

    def check(times):
        for key, m in mine.items():
            for _ in range(times):  # direct run, capture and replay
                out = torch.zeros(H, W, device="cuda")
                torch.cuda.synchronize()
                assert m.match_device(dl, dr, out), m.last_error()
                torch.cuda.synchronize()
                assert np.array_equal(out.cpu().numpy().view(np.uint32), ref[key].view(np.uint32)), key
    check(3)
    others = [_plain(fsc, 64) for _ in range(9)]
    check(3)
    for m in others:
        m.Release()
    check(2)
    assert engine_lib.sgm_debug_wait_timeouts() == 0


@pytest.mark.parametrize("key", [64, 256, "pyramid"])
def test_first_match_inside_a_callers_graph(engine_lib, oracle_mod, key):
    import torch
    import fasterstereocuda_b200 as fsc
    L, R, _ = scenes.kitti_like(92, W, H)
    ref = _references(oracle_mod, L, R)[key]
    m = _pyramid(fsc) if key == "pyramid" else _plain(fsc, key)
    dl, dr = torch.zeros(H, W, dtype=torch.uint8, device="cuda"), torch.zeros(H, W, dtype=torch.uint8, device="cuda")
    out = torch.zeros(H, W, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        assert m.match_device(dl, dr, out, stream=s.cuda_stream), m.last_error()
    for _ in range(2):
        dl.copy_(torch.from_numpy(L))
        dr.copy_(torch.from_numpy(R))
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32))
