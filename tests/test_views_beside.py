"""The views of a plain level on streams beside each other (levels of at least 888 x 296 pixels on 148 SMs)
and together (just below), against the oracle: first calls and graph replays with other images through
the host API and on a caller's stream, and a first call inside a caller's capture."""
import gc

import numpy as np
import pytest

from fasterstereocuda_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,M,D,cs", [(888, 296, 0, 64, 1), (887, 296, 0, 64, 1), (888, 295, 3, 128, 0),
                                        (901, 297, -5, 128, 0), (889, 299, 2, 256, 1), (890, 300, 0, 32, 0)])
def test_match(engine_lib, oracle_mod, W, H, M, D, cs):
    import torch

    import fasterstereocuda_b200 as fsc
    O = oracle_mod
    pairs, want = [], []
    for k in range(2):
        L, R, _ = scenes.planar_pair(700 + k, W, H, dmin=2.0, dmax=min(60.0, D - 4.0))
        pairs.append((torch.from_numpy(L).cuda(), torch.from_numpy(R).cuda()))
        want.append(O.match(O.Config(width=W, height=H, min_disp=M, disp_range=D, cs_type=cs, p1=10, p2=150), L, R)["disp"])
    opt = fsc.CuSGMOption(p1=10, p2_init=150, cs_type=cs, num_paths=4, do_lr_check=True, do_median_filter=True,
                          lr_threshold=1.0, unique_threshold=0.95, using_constant_p2=True)
    gc.collect()  # the only matcher, if no other test's is still held
    s = fsc.StereoCuda()
    assert s.Init(W, H, M, D, opt), s.last_error()
    for i in range(6):
        disp = np.zeros((H, W), np.float32)
        assert s.Match(*(im.cpu().numpy() for im in pairs[i % 2]), disp), s.last_error()
        assert np.array_equal(disp.view(np.uint32), want[i % 2].view(np.uint32)), i
    outs = [torch.zeros(H, W, device="cuda") for _ in range(6)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    for i, out in enumerate(outs):  # no wait between the calls
        assert s.match_device(*pairs[i % 2], out, stream=stream.cuda_stream), s.last_error()
    torch.cuda.synchronize()
    del s
    gc.collect()
    c = fsc.StereoCuda()
    assert c.Init(W, H, M, D, opt), c.last_error()
    graph, cap = torch.cuda.CUDAGraph(), torch.zeros(H, W, device="cuda")
    with torch.cuda.graph(graph, stream=stream):
        assert c.match_device(*pairs[0], cap, stream=stream.cuda_stream), c.last_error()
    graph.replay()
    torch.cuda.synchronize()
    for i, got in enumerate(outs + [cap]):
        exp = want[0 if i == len(outs) else i % 2]
        assert np.array_equal(got.cpu().numpy().view(np.uint32), exp.view(np.uint32)), i
    assert engine_lib.sgm_debug_wait_timeouts() == 0
