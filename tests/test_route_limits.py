"""Images past a limit of the warp-per-scanline kernels keep the general ones: more rows than a grid has
in y (65535, the cost kernel's), rows whose bytes overflow a tensor map's coordinate. The routes on the
CPU with the runtime's stand-in; the bits on a GPU."""
import numpy as np
import pytest

from tests import fake_runtime

LATENCY = {"k_hscan_plain4", "k_vscan_plain4", "k_hscan_plain256", "k_vscan_plain256"}


@pytest.fixture(scope="module")
def fake(engine_lib, tmp_path_factory):
    return fake_runtime.build(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("W,H,D,p1,p2", [(16, 65536, 256, 10, 150), (16, 65536, 64, 50, 20), (16, 65536, 128, 10, 20000),
                                         (8388608, 2, 256, 10, 150), (33554432, 1, 64, 10, 150)])
def test_plain_route(fake, W, H, D, p1, p2):
    ok, err, ks, lines = fake_runtime.run(fake, f"""
s = plain({W}, {H}, {D}, p1={p1}, p2_init={p2}, do_lr_check=False)
take()
ok = device(s)
lines = take()
out([ok, s.last_error(), kernels(lines), lines])
""")
    assert ok, err
    assert not LATENCY & set(ks), ks
    assert not [x for x in lines if x.startswith("REFUSED")]


@pytest.mark.parametrize("W,H,D", [(16, 65535, 256), (4194304, 2, 256), (16, 65535, 64), (16777216, 2, 64)])
def test_plain_route_within_the_limits(fake, W, H, D):
    ok, err, ks = fake_runtime.run(fake, f"""
s = plain({W}, {H}, {D}, do_lr_check=False)
take()
ok = device(s)
out([ok, s.last_error(), kernels(take())])
""")
    assert ok, err
    assert LATENCY & set(ks), ks


@pytest.mark.gpu
@pytest.mark.parametrize("D,p1,p2", [(256, 10, 150), (64, 50, 20)])
def test_tall_image(engine_lib, oracle_mod, D, p1, p2):
    import torch
    import fasterstereocuda_b200 as fsc
    W, H = 24, 65537
    rng = np.random.default_rng(D)
    L, R = (rng.integers(0, 256, (H, W)).astype(np.uint8) for _ in range(2))
    s = fsc.StereoCuda()
    assert s.Init(W, H, 0, D, fsc.CuSGMOption(p1=p1, p2_init=p2, cs_type=0, num_paths=4, lr_threshold=1.0,
                                              unique_threshold=0.95, using_constant_p2=True)), s.last_error()
    out = torch.zeros(H, W, device="cuda")
    dl, dr = torch.from_numpy(L).cuda(), torch.from_numpy(R).cuda()
    torch.cuda.synchronize()
    assert s.match_device(dl, dr, out), s.last_error()
    torch.cuda.synchronize()
    want = oracle_mod.match(oracle_mod.Config(width=W, height=H, disp_range=D, cs_type=0, p1=p1, p2=p2, do_lr_check=0,
                                              do_median=0), L, R)["disp"]
    assert (want != -999999.0).any()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
