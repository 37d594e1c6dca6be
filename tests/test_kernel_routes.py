"""Which kernels a call takes, by what else the process holds and by size, on the stand-in for the CUDA
runtime: the forms give the same bits, so a test of those alone would pass on either."""
import pytest

from tests import fake_runtime

HELP = """
def match(m):
    take()
    assert device(m), m.last_error()
    return take()
def streams(lines, kernel):
    return {l.split(" stream ")[1].split()[0] for l in lines if l.startswith("launch") and kernel in l}
"""


@pytest.fixture(scope="module")
def run(engine_lib, tmp_path_factory):
    lib = fake_runtime.build(tmp_path_factory.mktemp("fake"))
    return lambda code: fake_runtime.run(lib, HELP + code)


@pytest.mark.parametrize("W,H,D,beside", [(888, 296, 64, True), (887, 296, 64, False), (888, 295, 64, False),
                                          (888, 296, 128, True), (888, 296, 256, True), (888, 295, 256, False)])
def test_views_beside_each_other_only_alone_and_large(run, W, H, D, beside):
    one, two, one_view = run(f"""
a = plain({W}, {H}, {D})
one = match(a)
b = plain(64, 64, 64)
two = match(a)
b.Release(); a.Release()
c = plain({W}, {H}, {D}, do_lr_check=False)
out([[len(streams(x, "scan_plain")), kernels(x).count("k_cost3")] for x in (one, two, match(c))])
""")
    assert one == ([3, 2] if beside else [2, 1])
    assert two == [2, 1]  # columns beside rows, both views a launch
    assert one_view == [2, 1]


@pytest.mark.parametrize("D", [64, 128])
def test_latency_kernels_up_to_eight_matchers(run, D):
    eight, nine, again = run(f"""
a = plain(320, 200, {D})
others = [plain(64, 64, 64) for _ in range(7)]
eight = match(a)
others.append(plain(64, 64, 64))
nine = match(a)
others.pop().Release()
p = pyramid(256, 160, 2)
p.Release()
out([kernels(eight), kernels(nine), len([l for l in match(a) if l.startswith("capture")])])
""")
    assert "k_hscan_plain4" in eight and "k_vscan_plain4" in eight
    assert "k_hpaths3" in nine and "k_vpaths3" in nine
    assert again == 1  # the second match with the latency kernels records them


@pytest.mark.parametrize("p1,p2,rule,narrow", [(127, 16383, 0, True), (128, 16383, 0, False), (127, 16384, 0, False),
                                               (50, 49, 0, False), (10, 150, 4, True), (10, 150, 1, False)])
def test_256_disparities(run, p1, p2, rule, narrow):
    ks = run(f"""
a = plain(320, 200, 256, p1={p1}, p2_init={p2}, ext=dict(tie_rule={rule}))
out(kernels(match(a)))
""")
    assert ("k_hscan_plain256" in ks and "k_vscan_plain256" in ks) == narrow
    assert ("k_hpaths_plain2" in ks) != narrow


def test_pyramid_forms(run):
    dev, many, host = run("""
def census_beside(x):  # a level's census beside the coarser level's scans has their shared-memory split
    return sum("k_census4" in l and l.endswith("carveout 100") for l in x)
p = pyramid(512, 320, 3)
x = match(p)
others = [plain(64, 64, 64) for _ in range(8)]
y = match(p)
im, o = np.zeros((320, 512), np.uint8), np.zeros((320, 512), np.float32)
take()
assert p.Match(im, im, o)
z = take()
out([[kernels(v), census_beside(v)] for v in (x, y, z)])
""")
    assert dev[0].count("k_vscan_wta_init4") == 2 and "k_wta_init4" not in dev[0] and dev[1] == 2
    assert "k_hpaths3_init" in many[0] and "k_hscan_init4" not in many[0] and many[1] == 0
    assert host[0].count("k_wta_init4") == 2 and "k_vscan_wta_init4" not in host[0] and host[1] == 2


@pytest.mark.parametrize("make,captures", [("plain(450, 375, 64)", 1), ("pyramid(512, 320, 3)", 1),
                                           ("plain(1000, 300, 64)", 2)])
def test_a_second_matcher_has_nothing_recorded_again(run, make, captures):
    """One graph for a match alone and beside others, except where their launches differ."""
    got = run(f"""
a = {make}
lines = []
for k in range(3):
    for _ in range(3):
        lines += match(a)
    if k == 0:
        b = plain(64, 64, 64)
    elif k == 1:
        b.Release()
out(sum(l.startswith("capture") for l in lines))
""")
    assert got == captures
