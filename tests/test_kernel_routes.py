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
