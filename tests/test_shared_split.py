"""Kernels that a lone match runs beside its scans take the scans' shared-memory split for those launches
alone: the split of the function, which every other match of the process launches with, stays the default
one. On the stand-in for the CUDA runtime."""
import pytest

from tests import fake_runtime


@pytest.mark.parametrize("make,kernel", [("plain(1000, 300, 64)", "k_cost3"), ("plain(1000, 300, 256)", "k_cost3"),
                                         ("pyramid(512, 320, 3)", "k_census4")])
def test_split_is_a_launch_attribute(engine_lib, tmp_path, make, kernel):
    lines = fake_runtime.run(fake_runtime.build(tmp_path), f"""
m = {make}
assert device(m) and device(m)
out(take())
""")
    assert not [x for x in lines if x.startswith("attribute") and kernel in x]
    launches = [x for x in lines if x.startswith("launch") and kernel in x]
    assert any(x.endswith("carveout 100") for x in launches), launches
    assert any(x.startswith("attribute") for x in lines)  # the scans' own
