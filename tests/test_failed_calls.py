"""A CUDA call that fails somewhere in a match: the match returns an error, the matcher keeps its own
streams and destroys each exactly once, and never the caller's; a stream capture in progress is ended
and the next match works. Every call of the first two matches (one direct, one recorded) is made to fail
in turn, on the stand-in for the CUDA runtime."""
import pytest

from tests import fake_runtime

MAKE = {"plain_beside": "plain(1000, 300, 64)", "plain_256": "plain(320, 200, 256)", "pyramid": "pyramid(512, 320, 3)"}


@pytest.fixture(scope="module")
def fake(engine_lib, tmp_path_factory):
    return fake_runtime.build(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("call", ["cudaStreamWaitEvent", "cudaEventRecord", "cudaLaunchKernel", "cudaGraphInstantiate",
                                  "cudaStreamBeginCapture", "cudaStreamEndCapture"])
@pytest.mark.parametrize("kind", list(MAKE))
def test_streams_after_a_failed_call(fake, kind, call):
    failures = fake_runtime.run(fake, f"""
import gc
USER = 0x99990
n = failures = 0
while True:
    take()
    m = {MAKE[kind]}
    made = [l.split()[1] for l in take() if l.startswith("stream")]
    fake.fake_fail({call!r}.encode(), n)
    results = [device(m, USER) for _ in range(2)]
    failed = any(l.startswith("FAILED") for l in take())
    fake.fake_fail(b"", -1)
    failures += failed
    assert all(results) != failed, (n, results)
    assert device(m, USER) and device(m), (n, m.last_error())
    lines = take()
    assert sum(l.startswith("capture") for l in lines) == sum(l.startswith("end capture") for l in lines)
    m.Release()
    gone = [l.split()[2] for l in take() if l.startswith("destroy stream")]
    assert sorted(gone) == sorted(made), (n, made, gone)
    if not failed:
        break
    n += 1
out(failures)
""")
    assert failures > 0
