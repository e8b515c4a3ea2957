"""Scene uploads through the pinned staging threads, the runtime faked (fake_cudart.cpp): when the call
returns, every byte has arrived whatever stream the renderer was given. A per-thread stream handle names a
stream of its own in each of the staging threads, so waiting for the caller's does not cover theirs.
And a staging thread that cannot be started, for whatever reason, leaves the work to the others."""
import pytest

from _fake_cuda import run

UPLOAD = """
r = PKG.GpsRenderer(64, 48, 1)
STREAM
n, sh = 200_003, np.random.default_rng(2).random(200_003 * 9, dtype=np.float32)
for k in range(3):
    r.set_gaussians_sh(scene(n, k), sh, 1)
    assert fake.fake_pending() == 0, (k, fake.fake_pending())
r.close()
"""


@pytest.mark.parametrize("stream", ["own", "per-thread"])
def test_every_byte_has_arrived(stream):
    run(UPLOAD.replace("STREAM", "" if stream == "own" else "r.set_stream(2)  # cudaStreamPerThread"))


def test_threads_that_cannot_be_started():
    run("""
fake.fake_fail_new.argtypes = [C.c_long]
r = PKG.GpsRenderer(64, 48, 1)
s = scene(200_003)
r.set_gaussians(s)
for k in range(4):
    fake.fake_fail_new(k)
    r.set_gaussians(s)
    fake.fake_fail_new(-1)
    assert fake.fake_pending() == 0 and r.gaussian_count() == len(s)
r.close()
""")
