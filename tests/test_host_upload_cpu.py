"""Scene uploads through the pinned staging threads, the runtime faked (fake_cudart.cpp): when the call
returns, every byte has arrived whatever stream the renderer was given. A per-thread stream handle names a
stream of its own in each of the staging threads, so waiting for the caller's does not cover theirs."""
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
