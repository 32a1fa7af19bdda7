"""Predictions for host rows go through the device in chunks (77824 rows at
width 256, 65536 otherwise) over a ring of four: at the edges of a chunk and of
the ring every row gets the bits that it gets in a call of its own rows."""
import numpy as np
import pytest

from ec2d import gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,chunk", [(256, 77824), (128, 65536)])
def test_chunk_edges(gpu_lib, width, chunk):
    net = gpu.WarmStartNet(hidden=2, width=width, seed=5)
    rng = np.random.default_rng(7)
    feat = rng.standard_normal((5 * chunk + 37, net.NIN)).astype(np.float32)
    pieces = [(k, min(k + 50000, len(feat))) for k in range(0, len(feat), 50000)]
    want = np.concatenate([net.predict(feat[a:b]) for a, b in pieces])
    for n in (1, 127, chunk - 1, chunk, chunk + 1, 4 * chunk, 4 * chunk + 1, len(feat)):
        np.testing.assert_array_equal(net.predict(feat[:n]), want[:n])
    # a net whose first call is the longest
    other = gpu.WarmStartNet(hidden=2, width=width, seed=5)
    np.testing.assert_array_equal(other.predict(feat), want)
