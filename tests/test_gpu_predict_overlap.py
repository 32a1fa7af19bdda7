"""Predictions into a buffer that overlaps the features: as a call whose results go
elsewhere, also where a chunk's results lie on the features of a later one."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 7 * 4 * 77824, 5 * 77824 + 3])
def test_results_over_features(gpu_lib, shift):
    n = 5 * 77824 + 11  # one chunk more than the ring
    net = gpu_lib.WarmStartNet(hidden=2, width=256, seed=5)
    rng = np.random.default_rng(7)
    feat = rng.standard_normal((n, net.NIN)).astype(np.float32)
    want = net.predict(feat)
    buf = np.zeros(shift + n * net.NIN, np.float32)
    buf[:n * net.NIN] = feat.reshape(-1)
    fp = ctypes.POINTER(ctypes.c_float)
    out = buf[shift:shift + n * net.NOUT]
    assert net.L.ec2d_mlp_predict(net.h, buf.ctypes.data_as(fp), n, out.ctypes.data_as(fp)) == 0
    np.testing.assert_array_equal(out.reshape(n, net.NOUT), want)
    net.close()
