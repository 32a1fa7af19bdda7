"""The fused network kernels (width 256, tcgen05) against the mma.sync kernels
at the sizes where their bookkeeping can go wrong: one and two tiles of 128
rows, batches that split in 32, 16, 8 and fewer parts, one hidden layer (no
stored layer between), two, and many; predictions of a part of a tile, a whole
one, and more tiles than SMs."""
import numpy as np
import pytest

import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _pair(gpu, hidden):
    """Two equal networks with non-zero biases: fused and mma.sync."""
    rng = np.random.default_rng(hidden)
    nets = [gpu.WarmStartNet(hidden=hidden, width=256, seed=4) for _ in range(2)]
    for l in range(nets[0].nlin):
        W, b = nets[0].get_weights(l)
        b[:mo.NOUT if l == nets[0].nlin - 1 else W.shape[0]] = rng.normal(
            0, 0.1, mo.NOUT if l == nets[0].nlin - 1 else W.shape[0])
        for n in nets:
            n.set_weights(l, W, b)
    nets[1].set_gemm(0)
    return nets


def _near(a, b, tol):
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b) + 1e-12, np.linalg.norm(a - b) / np.linalg.norm(b)


# two paths differ in FP32 summation order only; a BF16 rounding that goes the
# other way (2^-8 of a value, about one in a hundred values) moves a layer by
# 2^-8 / sqrt(100) = 4e-4, and a gradient through 2 hidden + 1 layers by no more
# than 10 such steps
@pytest.mark.parametrize("hidden", [1, 2, 6, 12])
@pytest.mark.parametrize("batch", [256, 512, 768, 1792, 2048, 4096])
def test_gradients(gpu_lib, hidden, batch):
    if hidden == 12 and batch > 512:
        pytest.skip("depth is covered at the small batches")
    f, m = _pair(gpu_lib, hidden)
    rng = np.random.default_rng(batch)
    x = rng.normal(size=(batch, mo.NIN)).astype(np.float32)
    y = rng.normal(size=(batch, mo.NOUT)).astype(np.float32)
    lf, lm = f.loss_grad(x, y), m.loss_grad(x, y)
    assert abs(lf - lm) <= 1e-3 * lm
    for l in range(f.nlin):
        for a, b in zip(f.get_grads(l), m.get_grads(l)):
            assert np.all(np.isfinite(a))
            _near(a, b, 5e-3)
    assert np.all(f.get_grads(0)[0][:, mo.NIN:] == 0.0)
    assert np.all(f.get_grads(f.nlin - 1)[0][mo.NOUT:, :] == 0.0)
    f.close(), m.close()


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 152 * 128 - 1, 152 * 128 + 1, 40001])
def test_predictions(gpu_lib, rows):
    f, m = _pair(gpu_lib, 6)
    nrm = np.concatenate([np.full(7, 0.5), np.full(7, 2.0), np.full(5, 0.1), np.full(5, 3.0)]).astype(np.float32)
    for n in (f, m):
        n.set_normalization(nrm)
    x = np.random.default_rng(rows).normal(0.5, 2.0, size=(rows, mo.NIN)).astype(np.float32)
    a, b = f.predict(x), m.predict(x)
    assert a.shape == (rows, mo.NOUT) and np.all(np.isfinite(a))
    _near(a, b, 5e-3)
    f.close(), m.close()
