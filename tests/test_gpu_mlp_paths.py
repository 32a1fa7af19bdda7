"""One network on both GEMM paths in turn: what a path computes after training on
the other one are the bits of a fresh network on that path with the same weights."""
import numpy as np
import pytest

import mlp_oracle as mo
from helpers import make_gpu, small_case

pytestmark = pytest.mark.gpu


def _samples(net):
    p, bl = small_case(nx=65, ny=17, Ma=0.5, AoA=1.0, Re=1.0e6, If_viscous=1, Iflag_turbulence_model=2, Iflag_flux=4,
                       Iflag_Scheme=5, CFL=5.0, first=2e-4)
    s = make_gpu(p, bl)
    s.init_flow()
    s.step(20)
    net.add_samples(s)
    net.fit_normalization()
    s.close()


@pytest.mark.parametrize("width", [128, 256])
@pytest.mark.parametrize("kind", [0, 1])
def test_train_then_switch(gpu_lib, width, kind):
    net = gpu_lib.WarmStartNet(hidden=2, width=width, seed=3)
    _samples(net)
    rng = np.random.default_rng(5)
    x = rng.normal(size=(512, mo.NIN)).astype(np.float32)
    y = rng.normal(size=(512, mo.NOUT)).astype(np.float32)
    net.set_gemm(kind)
    net.train(20, batch=512, lr=1e-2)
    net.set_gemm(1 - kind)
    fresh = gpu_lib.WarmStartNet(hidden=2, width=width, seed=4)
    fresh.set_gemm(1 - kind)
    fresh.set_normalization(net.get_normalization())
    for l in range(net.nlin):
        fresh.set_weights(l, *net.get_weights(l))
    np.testing.assert_array_equal(net.predict(x), fresh.predict(x))
    assert net.loss_grad(x, y) == fresh.loss_grad(x, y)
    for l in range(net.nlin):
        for a, b in zip(net.get_grads(l), fresh.get_grads(l)):
            np.testing.assert_array_equal(a, b)
    net.close(), fresh.close()
