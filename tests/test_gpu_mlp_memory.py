"""A batch whose buffers the device does not hold is refused as out of memory, gives
back what it had taken, and leaves the network as it was: gradients and training
steps of an earlier batch are those of a network that never asked."""
import gc

import numpy as np
import pytest
import torch

import mlp_oracle as mo
from ec2d import gpu
from helpers import make_gpu, small_case

pytestmark = pytest.mark.gpu

EC2D_ERR_NOMEM = 6
TOO_LARGE = 1 << 29  # 275 GB for the activations of one layer


@pytest.mark.parametrize("kind", [0, 1])
def test_refused_batch(gpu_lib, kind):
    p, bl = small_case(nx=65, ny=17, Ma=0.5, AoA=1.0, Re=1.0e6, If_viscous=1, Iflag_turbulence_model=2, Iflag_flux=4,
                       Iflag_Scheme=5, CFL=5.0, first=2e-4)
    s = make_gpu(p, bl)
    s.init_flow()
    s.step(20)
    rng = np.random.default_rng(5)
    x = rng.normal(size=(512, mo.NIN)).astype(np.float32)
    y = rng.normal(size=(512, mo.NOUT)).astype(np.float32)
    outs = []
    for ask in (True, False):
        net = gpu_lib.WarmStartNet(hidden=3, width=256, seed=3)
        net.set_gemm(kind)
        net.add_samples(s)
        net.fit_normalization()
        net.train(3, batch=512, lr=1e-3)
        if ask:
            gc.collect()  # (contexts and nets of other tests)
            free = torch.cuda.mem_get_info()[0]
            with pytest.raises(gpu.EC2DError) as e:
                net.train(1, batch=TOO_LARGE, lr=1e-3)
            assert e.value.code == EC2D_ERR_NOMEM
            assert torch.cuda.mem_get_info()[0] >= free
        loss = net.loss_grad(x, y)
        grads = [a for l in range(net.nlin) for a in net.get_grads(l)]
        net.train(3, batch=512, lr=2e-3)  # a step recorded after the refusal
        net.train(2, batch=1024, lr=2e-3)
        outs.append([np.float64(loss), *grads, *[a for l in range(net.nlin) for a in net.get_weights(l)]])
        net.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
    s.close()


def _taken(kind, call):
    net = gpu.WarmStartNet(hidden=6, width=256, seed=3)
    net.set_gemm(kind)
    gc.collect()
    free = torch.cuda.mem_get_info()[0]
    call(net)
    n = free - torch.cuda.mem_get_info()[0]
    net.close()
    return n


def test_gradients_of_large_batches(gpu_lib):
    """the fused kernels take no more than the separate ones, whose buffers they do without"""
    x, y = np.zeros((65536, mo.NIN), np.float32), np.zeros((65536, mo.NOUT), np.float32)
    _taken(1, lambda net: net.loss_grad(x[:256], y[:256]))
    assert _taken(1, lambda net: net.loss_grad(x, y)) <= _taken(0, lambda net: net.loss_grad(x, y))
