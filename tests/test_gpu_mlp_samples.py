"""A training step draws from the samples that the network has at the call: after
samples were added or cleared between two calls of the same batch and rate, the
weights are those of a network whose second call records its step anew."""
import numpy as np
import pytest

from helpers import make_gpu, small_case

pytestmark = pytest.mark.gpu


def _solved(aoa):
    p, bl = small_case(nx=65, ny=17, Ma=0.5, AoA=aoa, Re=1.0e6, If_viscous=1, Iflag_turbulence_model=2, Iflag_flux=4,
                       Iflag_Scheme=5, CFL=5.0, first=2e-4)
    s = make_gpu(p, bl)
    s.init_flow()
    s.step(20)
    return s


@pytest.mark.parametrize("width", [128, 256])
@pytest.mark.parametrize("clear", [False, True])
def test_samples_between_calls(gpu_lib, width, clear):
    a, b = _solved(1.0), _solved(3.0)
    nets = [gpu_lib.WarmStartNet(hidden=2, width=width, seed=3) for _ in range(2)]
    for k, net in enumerate(nets):
        net.add_samples(a)
        if clear:
            net.add_samples(b)
        net.fit_normalization()
        net.train(5, batch=512, lr=1e-3)
        if clear:
            net.clear_samples()
            net.add_samples(a)
        else:
            net.add_samples(b)
        if k:
            net.train(0, batch=512, lr=2e-3)  # no step, another rate: the next call records its own
        net.train(5, batch=512, lr=1e-3)
    for l in range(nets[0].nlin):
        for x, y in zip(nets[0].get_weights(l), nets[1].get_weights(l)):
            np.testing.assert_array_equal(x, y)
    for s in (a, b, *nets):
        s.close()


def test_samples_beyond_the_first_allocation(gpu_lib):
    """the pool moves when it grows past 2^20 rows: training goes on from the new one"""
    a = _solved(1.0)
    net = gpu_lib.WarmStartNet(hidden=2, width=256, seed=3)
    net.add_samples(a)
    net.fit_normalization()
    net.train(2, batch=512, lr=1e-3)
    while net.num_samples() <= 1 << 20:
        net.add_samples(a)
    assert np.isfinite(net.train(2, batch=512, lr=1e-3))
    net.close(), a.close()
