"""What a context takes on the device does not depend on the kernels chosen for it: a
level with the slopes pass (k_slopes) takes what one without takes, in FP64 and after a
switch to FP32 sweeps, and the SST model's scratch is five planes (k and omega of the
faces go into planes that the context has anyway)."""
import gc

import pytest
import torch

from ec2d import gpu, grids
from ec2d.inputs import Params

pytestmark = pytest.mark.gpu


def _taken(nx, ny, scheme, turb, bits=64):
    p = Params(Ma=0.4, Re=1e6, If_viscous=1, Iflag_turbulence_model=turb, Iflag_flux=6, Iflag_Scheme=scheme, CFL=1.0,
               Time_Method=0, P_outlet=1.0 / (1.4 * 0.16), **(dict(Kt_inf=1e-6, Wt_inf=1e-2) if turb == 3 else {}))
    bl = grids.flat_plate(nx, ny, first=2e-3, ratio=1.005)
    gc.collect()  # (contexts and nets of other tests)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    g = gpu.Solver([(p, bl)])
    g.set_lusgs_precision(bits)
    g.init_flow()
    g.residual()
    g.sync()
    n = free - torch.cuda.mem_get_info()[0]
    g.close()
    return n


@pytest.mark.parametrize("nx,ny,bits", [(385, 257, 64), (385, 257, 32), (1025, 257, 64), (1025, 513, 64)])
def test_slopes_take_no_memory(gpu_lib, nx, ny, bits):
    _taken(33, 33, 5, 0)  # the process's own first allocations
    # MUSCL3 (with the pass) against NND2 (never)
    assert _taken(nx, ny, 5, 0, bits) == _taken(nx, ny, 1, 0, bits)


def test_sst_scratch(gpu_lib):
    nx, ny = 4097, 257
    _taken(33, 33, 5, 3)
    frame = 2 * (nx + 5) * (ny + 5) * 8
    # beside SA: one variable more in U, Res, dU and Un, 2 x 3 more words per cell in the
    # sweep records, and the scratch; allocations are rounded up to 2 MiB at most, five of them
    assert _taken(nx, ny, 5, 3) - _taken(nx, ny, 5, 2) <= (4 + 6 + 5) * frame + 5 * 2 ** 21
