"""Residuals of levels at and just below the size from which the limited slopes are
formed per cell (262144 cells, k_slopes) against the CPU oracle, within the bound of
the other residual tests; above it also for a scheme that has no slopes, and after
a switch to FP32 sweeps."""
import pytest

from ec2d import grids
from ec2d.inputs import Params
from helpers import compare_residual, copy_state, make_gpu, make_oracle, perturb_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,flux,scheme,turb", [(513, 257, 6, 5, 0), (512, 257, 6, 5, 0), (513, 257, 4, 5, 2),
                                                    (513, 257, 6, 2, 0), (2049, 65, 3, 5, -1)])
def test_slope_levels(gpu_lib, nx, ny, flux, scheme, turb):
    p = Params(Ma=0.4, Re=1e5, If_viscous=int(turb >= 0), Iflag_turbulence_model=max(turb, 0), Iflag_flux=flux,
               Iflag_Scheme=scheme, CFL=1.0, Time_Method=0, P_outlet=1.0 / (1.4 * 0.16))
    bl = grids.flat_plate(nx, ny, first=2e-3, ratio=1.01)
    orc, g = make_oracle(p, bl, threads=16), make_gpu(p, bl)
    orc.init_flow(), g.init_flow()
    perturb_state(orc, amp=0.01, seed=nx)
    copy_state(orc, g)
    orc.residual(), g.residual()
    compare_residual(orc, g)
    g.set_lusgs_precision(32)
    g.residual()
    compare_residual(orc, g)
    g.close()
